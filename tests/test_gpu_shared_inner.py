"""Inner products whose outputs share plaintexts, and rescales on their own inputs.

afhe_eval_diag_inner_batch adds up a group's plaintexts before it multiplies
and forms a group of the outputs with the same units: here several sources
with the same units and giant steps, in groups of all, some and one of them,
one output with more units than the sums hold between two reductions (with
plaintexts that are all q - 1), one without units; equal word for word to
afhe_eval_mac_plain_batch. afhe_rescale_batch reads its inputs in place where
outputs start on them or lie apart; equal to the outputs of separate
polynomials in every arrangement.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FheContext, galois_elt
from tests.helpers import primes_for, uniform_residues
from tests.test_gpu_mac_plain import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,q_bits,local,accumulate", [
    (16, 50, True, False), (8, 45, True, True), (4, 50, True, False), (1, 50, True, False), (16, 60, True, True),
    (2, 60, True, False), (16, 50, False, True), (1, 60, False, False)])
def test_shared_units(nb, q_bits, local, accumulate):
    log_n, limbs, giants = 13, 3, 8
    q, p = primes_for(log_n, limbs, q_bits, 1, 61 if q_bits == 60 else 60)
    n = 1 << log_n
    w = limbs * n
    ctx = FheContext(CkksParams(log_n, q, p, 1), poly_words=640 * w, key_words=1024)
    try:
        rng = np.random.default_rng([nb, q_bits])
        rows = [uniform_residues(rng, q, n) for _ in range(400)]
        for k in range(60, 100):
            rows[k] = np.repeat(np.array(q, dtype=np.uint64) - 1, n)        # plaintexts of all q - 1
        ctx.write_poly(0, np.concatenate(rows))
        srcs = [(2 * i * w, (2 * i + 1) * w) for i in range(24)]            # [0, 48 w)
        gals = [1, galois_elt(log_n, -256), galois_elt(log_n, 512 if local else 5)]
        stride = w
        near = lambda g: [(100 + 20 * k + nb * g) * w for k in range(5)]    # noqa: E731  (up to 100 + 80 + 16 * 8)
        far = lambda g: [(60 + (7 * k + g) % 24) * w for k in range(300)]   # noqa: E731
        jobs = [(s, near(g)) for s in (0, 3, 5) for g in range(giants)]     # three sources, one list
        jobs += [(s, near(g)[1:4]) for s in (1, 2) for g in range(giants)]  # two with another
        jobs += [(4, far(0)), (6, far(0)), (7, far(0)[:1]), (8, [])]
        outs = [((400 + 2 * j) * w, (401 + 2 * j) * w) for j in range(len(jobs))]
        outs_b = [(a + 100 * w, b + 100 * w) for a, b in outs]
        for o, ob in zip(outs, outs_b):
            for a, b in zip(o, ob):
                x = uniform_residues(rng, q, n)
                ctx.write_poly(a, x)
                ctx.write_poly(b, x)
        src = (L.CtRef * (len(jobs) * nb))(*[L.CtRef(*srcs[(s + b) % 24]) for s, _ in jobs for b in range(nb)])
        upt = np.array([u for _, us in jobs for u in us], dtype=np.uint64)
        ugal = np.array([gals[k % 3] for _, us in jobs for k in range(len(us))], dtype=np.uint32)
        first = np.concatenate([[0], np.cumsum([len(us) for _, us in jobs])]).astype(np.uint32)
        oa = (L.CtRef * len(jobs))(*[L.CtRef(*c) for c in outs])
        L.check(ctx.lib.afhe_eval_diag_inner_batch(ctx.h, oa, len(jobs), src, nb, upt.ctypes.data_as(L.P64),
                                                   ugal.ctypes.data_as(L.P32), first.ctypes.data_as(L.P32), stride,
                                                   limbs, int(accumulate)), "diag_inner")
        mac = [[(srcs[(s + b) % 24], [(u + b * stride, gals[k % 3]) for k, u in enumerate(us)]) for b in range(nb)]
               for s, us in jobs]
        for s in range(0, len(jobs), 8):        # a term per plaintext: fewer outputs fit its descriptors
            assert call(ctx, outs_b[s:s + 8], mac[s:s + 8], limbs, accumulate) == L.OK, ctx.lib.afhe_last_error()
        for j, (a, b) in enumerate(zip(outs, outs_b)):
            assert np.array_equal(ctx.read_poly(a[0], w), ctx.read_poly(b[0], w)), j
            assert np.array_equal(ctx.read_poly(a[1], w), ctx.read_poly(b[1], w)), j
    finally:
        ctx.close()


@pytest.mark.parametrize("log_n,limbs", [(10, 2), (13, 3), (15, 3)])
def test_rescale_over_its_inputs(log_n, limbs):
    q, p = primes_for(log_n, limbs, 40, 1, 60)
    n = 1 << log_n
    w = limbs * n
    ctx = FheContext(CkksParams(log_n, q, p, 1), poly_words=64 * w, key_words=1024)
    count = 5
    try:
        rng = np.random.default_rng([log_n, limbs])
        data = [uniform_residues(rng, q, n) for _ in range(2 * count)]
        ins = [(2 * i * w, (2 * i + 1) * w) for i in range(count)]

        def run(outs):
            ctx.write_poly(0, np.concatenate(data))
            a = (L.CtRef * count)(*[L.CtRef(*c) for c in ins])
            d = (L.CtRef * count)(*[L.CtRef(*c) for c in outs])
            L.check(ctx.lib.afhe_rescale_batch(ctx.h, a, d, count, limbs), "rescale")
            return [ctx.read_poly(o, w - n) for c in outs for o in c]

        apart = run([((32 + 2 * i) * w, (33 + 2 * i) * w) for i in range(count)])
        arrangements = {
            "in place": ins,
            "one moved": ins[:-1] + [(40 * w, 41 * w)],
            "a limb on": [(a + n, b + n) for a, b in ins],
            "polynomials swapped": [(b, a) for a, b in ins],
            "turned": ins[1:] + ins[:1],
        }
        for name, outs in arrangements.items():
            for x, y in zip(apart, run(outs)):
                assert np.array_equal(x, y), name
    finally:
        ctx.close()


@pytest.mark.parametrize("log_n,limbs,q_bits", [(11, 2, 40), (13, 3, 55), (14, 3, 40)])
def test_plaintext_product_over_its_operands(log_n, limbs, q_bits):
    """The product formed inside the rescale equals the one through temporaries
    (outputs over the plaintexts or another input), shared plaintexts included."""
    q, p = primes_for(log_n, limbs, q_bits, 1, 60)
    n = 1 << log_n
    w = limbs * n
    ctx = FheContext(CkksParams(log_n, q, p, 1), poly_words=64 * w, key_words=1024)
    count = 5
    try:
        rng = np.random.default_rng([log_n, limbs])
        data = [uniform_residues(rng, q, n) for _ in range(3 * count)]
        data[0] = np.repeat(np.array(q, dtype=np.uint64) - 1, n)
        data[2 * count] = data[0]
        ins = [(2 * i * w, (2 * i + 1) * w) for i in range(count)]
        pts = [(2 * count + i % 3) * w for i in range(count)]

        def run(outs):
            ctx.write_poly(0, np.concatenate(data))
            a = (L.CtRef * count)(*[L.CtRef(*c) for c in ins])
            d = (L.CtRef * count)(*[L.CtRef(*c) for c in outs])
            f = (L.u64 * count)(*pts)
            L.check(ctx.lib.afhe_eval_mult_plain_rescale_batch(ctx.h, a, f, d, count, limbs), "mult_plain_rescale")
            return [ctx.read_poly(o, w - n) for c in outs for o in c]

        over = run([((2 * count) * w, (2 * count + 1) * w)] + [((32 + 2 * i) * w, (33 + 2 * i) * w) for i in range(1, count)])
        arrangements = {
            "apart": [((32 + 2 * i) * w, (33 + 2 * i) * w) for i in range(count)],
            "in place": ins,
            "turned": ins[1:] + ins[:1],
        }
        for name, outs in arrangements.items():
            for x, y in zip(over, run(outs)):
                assert np.array_equal(x, y), name
    finally:
        ctx.close()

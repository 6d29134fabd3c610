"""Operands of afhe_eval_diag_inner_batch at the edges of its shared-memory form.

Where a source polynomial starts at an odd word, its 16-byte copies would not be
aligned: the call takes the form that reads word by word. One odd polynomial
among even ones, first, last and in the middle, c0 or c1; equal word for word
to afhe_eval_mac_plain_batch. Words that are no residues, in either form.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FheContext, galois_elt
from tests.helpers import primes_for, uniform_residues
from tests.test_gpu_mac_plain import call

pytestmark = pytest.mark.gpu

LOG_N, LIMBS = 11, 2


def diag(ctx, outs, srcs, nb, units, gals, stride, limbs, accumulate=0):
    """One call: outs[j] from sources srcs[j] (nb of them) and units[j] (plaintext offsets)."""
    oa = (L.CtRef * len(outs))(*[L.CtRef(*c) for c in outs])
    src = (L.CtRef * (len(outs) * nb))(*[L.CtRef(*c) for s in srcs for c in s])
    upt = np.array([u for us in units for u in us] or [0], dtype=np.uint64)
    ugal = np.array([gals[k % len(gals)] for us in units for k in range(len(us))] or [1], dtype=np.uint32)
    first = np.concatenate([[0], np.cumsum([len(us) for us in units])]).astype(np.uint32)
    return ctx.lib.afhe_eval_diag_inner_batch(ctx.h, oa, len(outs), src, nb, upt.ctypes.data_as(L.P64),
                                              ugal.ctypes.data_as(L.P32), first.ctypes.data_as(L.P32), stride, limbs,
                                              accumulate)


@pytest.mark.parametrize("nb,q_bits", [(1, 50), (4, 50), (16, 50), (2, 60), (16, 60)])
@pytest.mark.parametrize("which", ["c0 of the first", "c1 of the last", "c0 in the middle"])
@pytest.mark.parametrize("nu", [3, 5])
def test_sources_at_odd_words(nb, q_bits, which, nu):
    q, p = primes_for(LOG_N, LIMBS, q_bits, 1, 61 if q_bits == 60 else 60)
    n = 1 << LOG_N
    w = LIMBS * n
    ctx = FheContext(CkksParams(LOG_N, q, p, 1), poly_words=180 * w, key_words=1024)
    try:
        rng = np.random.default_rng([nb, q_bits])
        srcs = [[(2 * b * w, (2 * b + 1) * w) for b in range(nb)] for _ in range(2)]
        j, b = {"c0 of the first": (0, 0), "c1 of the last": (1, nb - 1), "c0 in the middle": (1, nb // 2)}[which]
        odd = 40 * w + 1
        srcs[j][b] = (srcs[j][b][0], odd) if which.startswith("c1") else (odd, srcs[j][b][1])
        for at in {o for s in srcs for c in s for o in c}:
            ctx.write_poly(at, uniform_residues(rng, q, n))
        for k in range(48, 48 + (nu + 1) * nb):
            ctx.write_poly(k * w, uniform_residues(rng, q, n))
        gals = [1, galois_elt(LOG_N, -64), galois_elt(LOG_N, -256)]
        units = [[(48 + nb * k) * w for k in range(nu)], [(48 + nb * k) * w for k in range(1, nu + 1)]]
        outs = [((160 + 2 * j) * w, (161 + 2 * j) * w) for j in range(2)]
        outs_b = [((170 + 2 * j) * w, (171 + 2 * j) * w) for j in range(2)]
        assert diag(ctx, outs, srcs, nb, units, gals, w, LIMBS) == L.OK, ctx.lib.afhe_last_error()
        mac = [[(srcs[j][b], [(u + b * w, gals[k % 3]) for k, u in enumerate(units[j])]) for b in range(nb)]
               for j in range(2)]
        assert call(ctx, outs_b, mac, LIMBS) == L.OK, ctx.lib.afhe_last_error()
        for a, b in zip(outs, outs_b):
            assert np.array_equal(ctx.read_poly(a[0], w), ctx.read_poly(b[0], w))
            assert np.array_equal(ctx.read_poly(a[1], w), ctx.read_poly(b[1], w))
    finally:
        ctx.close()


@pytest.mark.parametrize("nb", [1, 4, 16])
@pytest.mark.parametrize("what", ["plaintexts", "sources", "both"])
@pytest.mark.parametrize("nu", [2, 5])
@pytest.mark.parametrize("local", [True, False])
def test_words_that_are_no_residues(nb, what, local, nu):
    """Below 2^50 the products split words in halves: other words are taken modulo
    their prime, any by the form for any placement, plaintexts below 2^57 and
    sources below 2^53 by the shared-memory form."""
    q = primes_for(LOG_N, LIMBS, 50, 1, 60)[0][:1] + primes_for(LOG_N, LIMBS, 36, 1, 60)[0][:1]
    p = primes_for(LOG_N, LIMBS, 50, 1, 60)[1]
    n = 1 << LOG_N
    w = LIMBS * n
    ctx = FheContext(CkksParams(LOG_N, q, p, 1), poly_words=200 * w, key_words=1024)
    try:
        rng = np.random.default_rng([nb, local])

        def poly(words, most):
            x = uniform_residues(rng, q, n)
            y = x.copy()
            if words:
                y[::3] = rng.integers(0, most, y[::3].size, dtype=np.uint64)
                y[1::7] = np.uint64(most - 1)
                y[2::11] = np.uint64(2 ** 50)
                y[5::13] = np.uint64(2 ** 50 - 1)
                x = np.concatenate([y[l * n:(l + 1) * n] % np.uint64(q[l]) for l in range(LIMBS)])
            return x, y

        srcs = [[(2 * b * w, (2 * b + 1) * w) for b in range(nb)]]
        gals = [galois_elt(LOG_N, 128 if local else 5), 1, galois_elt(LOG_N, -64)]
        units = [[(40 + nb * k) * w for k in range(nu)]]
        most = (1 << 53, 1 << 57) if local else (1 << 64, 1 << 64)
        data = {k: poly(what != "plaintexts", most[0]) if k < 32 else poly(what != "sources", most[1])
                for k in [*range(2 * nb), *range(40, 40 + nu * nb)]}
        got = []
        for form in range(2):              # residues through the sums of products, then the words
            for k, v in data.items():
                ctx.write_poly(k * w, v[form])
            out = [((150 + 2 * form) * w, (151 + 2 * form) * w)]
            if form == 0:
                mac = [[(srcs[0][b], [(u + b * w, gals[k % 3]) for k, u in enumerate(units[0])]) for b in range(nb)]]
                assert call(ctx, out, mac, LIMBS) == L.OK, ctx.lib.afhe_last_error()
            else:
                assert diag(ctx, out, srcs, nb, units, gals, w, LIMBS) == L.OK, ctx.lib.afhe_last_error()
            got.append([ctx.read_poly(o, w) for o in out[0]])
        assert np.array_equal(got[0][0], got[1][0])
        assert np.array_equal(got[0][1], got[1][1])
    finally:
        ctx.close()


@pytest.mark.parametrize("nb", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("q_bits", [50, 61])
@pytest.mark.parametrize("nu,shared", [(1, False), (2, False), (3, False), (4, False), (1, True), (3, True)])
def test_few_units(nb, q_bits, nu, shared):
    """Outputs of one to three units are read straight through, unless they share
    their plaintexts; plaintexts and sources of all q - 1 among them."""
    q, p = primes_for(LOG_N, LIMBS, q_bits, 1, 60)
    n = 1 << LOG_N
    w = LIMBS * n
    top = np.repeat(np.array(q, dtype=np.uint64) - 1, n)
    ctx = FheContext(CkksParams(LOG_N, q, p, 1), poly_words=260 * w, key_words=1024)
    try:
        rng = np.random.default_rng([nb, q_bits, nu])
        for k in range(40 + 3 * nu * nb):
            ctx.write_poly(k * w, top if k % 5 < 2 else uniform_residues(rng, q, n))
        gals = [1, galois_elt(LOG_N, -64), galois_elt(LOG_N, 256)]
        srcs = [[((2 * b + j) * w, (2 * b + 1 + j) * w) for b in range(nb)] for j in range(3)]
        units = [[(40 + nb * (k + (0 if shared else j) * nu)) * w for k in range(nu)] for j in range(3)]
        outs = [((240 + 2 * j) * w, (241 + 2 * j) * w) for j in range(3)]
        outs_b = [((250 + 2 * j) * w, (251 + 2 * j) * w) for j in range(3)]
        for accumulate in (0, 1):
            assert diag(ctx, outs, srcs, nb, units, gals, w, LIMBS, accumulate) == L.OK, ctx.lib.afhe_last_error()
            mac = [[(srcs[j][b], [(u + b * w, gals[k % 3]) for k, u in enumerate(units[j])]) for b in range(nb)]
                   for j in range(3)]
            assert call(ctx, outs_b, mac, LIMBS, accumulate) == L.OK, ctx.lib.afhe_last_error()
            for a, b in zip(outs, outs_b):
                assert np.array_equal(ctx.read_poly(a[0], w), ctx.read_poly(b[0], w)), accumulate
                assert np.array_equal(ctx.read_poly(a[1], w), ctx.read_poly(b[1], w)), accumulate
    finally:
        ctx.close()

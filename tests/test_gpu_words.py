"""Transforms and key switches of words that are no residues.

A forward transform takes words below 4q, an inverse one and a key switch words
below 2q (the ranges of butterflies with lazy reductions), modulo their primes:
at primes just below and above 2^50 (the two forms of the arithmetic), at a
small one and the largest allowed, equal to the oracle's results for the
residues, and for key switches on both paths with registered and unregistered
keys, one digit and several. What is only added (a rotation's c0, an accumulated
ciphertext) may make a sum that is no residue: congruent, and for the accumulated
ciphertext the same words on both paths.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.autotune import get_ntt_plan, set_ntt_plan
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext, find_ntt_primes
from oracle.composite import OracleCKKS
from oracle.oracle import tables_py as T
from tests.test_gpu_prime_classes import above

pytestmark = pytest.mark.gpu


def primes(log_n, count):
    qs = []
    for q in ([above(log_n, 50)], *(find_ntt_primes(log_n, b, 1, []) for b in (50, 61, 36, 55))):
        qs += [x for x in q if x not in qs]
    return qs[:count]


def words(rng, qs, n, most):
    """Words of limbs qs: some of [0, most q), some residues, the edges of the range."""
    out = []
    for q in qs:
        x = rng.integers(0, most * q, n, dtype=np.uint64)
        x[:n // 2:3] %= np.uint64(q)
        x[1], x[5], x[7], x[-1] = most * q - 1, q, (most - 1) * q, most * q - 1
        x[n // 2:n // 2 + 64] = most * q - 1
        x[n // 2 + 64:n // 2 + 128] = np.array([0, most * q - 1] * 32, dtype=np.uint64)
        out.append(x)
    return np.concatenate(out)


def reduced(x, qs):
    n = x.size // len(qs)
    return np.concatenate([x[i * n:(i + 1) * n] % np.uint64(q) for i, q in enumerate(qs)])


@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("log_n", [10, 12, 13, 14, 15, 16])
def test_transforms_of_words(log_n, plan, orc):
    qs = primes(log_n, 5)
    n = 1 << log_n
    rng = np.random.default_rng(log_n)
    keep = get_ntt_plan(log_n)
    try:
        set_ntt_plan(log_n, plan)
        with FheContext(CkksParams(log_n, qs, find_ntt_primes(log_n, 60, 1, qs), 1), poly_words=2 * n * len(qs),
                        key_words=1024, max_batch=1) as ctx:
            drv = FHEHostDriver(ctx)
            for most, run in ((4, drv.ntt), (2, drv.intt)):
                x = words(rng, qs, n, most)
                ctx.write_poly(0, x)
                run(0, x.size, len(qs))
                got = ctx.read_poly(x.size, x.size)
                for i, q in enumerate(qs):
                    s = slice(i * n, (i + 1) * n)
                    r = x[s] % np.uint64(q)
                    tw, itw = T.twiddles(log_n, q)
                    want = orc.ntt(r, tw, q) if most == 4 else orc.intt(r, itw, q)
                    assert np.array_equal(got[s], want), (q, most)
    finally:
        set_ntt_plan(log_n, keep)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("log_n,nq,alpha", [(10, 3, 3), (10, 5, 2), (12, 4, 4), (13, 3, 1), (14, 4, 4), (15, 3, 2)])
def test_key_switch_of_words(log_n, nq, alpha, fused, orc):
    qs = primes(log_n, nq)
    ps = find_ntt_primes(log_n, 49, 1, qs) + find_ntt_primes(log_n, 60, 1, qs)
    p = CkksParams(log_n, qs, ps, alpha)
    n, kw, w = p.n, p.key_words(), nq << log_n
    rng = np.random.default_rng([log_n, nq])
    keys = [np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * p.dnum) for q in qs + ps])
            for _ in range(2)]
    halves = [(k[:kw // 2], k[kw // 2:]) for k in keys]
    ora = OracleCKKS(log_n, qs, ps, alpha, orc)
    with FheContext(p, poly_words=6 * w, key_words=2 * kw, max_batch=2) as ctx:
        if fused and ctx.get_option(L.OPT_KS_FUSED) != 1:
            pytest.skip("the one-kernel key switch does not run on this GPU at this ring degree")
        drv = FHEHostDriver(ctx)
        for k in range(2):
            ctx.write_key(k * kw, keys[k])
        drv.add_rotation_key(1, 0)
        ctx.set_option(L.OPT_KS_FUSED, int(fused))
        ctx.set_option(L.OPT_FUSED_MIN, 1)
        x, y = words(rng, qs, n, 2), words(rng, qs, n, 4)
        acc = [words(rng, qs, n, 4) for _ in range(2)]
        rx, ry = reduced(x, qs), reduced(y, qs)
        for evk in range(2):                       # a registered key, and one that is not
            ctx.write_poly(0, x)
            drv.key_switch(0, evk * kw, w, 2 * w, nq)
            want = ora.key_switch(rx, *halves[evk], nq)
            for h in range(2):
                assert np.array_equal(ctx.read_poly((1 + h) * w, w), want[h]), (evk, h)
        # a rotation: c1 is switched, c0 and the accumulated ciphertext are added
        want = ora.eval_rotate_single_step((ry, rx), 1, {1: halves[0]}, nq)
        for k, v in enumerate((y, x, *acc)):
            ctx.write_poly(k * w, v)
        drv.eval_rotate_single_step(0, w, 4 * w, 5 * w, 1, nq)
        got = [ctx.read_poly(4 * w, w), ctx.read_poly(5 * w, w)]
        assert np.array_equal(reduced(got[0], qs), want[0])
        assert np.array_equal(got[1], want[1])
        ctx.write_poly(0, ry)
        a, d = (L.CtRef * 1)(L.CtRef(0, w)), (L.CtRef * 1)(L.CtRef(2 * w, 3 * w))
        L.check(ctx.lib.afhe_eval_rotate_accumulate_batch(ctx.h, a, d, 1, 1, nq), "rotate_accumulate")
        qrow = np.repeat(np.array(qs, dtype=np.uint64), n)
        for h in range(2):
            s = want[h] + acc[h]                   # (below 5q < 2^64)
            assert np.array_equal(ctx.read_poly((2 + h) * w, w), np.where(s >= qrow, s - qrow, s)), h

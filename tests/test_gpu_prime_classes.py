"""Transforms and key switches with primes on both sides of 2^50.

A transform's arithmetic follows its prime: whole numbers in doubles below
2^50, split 32-bit products above (up to 2^61). Here one context mixes primes
at the edges of both ranges (the largest below 2^61, the smallest above 2^50,
the largest below 2^50, a small one), with residues at the edges of [0, q)
besides uniform ones: transforms equal the oracle's (the reference's loop,
hls/src/ntt.cpp:4-80), and the one-kernel key switch equals the kernel pipeline
at every ring degree and the oracle at the small ones, with one and with
several digits, registered and unregistered keys.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext, find_ntt_primes
from oracle.composite import OracleCKKS
from oracle.oracle import tables_py as T

pytestmark = pytest.mark.gpu


def is_prime(n: int) -> bool:
    d, r = n - 1, 0
    while d % 2 == 0:
        d, r = d // 2, r + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(r - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def above(log_n: int, bits: int) -> int:
    """The smallest prime above 2^bits that is 1 mod 2N."""
    q = (1 << bits) + 1
    while not is_prime(q):
        q += 2 << log_n
    return q


def edge_primes(log_n: int) -> list[int]:
    q = find_ntt_primes(log_n, 61, 1) + [above(log_n, 50)]
    q += find_ntt_primes(log_n, 50, 1, q)
    return q + find_ntt_primes(log_n, 36, 1, q)


def edge_rows(rng, q: int, n: int) -> np.ndarray:
    """Uniform, all 0, all q - 1, alternating, a single q - 1."""
    one = np.zeros(n, dtype=np.uint64)
    one[n // 3] = q - 1
    alt = np.where(np.arange(n) % 2 == 0, 0, q - 1).astype(np.uint64)
    return np.stack([rng.integers(0, q, n, dtype=np.uint64), np.zeros(n, dtype=np.uint64),
                     np.full(n, q - 1, dtype=np.uint64), alt, one])


@pytest.mark.parametrize("log_n", [10, 12, 13, 14, 16])
def test_transforms_at_the_edges(log_n, orc):
    qs = edge_primes(log_n)
    p = CkksParams(log_n, qs, find_ntt_primes(log_n, 60, 1, qs), 4)
    n, w = p.n, len(qs) << log_n
    rng = np.random.default_rng(log_n)
    rows = [edge_rows(rng, q, n) for q in qs]
    polys = [np.concatenate([rows[i][k] for i in range(len(qs))]) for k in range(5)]
    with FheContext(p, poly_words=5 * w, key_words=1024, max_batch=1) as ctx:
        offs = (L.u64 * 5)(*[k * w for k in range(5)])
        for k in range(5):
            ctx.write_poly(k * w, polys[k])
        L.check(ctx.lib.afhe_ntt_batch(ctx.h, offs, 5, len(qs), 0), "ntt_batch")
        got = [ctx.read_poly(k * w, w) for k in range(5)]
        L.check(ctx.lib.afhe_ntt_batch(ctx.h, offs, 5, len(qs), 1), "ntt_batch")
        back = [ctx.read_poly(k * w, w) for k in range(5)]
    for i, q in enumerate(qs):
        tw, _ = T.twiddles(log_n, q)
        for k in range(5):
            assert np.array_equal(got[k][i * n:(i + 1) * n], orc.ntt(rows[i][k], tw, q)), (q, k)
    for k in range(5):
        assert np.array_equal(back[k], polys[k]), k


@pytest.mark.parametrize("registered", [True, False])
@pytest.mark.parametrize("alpha", [1, 2, 4])
@pytest.mark.parametrize("log_n", [10, 11, 12, 13, 14, 15, 16])
def test_key_switch_with_mixed_primes(log_n, alpha, registered, orc):
    qs = edge_primes(log_n)
    ps = find_ntt_primes(log_n, 49, 1, qs) + find_ntt_primes(log_n, 60, 1, qs)
    p = CkksParams(log_n, qs, ps, alpha)
    n, kw = p.n, p.key_words()
    rng = np.random.default_rng([log_n, alpha])
    key = np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * p.dnum) for q in qs + ps])
    with FheContext(p, poly_words=6 * len(qs) * n, key_words=kw, max_batch=2) as ctx:
        drv, w = FHEHostDriver(ctx), len(qs) * n
        ctx.write_key(0, key)
        if registered:
            drv.add_rotation_key(1, 0)
        if ctx.get_option(L.OPT_KS_FUSED) != 1:
            pytest.skip("the one-kernel key switch does not run on this GPU at this ring degree")
        ctx.set_option(L.OPT_FUSED_MIN, 1)
        for lv in (len(qs), 3, 1):
            for row in (0, 2):
                x = np.concatenate([edge_rows(rng, q, n)[row] for q in qs[:lv]])
                ctx.write_poly(0, x)
                out = []
                for fused in (1, 0):
                    ctx.set_option(L.OPT_KS_FUSED, fused)
                    drv.key_switch(0, 0, w, 2 * w, lv)
                    out.append([ctx.read_poly(w, lv * n), ctx.read_poly(2 * w, lv * n)])
                for a, b in zip(*out):
                    assert np.array_equal(a, b), (lv, row)
                if log_n <= 11:
                    ora = OracleCKKS(log_n, qs, ps, alpha, orc)
                    for a, b in zip(out[0], ora.key_switch(x, key[:kw // 2], key[kw // 2:], lv)):
                        assert np.array_equal(a, b), (lv, row)

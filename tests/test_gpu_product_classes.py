"""Products and rescales with primes on both sides of 2^50, against the oracle.

Pointwise products take doubles below 2^50 and 128 bits above, the rescale's and
the key switch's constants each prime's own form, and base conversions sum their
products before one reduction. One context mixes primes at the edges of both
ranges, has more digits than the inner product loads at a time (five and six),
and multiplies uniform residues and residues that are all q - 1.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext, find_ntt_primes
from oracle.composite import OracleCKKS
from tests.test_gpu_prime_classes import above

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,alpha", [(10, 1), (10, 3), (11, 2), (13, 1), (14, 2)])
def test_products_against_oracle(log_n, alpha, orc):
    qs = [above(log_n, 50)]
    for bits in (50, 61, 36, 45, 55):
        qs += find_ntt_primes(log_n, bits, 1, qs)
    ps = find_ntt_primes(log_n, 49, 1, qs) + find_ntt_primes(log_n, 60, 2, qs)
    p = CkksParams(log_n, qs, ps, alpha)
    n, kw, w = p.n, p.key_words(), len(qs) << log_n
    rng = np.random.default_rng([log_n, alpha])
    key = np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * p.dnum) for q in qs + ps])
    ora = OracleCKKS(log_n, qs, ps, alpha, orc)
    with FheContext(p, poly_words=8 * w, key_words=kw, max_batch=2) as ctx:
        drv = FHEHostDriver(ctx)
        ctx.write_key(0, key)
        drv.set_relin_key(0)
        for lv in (len(qs), 5, 2):
            for top in (False, True):
                def poly():
                    return np.concatenate([np.full(n, q - 1, dtype=np.uint64) if top else
                                           rng.integers(0, q, n, dtype=np.uint64) for q in qs[:lv]])
                x = [poly() for _ in range(4)]
                for k in range(4):
                    ctx.write_poly(k * w, x[k])
                a, b = (L.CtRef * 1)(L.CtRef(0, w)), (L.CtRef * 1)(L.CtRef(2 * w, 3 * w))
                d = (L.CtRef * 1)(L.CtRef(4 * w, 5 * w))
                pt = (L.u64 * 1)(2 * w)
                L.check(ctx.lib.afhe_eval_mult_plain_rescale_batch(ctx.h, a, pt, d, 1, lv), "mult_plain")
                want = ora.eval_mult_plain_rescale((x[0], x[1]), x[2], lv)
                for h in range(2):
                    assert np.array_equal(ctx.read_poly((4 + h) * w, (lv - 1) * n), want[h]), (lv, top, h)
                L.check(ctx.lib.afhe_eval_mult_relin_rescale_batch(ctx.h, a, b, d, 1, lv), "mult")
                want = ora.eval_mult_relin_rescale((x[0], x[1]), (x[2], x[3]), (key[:kw // 2], key[kw // 2:]), lv)
                for h in range(2):
                    assert np.array_equal(ctx.read_poly((4 + h) * w, (lv - 1) * n), want[h]), (lv, top, h)


@pytest.mark.parametrize("bits", [36, 50, 61])
def test_products_of_words_that_are_no_residues(bits):
    """Pointwise products reduce any two words exactly, whatever the prime's form."""
    log_n = 11
    q = find_ntt_primes(log_n, bits, 1, [])
    n = 1 << log_n
    p = CkksParams(log_n, q, find_ntt_primes(log_n, 60, 1, q), 1)
    rng = np.random.default_rng(bits)
    a = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    b = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    a[::3] %= np.uint64(q[0])
    b[::2] %= np.uint64(q[0])
    with FheContext(p, poly_words=3 * n, key_words=1024, max_batch=1) as ctx:
        ctx.write_poly(0, a)
        ctx.write_poly(n, b)
        FHEHostDriver(ctx).poly_mul_ntt(0, n, 2 * n, 1)
        got = ctx.read_poly(2 * n, n)
    want = (a.astype(object) * b.astype(object)) % q[0]
    assert np.array_equal(got, want.astype(np.uint64))

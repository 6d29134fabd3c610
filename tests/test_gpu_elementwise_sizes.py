"""Sums, differences and products of polynomials at both block shapes.

Launches of up to 2^16 words take one coefficient a thread, larger ones four: sizes
below, at and above that, primes below and above 2^50, equal to whole-number
arithmetic.
"""
import numpy as np
import pytest

from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext, find_ntt_primes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,limbs", [(10, 1), (10, 2), (14, 3), (15, 2), (15, 3), (16, 1), (16, 2)])
def test_elementwise(log_n, limbs):
    qs = [find_ntt_primes(log_n, bits, 1, [])[0] for bits in (60, 50, 36)][:limbs]
    p = CkksParams(log_n, qs, find_ntt_primes(log_n, 61, 1, qs), 1)
    n, w = p.n, limbs << log_n
    rng = np.random.default_rng([log_n, limbs])
    with FheContext(p, poly_words=3 * w, key_words=1024, max_batch=1) as ctx:
        drv = FHEHostDriver(ctx)
        a, b = (np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for q in qs]) for _ in range(2))
        for x in (a, b):
            x[:3], x[-1] = [0, 1, qs[0] - 1], qs[-1] - 1
        ctx.write_poly(0, np.concatenate([a, b]))
        q = np.repeat(np.array(qs, dtype=object), n)
        x, y = a.astype(object), b.astype(object)
        for run, want in ((drv.poly_add, (x + y) % q), (drv.poly_sub, (x - y) % q), (drv.poly_mul_ntt, x * y % q)):
            run(0, w, 2 * w, limbs)
            assert np.array_equal(ctx.read_poly(2 * w, w), want.astype(np.uint64)), run.__name__

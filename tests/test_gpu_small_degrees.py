"""Key switches at the small ring degrees, N = 2^10 to 2^12.

One CTA carries a ciphertext, 8 values a thread up to half a wave and 16 above it.
The line between the paths: below it every launch is the kernel pipeline's, from it
on the one kernel's, beyond a whole wave both; word for word the pipeline's
results, one digit and several, primes below and above 2^50.
"""
import numpy as np
import pytest
import torch

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext, find_ntt_primes

pytestmark = pytest.mark.gpu

# percent of a wave, by ring degree and digits (up to three)
LINE = {10: (3, 3, 12), 11: (11, 12, 18), 12: (25, 25, 32)}


@pytest.mark.parametrize("log_n,nq,np_,alpha", [(10, 2, 2, 2), (10, 2, 1, 1), (10, 5, 1, 1), (11, 2, 2, 2), (11, 3, 2, 2),
                                                (11, 4, 1, 1), (12, 2, 2, 2), (12, 3, 1, 1)])
@pytest.mark.parametrize("prep", [True, False])
def test_both_paths_around_the_line(log_n, nq, np_, alpha, prep):
    qs = find_ntt_primes(log_n, 50, 1, []) + find_ntt_primes(log_n, 58, nq - 1, [])
    p = CkksParams(log_n, qs, find_ntt_primes(log_n, 60, np_, qs), alpha)
    n, w = p.n, nq << log_n
    rng = np.random.default_rng([log_n, nq])
    key = np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * p.dnum) for q in p.q + p.p])
    with FheContext(p, poly_words=4 * w, key_words=p.key_words(), max_batch=8) as probe:
        if probe.get_option(L.OPT_KS_FUSED) != 1:
            pytest.skip("the one-kernel key switch does not run on this GPU")
        cap = probe.get_option(L.OPT_KS_CAPACITY)
    line = max(1, cap * LINE[log_n][min(p.dnum, 3) - 1] // 100)
    counts = sorted({1, line - 1, line, cap // 2, cap // 2 + 1, cap, cap + 1, cap + line})
    S = 16
    with FheContext(p, poly_words=(2 * S + 2 * max(counts)) * w, key_words=p.key_words(), max_batch=max(counts)) as ctx:
        drv = FHEHostDriver(ctx)
        ctx.write_key(0, key)
        if not prep:
            ctx.set_option(L.OPT_KS_FUSED, 0)          # (registered without a prepared copy)
        drv.add_rotation_key(1, 0)
        ctx.set_option(L.OPT_KS_FUSED, 1)
        ctx.write_poly(0, np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * S) for q in p.q]))
        default = max(1, torch.cuda.get_device_properties(0).multi_processor_count // 2)    # stands for the line

        def run(count, fused, least):
            ctx.set_option(L.OPT_KS_FUSED, fused)
            ctx.set_option(L.OPT_FUSED_MIN, least)
            ins = (L.CtRef * count)(*[L.CtRef((2 * (k % S)) * w, (2 * (k % S) + 1) * w) for k in range(count)])
            d = (L.CtRef * count)(*[L.CtRef(2 * (S + k) * w, (2 * (S + k) + 1) * w) for k in range(count)])
            before = ctx.lib.afhe_kernel_launches()
            L.check(ctx.lib.afhe_eval_rotate_batch(ctx.h, ins, d, count, 1, nq), "rotate")
            return ctx.lib.afhe_kernel_launches() - before, ctx.read_poly(2 * S * w, 2 * count * w)

        for count in counts:
            pipe, want = run(count, 0, default)
            one, got = run(count, 1, 1)
            assert one < pipe and np.array_equal(got, want), count
            rest = count % cap
            launches, got = run(count, 1, default)
            both = pipe + one if count > rest else pipe
            assert launches == (one if rest == 0 or (rest >= line and count > 1) else both), count
            assert np.array_equal(got, want), count

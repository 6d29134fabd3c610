"""Batches that both key switch paths share: whole waves on the one-kernel path,
the remainder on the kernel pipeline.

Rotations by one key, by a key for each entry, and rotations added to the
output, at counts below, at and above the capacity, with the line drawn by level
and by AFHE_OPT_FUSED_MIN: word for word the pipeline's results.
"""
import numpy as np
import pytest

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,levels", [(13, 3), (15, 2)])
def test_shared_batches(log_n, levels):
    p = CkksParams.generate(log_n, levels, 45, 1, 60, 2)
    n, w, S = p.n, levels << log_n, 24
    rng = np.random.default_rng(log_n)
    key = np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(4 * p.dnum) for q in p.q + p.p])
    with FheContext(p, poly_words=(2 * S + 2 * 200) * w, key_words=2 * p.key_words(), max_batch=200) as ctx:
        drv = FHEHostDriver(ctx)
        ctx.write_key(0, key)
        drv.add_rotation_key(1, 0)
        drv.add_rotation_key(2, p.key_words())
        if ctx.get_option(L.OPT_KS_FUSED) != 1:
            pytest.skip("the one-kernel key switch does not run on this GPU at this ring degree")
        cap = ctx.get_option(L.OPT_KS_CAPACITY)
        by_level = max(1, 148 // (2 * (1 << (log_n - 13))))    # the default's value: the line drawn by level
        ctx.write_poly(0, np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2 * S) for q in p.q]))
        start = np.concatenate([rng.integers(0, q, n, dtype=np.uint64) for _ in range(2) for q in p.q])

        def run(kind, count, lv):
            ins = (L.CtRef * count)(*[L.CtRef((2 * (k % S)) * w, (2 * (k % S) + 1) * w) for k in range(count)])
            outs = [(2 * (S + k) * w, (2 * (S + k) + 1) * w) for k in range(count)]
            d = (L.CtRef * count)(*[L.CtRef(*o) for o in outs])
            if kind == "acc":
                for o in outs:
                    ctx.write_poly(o[0], start)
                L.check(ctx.lib.afhe_eval_rotate_accumulate_batch(ctx.h, ins, d, count, 1, lv), "rotate_accumulate")
            elif kind == "steps":
                steps = (L.C.c_int32 * count)(*[1 + k % 2 for k in range(count)])
                L.check(ctx.lib.afhe_eval_rotate_steps_batch(ctx.h, ins, d, steps, count, lv), "rotate_steps")
            else:
                L.check(ctx.lib.afhe_eval_rotate_batch(ctx.h, ins, d, count, 1, lv), "rotate")
            return [ctx.read_poly(x, lv * n) for o in outs for x in o]

        for kind in ("one", "steps", "acc"):
            for lv in (levels, 1):
                for count in sorted({2, cap - 1, cap, min(200, cap + 3), min(200, 3 * cap + 1)}):
                    ctx.set_option(L.OPT_KS_FUSED, 0)
                    want = run(kind, count, lv)
                    ctx.set_option(L.OPT_KS_FUSED, 1)
                    for least in (by_level, 1, 5, cap):
                        ctx.set_option(L.OPT_FUSED_MIN, least)
                        for k, (a, b) in enumerate(zip(want, run(kind, count, lv))):
                            assert np.array_equal(a, b), (kind, lv, count, least, k)

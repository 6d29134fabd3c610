"""Twiddle tables hold second pairs for the primes that read them.

Only primes from 2^50 on (split products) read a second 16-byte pair for each
twiddle: a context's tables grow by those rows alone. Contexts loaded by
OP_LOAD_CONTEXT change between the two kinds in either order: transforms equal
the oracle's.
"""
import numpy as np
import pytest
import torch

from anns_fhe_b200 import _lib as L
from anns_fhe_b200.driver import CkksParams, FheContext, find_ntt_primes
from tests.helpers import AccelImage, uniform_residues

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def taken(p):
    """Device memory that a context takes."""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with FheContext(p, poly_words=1024, key_words=1024, max_batch=1) as ctx:
        ctx.sync()
        return before - torch.cuda.mem_get_info()[0]


def test_second_pairs_of_split_primes_alone():
    log_n, nq, np_ = 16, 14, 2                     # 1 MiB a row
    small = find_ntt_primes(log_n, 49, nq + np_, [])
    large = find_ntt_primes(log_n, 60, nq + np_, [])
    taken(CkksParams(log_n, small[:1], small[1:2], 1))     # (modules loaded)
    none, last, every = (taken(CkksParams(log_n, q, p, nq)) for q, p in
                         ((small[:nq], small[nq:]), (small[:nq], large[nq:]), (large[:nq], large[nq:])))
    # second pairs both ways: 4 and 32 MiB; allocations are whole 2 MiB blocks
    assert last - none <= 12 * MIB
    assert every - none >= 24 * MIB


@pytest.mark.parametrize("order", [(49, 60, 49), (60, 49, 60)])
@pytest.mark.parametrize("log_n", [12, 14])
def test_loaded_contexts_of_either_kind(log_n, order, orc):
    images = {}
    for bits in set(order):
        qs = find_ntt_primes(log_n, bits, 2, [])
        images[bits] = AccelImage(log_n, qs, find_ntt_primes(log_n, bits, 1, qs), 1, 2)
    n, w = 1 << log_n, 2 << log_n
    own = images[order[0]]
    with FheContext(CkksParams(log_n, own.q, own.p, 1), poly_words=2 * w,
                    key_words=max(i.key_words for i in images.values()), max_batch=1) as ctx:
        rng = np.random.default_rng(log_n)
        for bits in order:
            img = images[bits]
            x = uniform_residues(rng, img.q, n)
            ctx.write_key(0, img.key)
            ctx.write_poly(0, x)
            for op, kw in ((L.OP_LOAD_CONTEXT, {}), (L.OP_NTT, dict(src_a_offset=0, dst_offset=w))):
                assert ctx.dispatch(img.args(op, 2, **kw)) == L.OK, ctx.lib.afhe_last_error()
            got = ctx.read_poly(w, w)
            for i, q in enumerate(img.q):
                s = slice(i * n, (i + 1) * n)
                assert np.array_equal(got[s], orc.ntt(x[s], img.tw_q[s], q)), (bits, q)

"""The work a user of this framework has it do, as cases that can be timed.

* one rotation of one ciphertext, at the smallest configuration and at the
  large one (latency: the plain path, one operator after another);
* the batched operators the query chain is made of: rotate-and-sum, rotations
  by a step each (baby steps), ciphertext products with relinearisation and
  rescale, plaintext products with rescale;
* the two batched primitives at N = 2^16: transforms (forward and inverse) and
  rotate-and-sum of ciphertexts at mixed levels;
* both server stages of the diagonal chain, through the native stage driver;
* the client's decryption and decoding of results from host buffers, and the
  server's encoding of plaintexts from host values.

Ring degrees, limb counts and batch sizes are those of the configurations in
anns_fhe_b200/workloads.py, primitives.py and bench.py. Residues (ciphertexts,
keys, evaluation-form plaintexts) are uniform in [0, q), as they are in use.
Key-switch options are the autotuner's cached choices where it has them, as
Workload(tune=True) applies them.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from anns_fhe_b200 import _lib as L
from anns_fhe_b200 import autotune
from anns_fhe_b200.ckks import CkksClient, Encoder, Slots, encode_plaintexts
from anns_fhe_b200.driver import CkksParams, FHEHostDriver, FheContext
from anns_fhe_b200.query import InteractiveQueryManager, QueryShape

# (log N, Q limbs, Q bits, P limbs, P bits, alpha, bits of the first Q prime)
SETS = {
    "small": (13, 3, 50, 1, 60, 1, None),       # the 4,096 x 64 configuration
    "reference": (14, 11, 45, 4, 60, 4, 60),    # the reference kernels' own shape
    "large": (15, 12, 50, 4, 60, 4, None),      # the 1M x 128 configuration
    "wide": (16, 24, 50, 8, 60, 8, None),       # the N = 2^16 primitives
}


def _case(name, kind, params, level, count, **more):
    return dict(name=name, kind=kind, params=params, level=level, count=count, **more)


def listed():
    return [
        # the plain path's operator on the smallest configuration: launches and latency
        _case("rotate_one_N8192", "rotate_one", "small", 3, 1),
        # the same on the large configuration at its full level: one ciphertext over the whole GPU
        _case("rotate_one_N32768_L12", "rotate_one", "large", 12, 1),
        # a tree-sum step of the small configuration's benchmark batch
        _case("rotate_sum_N8192_x296", "rotate_sum", "small", 2, 296),
        # ciphertext products at the reference's shape, three digits, wide first and special primes
        _case("mult_N16384_x32", "mult", "reference", 10, 32),
        # the baby steps of 16 queries: the largest share of the large configuration's step
        _case("baby_steps_N32768_x240", "rotate_steps", "large", 2, 240, steps=15),
        # a tree-sum step at the queries' own level: three digits, an odd count
        _case("rotate_sum_N32768_L11_x45", "rotate_sum", "large", 11, 45),
        # masks and plaintext products of the packed chain: multiply and rescale
        _case("mult_plain_N32768_x100", "mult_plain", "large", 3, 100),
        # batched transforms, both directions
        _case("ntt_N65536_x32", "ntt", "wide", 24, 32),
        # rotate-and-sum of ciphertexts at levels 8 to 24, in one call
        _case("rotate_levels_N65536_x20", "rotate_levels", "wide", 24, 20, low=8),
        # the server's two stages for a group of queries, four queries per list as in the benchmark
        _case("server_N32768_q32", "server", "large", 2, 32, lists=128, probes=16),
        # the client decrypts and decodes a group's results
        _case("decrypt_N32768_x128", "decrypt", "large", 1, 128),
        # the server encodes plaintexts of the packed chain
        _case("encode_N32768_x64", "encode", "large", 3, 64),
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["rotate_one", "rotate_sum", "rotate_steps", "mult", "mult_plain", "ntt", "rotate_levels",
                       "server", "decrypt", "encode"])
    if kind == "rotate_one":
        params = rng.choice(["small", "reference", "large", "wide"])
        return dict(kind=kind, params=params, level=rng.randint(1, SETS[params][1]), count=1)
    if kind in ("rotate_sum", "mult", "mult_plain"):
        params = rng.choice(["small", "reference", "large"])
        level = rng.randint(1 if kind == "rotate_sum" else 2, SETS[params][1])
        most = {"small": 400, "reference": 100, "large": 200}[params]
        return dict(kind=kind, params=params, level=level, count=_spread(rng, 2, max(4, most // level)))
    if kind == "rotate_steps":
        params = rng.choice(["small", "large"])
        steps = rng.choice([3, 7, 15])
        return dict(kind=kind, params=params, level=rng.randint(1, 3), count=steps * _spread(rng, 1, 240 // steps),
                    steps=steps)
    if kind == "ntt":
        params = rng.choice(["small", "reference", "large", "wide"])
        return dict(kind=kind, params=params, level=rng.randint(1, SETS[params][1]), count=_spread(rng, 1, 32))
    if kind == "rotate_levels":
        low = rng.randint(2, 10)
        return dict(kind=kind, params="wide", level=rng.randint(low + 1, 24), count=_spread(rng, 2, 16), low=low)
    if kind == "server":
        lists = rng.choice([40, 64, 100, 128])
        return dict(kind=kind, params="large", level=2, count=_spread(rng, 1, 32), lists=lists,
                    probes=rng.choice([4, 8, 16]))
    if kind == "decrypt":
        params = rng.choice(["small", "large"])
        return dict(kind=kind, params=params, level=1, count=_spread(rng, 1, 128))
    params = rng.choice(["small", "large"])
    return dict(kind="encode", params=params, level=rng.randint(1, 3), count=_spread(rng, 1, 64))


# ---------------------------------------------------------------------------
# what a user's program has in hand before the call
# ---------------------------------------------------------------------------
def _params(case) -> CkksParams:
    log_n, nq, qb, np_, pb, alpha, first = SETS[case["params"]]
    return CkksParams.generate(log_n, nq, qb, np_, pb, alpha, first_bits=first)


class _Arena:
    """A device arena of a context as torch sees it (keeps the context alive)."""

    def __init__(self, ctx, address, words):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (words,), "typestr": "<i8", "version": 3,
                                         "strides": None}


def _poly(ctx):
    return torch.as_tensor(_Arena(ctx, ctx.lib.afhe_poly_gmem(ctx.h), ctx.poly_words), device="cuda")


def _fill(view, primes, gen):
    """Uniform residues: view is (polynomials, limbs, N), limb i below primes[i]."""
    for i, q in enumerate(primes):
        for a in range(0, view.shape[0], 2048):
            part = view[a:a + 2048, i]
            part.copy_(torch.randint(0, q, part.shape, generator=gen, device="cuda", dtype=torch.int64))


def _context(case, p, words, keys, lanes):
    ctx = FheContext(p, poly_words=words, key_words=max(1024, keys * p.key_words()), max_batch=lanes)
    tuned = autotune.load(autotune.cache_path(p), 256 if case["params"] == "large" else 296) or {}
    c = tuned.get(case["level"])
    if c is not None and ctx.get_option(L.OPT_KS_FUSED) == 1:
        ctx.set_option(L.OPT_KS_FUSED, int(c.fused))
        ctx.set_option(L.OPT_CHUNK, min(int(c.chunk), lanes))
        ctx.set_option(L.OPT_KS_EPT, int(c.ept))
        ctx.set_option(L.OPT_KS_SLICE, int(c.slice))
        if c.fused_min:
            ctx.set_option(L.OPT_FUSED_MIN, int(c.fused_min))
    return ctx, tuned


def _keys(ctx, p, gen, steps, relin=False):
    """Uniform evaluation keys, registered for the rotation steps (and relinearisation)."""
    kw, n = p.key_words(), p.n
    mem = torch.as_tensor(_Arena(ctx, ctx.lib.afhe_key_gmem(ctx.h), ctx.key_words), device="cuda")
    count = len(steps) + int(relin)
    _fill(mem[:count * kw].view(count * 2 * p.dnum, p.L + p.K, n), p.q + p.p, gen)
    torch.cuda.synchronize()
    drv = FHEHostDriver(ctx)
    for k, s in enumerate(steps):
        drv.add_rotation_key(s, k * kw)
    if relin:
        drv.set_relin_key(len(steps) * kw)
    return drv


def _refs(first, count, w):
    """`count` ciphertexts back to back from word `first`, w words a polynomial."""
    a = np.arange(2 * count, dtype=np.uint64) * np.uint64(w) + np.uint64(first)
    return (L.CtRef * count).from_buffer_copy(a.tobytes())


def _offsets(values):
    return (L.u64 * len(values))(*[int(v) for v in values])


def prepare(case, seed):
    p = _params(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    s = {"case": case, "p": p}
    globals()["_prepare_" + case["kind"]](case, p, gen, int(seed), s)
    torch.cuda.synchronize()
    return s


def _prepare_rotate_one(case, p, gen, seed, s):
    w = case["level"] * p.n
    s["ctx"], _ = _context(case, p, 4 * w, 1, 1)
    mem = _poly(s["ctx"])
    _fill(mem[:2 * w].view(2, case["level"], p.n), p.q[:case["level"]], gen)
    s["drv"] = _keys(s["ctx"], p, gen, [1])
    s["w"], s["out"] = w, mem[2 * w:].view(2, case["level"], p.n)


def _prepare_rotate_sum(case, p, gen, seed, s):
    n, lv, w = case["count"], case["level"], case["level"] * p.n
    s["ctx"], _ = _context(case, p, 4 * n * w, 1, n)
    mem = _poly(s["ctx"])
    _fill(mem.view(4 * n, lv, p.n), p.q[:lv], gen)
    _keys(s["ctx"], p, gen, [2])
    s["in"], s["acc"] = _refs(0, n, w), _refs(2 * n * w, n, w)
    s["out"] = mem[2 * n * w:].view(n, 2, lv, p.n)


def _prepare_rotate_steps(case, p, gen, seed, s):
    n, lv, k, w = case["count"], case["level"], case["steps"], case["level"] * p.n
    q = n // k
    s["ctx"], _ = _context(case, p, 2 * (q + n) * w, k, min(n, 256))
    mem = _poly(s["ctx"])
    _fill(mem[:2 * q * w].view(2 * q, lv, p.n), p.q[:lv], gen)
    _keys(s["ctx"], p, gen, list(range(1, k + 1)))
    src = _refs(0, q, w)
    s["in"] = (L.CtRef * n)(*[src[i // k] for i in range(n)])
    s["dst"] = _refs(2 * q * w, n, w)
    s["steps"] = (L.i32 * n)(*[1 + i % k for i in range(n)])
    s["out"] = mem[2 * q * w:].view(n, 2, lv, p.n)


def _prepare_mult(case, p, gen, seed, s):
    n, lv, w = case["count"], case["level"], case["level"] * p.n
    wo = (lv - 1) * p.n
    s["ctx"], _ = _context(case, p, 4 * n * w + 2 * n * wo, 1, n)
    mem = _poly(s["ctx"])
    _fill(mem[:4 * n * w].view(4 * n, lv, p.n), p.q[:lv], gen)
    _keys(s["ctx"], p, gen, [], relin=True)
    s["a"], s["b"], s["dst"] = _refs(0, n, w), _refs(2 * n * w, n, w), _refs(4 * n * w, n, wo)
    s["out"] = mem[4 * n * w:].view(n, 2, lv - 1, p.n)


def _prepare_mult_plain(case, p, gen, seed, s):
    n, lv, w = case["count"], case["level"], case["level"] * p.n
    wo = (lv - 1) * p.n
    s["ctx"], _ = _context(case, p, 3 * n * w + 2 * n * wo, 0, n)
    mem = _poly(s["ctx"])
    _fill(mem[:3 * n * w].view(3 * n, lv, p.n), p.q[:lv], gen)
    s["a"], s["pt"] = _refs(0, n, w), _offsets([(2 * n + i) * w for i in range(n)])
    s["dst"] = _refs(3 * n * w, n, wo)
    s["out"] = mem[3 * n * w:].view(n, 2, lv - 1, p.n)


def _prepare_ntt(case, p, gen, seed, s):
    n, lv, w = case["count"], case["level"], case["level"] * p.n
    s["ctx"], _ = _context(case, p, 2 * n * w, 0, 1)
    mem = _poly(s["ctx"])
    _fill(mem.view(2 * n, lv, p.n), p.q[:lv], gen)
    s["fwd"], s["inv"] = _offsets([i * w for i in range(n)]), _offsets([(n + i) * w for i in range(n)])
    s["out"] = mem.view(2, n, lv, p.n)


def _prepare_rotate_levels(case, p, gen, seed, s):
    n, top, w = case["count"], case["level"], case["level"] * p.n
    rng = np.random.default_rng([case["low"], top, n])       # the levels belong to the case
    levels = rng.integers(case["low"], top + 1, n)
    s["ctx"], _ = _context(case, p, 4 * n * w, 1, n)
    mem = _poly(s["ctx"])
    _fill(mem.view(4 * n, top, p.n), p.q[:top], gen)
    _keys(s["ctx"], p, gen, [4])
    s["in"], s["acc"] = _refs(0, n, w), _refs(2 * n * w, n, w)
    s["levels"] = (C.c_uint32 * n)(*[int(x) for x in levels])
    s["out"] = mem[2 * n * w:].view(n, 2, top, p.n)


def _unit_counts(case):
    """Vectors per list: about a thousand, as the large configuration's index has them."""
    rng = np.random.default_rng([case["lists"], 17])
    return rng.integers(700, 1250, case["lists"]).astype(np.uint32)


def _probes(case):
    """Each query's lists; popular lists are probed by several queries."""
    rng = np.random.default_rng([case["lists"], case["probes"], case["count"]])
    return np.stack([rng.permutation(case["lists"])[:case["probes"]] for _ in range(case["count"])]).astype(np.uint32)


def _prepare_server(case, p, gen, seed, s):
    D, lv, nq, lists, n = 128, case["level"], case["count"], case["lists"], p.n
    sh = QueryShape(D=D, n_list=lists, slots=n // 2, nprobe=case["probes"], top_k=8, scale=2.0 ** 40,
                    compaction="diagonal", eval_level=lv)
    lanes, w, w1 = 128, lv * n, (lv - 1) * n
    pool = InteractiveQueryManager.inner_pool(lanes, sh.n2)
    counts = _unit_counts(case)
    most = max(int(np.sum(-(-counts[pr].astype(np.int64) // D) * D)) for pr in _probes(case))
    n_res = -(-most // sh.slots) + 1
    nb = sh.n1 - 1
    # regions in words: queries, norms, diagonals (centroids first), norms, baby steps, pool, results
    at, regions = 0, {}
    for name, words in (("query", 2 * nq * w), ("dim", 2 * nq * w1), ("diag", (1 + lists) * D * w),
                        ("unorm", (1 + lists) * w1), ("baby", 2 * nq * nb * w), ("pool", 2 * pool * w),
                        ("compact", 2 * nq * w1), ("result", 2 * nq * n_res * w1)):
        regions[name] = at
        at += words
    steps = list(range(1, sh.n1)) + [sh.n1 * g for g in range(1, sh.n2)]
    ctx, tuned = _context(case, p, at, len(steps), lanes)
    s["ctx"] = ctx
    mem = _poly(ctx)

    def part(name, polys, limbs):
        return mem[regions[name]:regions[name] + polys * limbs * n].view(polys, limbs, n)
    _fill(part("query", 2 * nq, lv), p.q[:lv], gen)
    _fill(part("dim", 2 * nq, lv - 1), p.q[:lv - 1], gen)
    _fill(part("diag", (1 + lists) * D, lv), p.q[:lv], gen)
    _fill(part("unorm", 1 + lists, lv - 1), p.q[:lv - 1], gen)
    _keys(ctx, p, gen, steps)
    lib, h = ctx.lib, C.c_void_p()
    shape = L.IvfpqShape(D, lists, n // 2, lanes, 2, lv)
    L.check(lib.afhe_ivfpq_create(ctx.h, C.byref(shape), C.byref(h)), "ivfpq_create")
    first = np.arange(lists + 1, dtype=np.uint32)
    L.check(lib.afhe_ivfpq_set_units(h, first.ctypes.data_as(L.P32), counts.ctypes.data_as(L.P32), lists),
            "ivfpq_set_units")
    pts = _offsets([regions["diag"] + (1 + u) * D * w for u in range(lists)])
    norms = _offsets([regions["unorm"] + (1 + u) * w1 for u in range(lists)])
    L.check(lib.afhe_ivfpq_set_diagonals(h, lv, regions["diag"], regions["unorm"], pts, norms, lists),
            "ivfpq_set_diagonals")
    L.check(lib.afhe_ivfpq_set_scratch(h, _refs(regions["pool"], pool, w), pool), "ivfpq_set_scratch")
    for level, c in tuned.items():
        o = L.KsOptions(int(c.fused), min(int(c.chunk), lanes), int(c.ept), int(c.slice), int(c.fused_min))
        L.check(lib.afhe_ivfpq_set_tuning(h, level, C.byref(o)), "ivfpq_set_tuning")
    queries = (L.IvfpqQuery * nq)()
    keep = []
    for i, pr in enumerate(_probes(case)):
        q = queries[i]
        q.ct_query = _refs(regions["query"] + 2 * i * w, 1, w)[0]
        q.ct_dim = _refs(regions["dim"] + 2 * i * w1, 1, w1)[0]
        q.compact = _refs(regions["compact"] + 2 * i * w1, 1, w1)[0]
        res, baby = _refs(regions["result"] + 2 * i * n_res * w1, n_res, w1), _refs(regions["baby"] + 2 * i * nb * w, nb, w)
        probes = (C.c_uint32 * len(pr))(*[int(x) for x in pr])
        keep += [res, baby, probes]
        q.results, q.n_results, q.level = C.cast(res, C.POINTER(L.CtRef)), n_res, p.L
        q.probes, q.nprobe = C.cast(probes, L.P32), len(pr)
        q.baby, q.n_baby = C.cast(baby, C.POINTER(L.CtRef)), nb
    s.update(handle=h, queries=queries, keep=keep,
             out=(part("compact", 2 * nq, lv - 1), part("result", 2 * nq * n_res, lv - 1)))


def _coefficients(case, n, seed):
    """Integer coefficients of the messages a client decrypts: a slot is then of the order of 100."""
    return np.rint(np.random.default_rng(seed).normal(0.0, 2.0 ** 30, (case["count"], n)))


SCALE = 2.0 ** 30      # of a result: Delta^2 / q at Delta = 2^40


def _prepare_decrypt(case, p, gen, seed, s):
    n, count, q = p.n, case["count"], p.q[0]
    words = 8 * (p.L + p.K) * n
    ctx = FheContext(p, poly_words=words + 4 * count * n, key_words=1024, max_batch=1)
    client = CkksClient(ctx, Slots(p, 0, words), seed=seed)
    mem = _poly(ctx)[words:].view(4, count, n)
    m = torch.from_numpy(_coefficients(case, n, seed).astype(np.int64))
    mem[0].copy_(torch.remainder(m, q))
    _fill(mem[1][:, None], [q], gen)                          # c1
    torch.cuda.synchronize()
    polys = _offsets([words + i * n for i in range(count)])
    L.check(ctx.lib.afhe_ntt_batch(ctx.h, polys, count, 1, 0), "ntt_batch")
    for i in range(count):                                    # c0 = m - c1 s
        a = words + i * n
        client.drv.poly_mul_ntt(a + count * n, client.s_slot, a + 2 * count * n, 1)
        client.drv.poly_sub(a, a + 2 * count * n, a + 3 * count * n, 1)
    ctx.sync()
    host = torch.empty((count, 2, n), dtype=torch.int64, pin_memory=True)
    host[:, 0].copy_(mem[3])
    host[:, 1].copy_(mem[1])
    s["decryptor"] = client.decryptor(count)
    s["host"], s["cts"] = host, host.numpy().view(np.uint64)
    s["scales"] = np.full(count, SCALE)
    ctx.close()


def _prepare_encode(case, p, gen, seed, s):
    n, count, w = p.n, case["count"], case["level"] * p.n
    s["ctx"], _ = _context(case, p, count * w, 0, 1)
    s["enc"] = Encoder(p.log_n)
    values = torch.empty((count, n // 2), dtype=torch.float64, pin_memory=True)
    values.copy_(torch.from_numpy(np.random.default_rng(seed).normal(0.0, 1.0, (count, n // 2))))
    s["host"], s["values"] = values, values.numpy()
    s["offs"] = np.arange(count, dtype=np.uint64) * np.uint64(w)
    s["out"] = _poly(s["ctx"]).view(count, case["level"], n)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _Held(np.ndarray):
    """A view of a decryptor's page-locked results that keeps the decryptor alive."""
    owner = None


def run(s):
    case = s["case"]
    kind, lv, n = case["kind"], case["level"], case["count"]
    if kind == "decrypt":
        slots = s["decryptor"].decrypt_decode_host(s["cts"], s["scales"], s["p"].n // 2).view(_Held)
        slots.owner = s["decryptor"]
        return slots
    ctx = s["ctx"]
    lib, h = ctx.lib, ctx.h
    if kind == "rotate_one":
        w = s["w"]
        s["drv"].eval_rotate_single_step(0, w, 2 * w, 3 * w, 1, lv)
    elif kind == "rotate_sum":
        L.check(lib.afhe_eval_rotate_accumulate_batch(h, s["in"], s["acc"], n, 2, lv), "rotate_accumulate_batch")
    elif kind == "rotate_steps":
        L.check(lib.afhe_eval_rotate_steps_batch(h, s["in"], s["dst"], s["steps"], n, lv), "rotate_steps_batch")
    elif kind == "mult":
        L.check(lib.afhe_eval_mult_relin_rescale_batch(h, s["a"], s["b"], s["dst"], n, lv), "mult_relin_rescale_batch")
    elif kind == "mult_plain":
        L.check(lib.afhe_eval_mult_plain_rescale_batch(h, s["a"], s["pt"], s["dst"], n, lv),
                "mult_plain_rescale_batch")
    elif kind == "ntt":
        L.check(lib.afhe_ntt_batch(h, s["fwd"], n, lv, 0), "ntt_batch")
        L.check(lib.afhe_ntt_batch(h, s["inv"], n, lv, 1), "ntt_batch")
    elif kind == "rotate_levels":
        L.check(lib.afhe_eval_rotate_accumulate_levels_batch(h, s["in"], s["acc"], s["levels"], n, 4),
                "rotate_accumulate_levels_batch")
    elif kind == "server":
        L.check(lib.afhe_ivfpq_stage1(s["handle"], s["queries"], n), "ivfpq_stage1")
        L.check(lib.afhe_ivfpq_stage3(s["handle"], s["queries"], n), "ivfpq_stage3")
    else:
        encode_plaintexts(ctx, s["enc"], s["values"], 2.0 ** 40, s["offs"], lv)
    return s["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _transform_ops(n):
    """A transform of one limb: N/2 log N butterflies of a product, a sum and a difference."""
    return n // 2 * (n.bit_length() - 1) * 3


def _key_switch(p, lv):
    """(operations, key bytes) of one key switch: the transforms of the hybrid
    method (each limb once to coefficients, the digits' other primes forward,
    both sums back over the special primes and forward over the limbs), the
    base conversions and the inner product, a product and a sum each."""
    n, parts = p.n, -(-lv // p.alpha)
    digits = [min(p.alpha, lv - j * p.alpha) for j in range(parts)]
    up = sum(lv - d + p.K for d in digits)
    transforms = lv + up + 2 * p.K + 2 * lv
    conv = sum(d * (lv - d + p.K) for d in digits) + 2 * p.K * lv
    ops = transforms * _transform_ops(n) + 2 * n * (conv + 2 * parts * (lv + p.K) + 4 * lv)
    return ops, 2 * parts * (lv + p.K) * n * 8


def _rescale_ops(p, lv):
    return 2 * lv * _transform_ops(p.n) + 2 * 2 * (lv - 1) * p.n


def work(case):
    p = _params(case)
    n, lv, c, kind = p.n, case["level"], case["count"], case["kind"]
    limb = n * 8
    ks, key = _key_switch(p, lv)
    if kind == "rotate_one":
        return {"bytes": 4 * lv * limb + key, "flops": ks}
    if kind == "rotate_sum":
        return {"bytes": c * 6 * lv * limb + key, "flops": c * ks}
    if kind == "rotate_steps":
        return {"bytes": (c // case["steps"] + c) * 2 * lv * limb + case["steps"] * key, "flops": c * ks}
    if kind == "mult":
        return {"bytes": c * (4 * lv + 2 * (lv - 1)) * limb + key,
                "flops": c * (ks + _rescale_ops(p, lv) + 10 * lv * n)}
    if kind == "mult_plain":
        return {"bytes": c * (3 * lv + 2 * (lv - 1)) * limb, "flops": c * (_rescale_ops(p, lv) + 4 * lv * n)}
    if kind == "ntt":
        return {"bytes": 4 * c * lv * limb, "flops": 2 * c * lv * _transform_ops(n)}
    if kind == "rotate_levels":
        levels = np.random.default_rng([case["low"], lv, c]).integers(case["low"], lv + 1, c)
        return {"bytes": sum(6 * int(x) * limb for x in levels) + key,
                "flops": sum(_key_switch(p, int(x))[0] for x in levels)}
    if kind == "server":
        D, n1, n2 = 128, 16, 8
        probes, counts = _probes(case), _unit_counts(case).astype(np.int64)
        units = len(np.unique(probes))
        results = sum(-(-int(np.sum(-(-counts[pr] // D) * D)) // (n // 2)) for pr in probes)
        outs = c + results
        ks1, key1 = _key_switch(p, lv - 1)
        products = (probes.size + c) * D * lv * 2 * n
        return {"bytes": c * 2 * lv * limb + c * 2 * limb + (1 + units) * (D * lv + lv - 1) * limb
                + outs * 2 * (lv - 1) * limb + (n1 - 1) * key + (n2 - 1) * key1,
                "flops": c * (n1 - 1) * ks + outs * ((n2 - 1) * ks1 + n2 * _rescale_ops(p, lv)) + 2 * products}
    if kind == "decrypt":
        return {"bytes": c * (2 * limb + n // 2 * 8), "flops": c * (_transform_ops(n) + 2 * n + 5 * n * p.log_n)}
    return {"bytes": c * (n // 2 * 8 + lv * limb), "flops": c * (lv * _transform_ops(n) + 5 * n * p.log_n)}


def exact(case, seed):
    """Decoded slots in 64 bits; residues are whole numbers and have to be equal."""
    if case["kind"] != "decrypt":
        return None
    n = 1 << SETS[case["params"]][0]
    k = np.arange(n)
    twist = np.exp(1j * np.pi * k / n)
    power, where = 1, np.empty(n // 2, dtype=np.int64)
    for j in range(n // 2):                                   # slot j is the value at the root of exponent 5^j
        where[j] = (power - 1) // 2
        power = power * 5 % (2 * n)
    return np.stack([(np.fft.ifft(row * twist) * n)[where].real / SCALE
                     for row in _coefficients(case, n, int(seed))])

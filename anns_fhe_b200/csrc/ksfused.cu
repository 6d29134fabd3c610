// ksfused.cu -- host side of the one-kernel key switch (ksfused.cuh): prepared
// keys, capacity, dispatch.
#include <map>
#include <mutex>

#include "ksfused.cuh"

namespace afhe {

namespace {

// The prepared copy of a key (evk_a digits, then evk_b digits; word w belongs
// to digit (w / nS) mod dnum, limb slot (w / n) mod S): pairs as KeyMul reads
// them, (k centred, k / q) as doubles for q < 2^50, else (k mod q, Shoup
// companion). A limb in its own digit (limbs [j alpha, (j + 1) alpha) of digit
// j) keeps its order; the others are read eight adjacent values per thread, so
// value 8 t + e of a slice of 2^LOGQ lies at e T + t.
__global__ void key_prep_kernel(const u64* __restrict__ key, ulonglong2* __restrict__ prep,
                                const PrimeConst* __restrict__ pc, int log_n, uint32_t L, uint32_t S, uint32_t dnum,
                                uint32_t alpha, int logq, u64 words) {
    const uint32_t qn = 1u << logq;
    for (u64 w = blockIdx.x * (u64)blockDim.x + threadIdx.x; w < words; w += (u64)gridDim.x * blockDim.x) {
        const u64 row = w >> log_n;
        const uint32_t slot = (uint32_t)(row % S), digit = (uint32_t)((row / S) % dnum);
        const u64 q = pc[slot].q;
        const u64 k = key[w] % q;
        ulonglong2 v;
        if (q < kFpLimit) {
            u64 o[4];
            transform_constant(k, q, o);
            v = make_ulonglong2(o[0], o[1]);
        } else {
            v = make_ulonglong2(k, shoup_companion(k, q));
        }
        u64 at = w;
        if (!(slot < L && slot / alpha == digit)) {
            const uint32_t x = (uint32_t)(w & (qn - 1));
            at = (w & ~(u64)(qn - 1)) + (x & 7) * (qn / 8) + x / 8;
        }
        prep[at] = v;
    }
}

}  // namespace

// The occupancy queries behind the capacity cost tens of microseconds, and
// the options that consult them are set around every batched operator, so the
// answers are kept per (device, N).
int key_switch_fused_capacity(int log_n) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, int> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const auto key = std::make_pair(dev, log_n);
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    const int cap = ksf::capacity(log_n);
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = cap;
    return cap;
}

bool key_switch_fused_supported(int log_n) { return key_switch_fused_capacity(log_n) > 0; }

size_t ks_fused_scratch_words(uint32_t n, uint32_t sizeQl, uint32_t K) { return (size_t)n * (sizeQl + 2 * K); }

cudaError_t launch_key_prep(const u64* key, ulonglong2* prep, const PrimeConst* pc, int log_n, uint32_t L, uint32_t S,
                            uint32_t dnum, uint32_t alpha, u64 words, cudaStream_t st) {
    if (words == 0) return cudaSuccess;
    u64 blocks = (words + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    key_prep_kernel<<<(unsigned)blocks, 256, 0, st>>>(key, prep, pc, log_n, L, S, dnum, alpha, ksf::slice_bits(log_n), words);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_key_switch_fused(int log_n, const OpTabs* lvtabs, uint32_t alpha, uint32_t sizeQl, uint32_t K, const u64* key, u64 evk_a,
                                    u64 evk_b, uint32_t key_stride, uint32_t key_pbase, u64* arena, u64* scratch,
                                    uint32_t nz, const ZBases& zb, cudaStream_t st, const KsFuse* fuse,
                                    const ulonglong2* prep, const ZField* lvz) {
    if (nz == 0) return cudaSuccess;
    ksf::KsFusedArgs a{};
    a.lvtabs = lvtabs;
    a.sizeQl = sizeQl;
    a.K = K;
    a.key = key;
    a.evk_a = evk_a;
    a.evk_b = evk_b;
    a.key_stride = key_stride;
    a.key_pbase = key_pbase;
    a.arena = arena;
    a.scratch = scratch;
    a.in = zb.src;
    a.out0 = zb.out;
    a.out1 = zb.aux;
    a.mid = zb.mid;
    if (fuse) a.f = *fuse;
    a.prep = prep;
    a.prep_b = evk_b - evk_a;
    if (lvz) {
        a.mixed = 1;
        a.lvz = *lvz;
    }
    if (!a.prep) return ksf::launch_raw(log_n, a, nz, st);
    return sizeQl <= alpha ? ksf::launch_single(log_n, a, nz, st)       // (sizeQl is the largest level)
                           : ksf::launch_multi(log_n, a, nz, st);
}

}  // namespace afhe

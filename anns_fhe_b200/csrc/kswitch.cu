// kswitch.cu -- the hybrid key switch as a pipeline of kernels
// (hardware_fpga_model/hls/src/key_switch.cpp:167-439): INTT of the input,
// base conversion fused into the ModUp NTTs' loads, inner product with the
// key, ModDown (kswitch_down.cu).
#include "internal.h"

namespace afhe {

// ---------------------------------------------------------------------------
// key switch (key_switch.cpp:167-439)
// ---------------------------------------------------------------------------
// Scratch layout per polynomial (S = slots_q + K limb slots, Q limb i at slot
// i, special limb k at slot slots_q + k):
//   coef   : slots_q * N   INTT of the input's Q limbs, times qHatInv (ModUp's first factor)
//   modup  : parts * S * N digit j's complementary limbs, evaluation form
//   ext0   : S * N         sum_j digit_j * evk_b   (then ModDown input)
//   ext1   : S * N         sum_j digit_j * evk_a
//   mid    : 2 * slots_q * N  two-pass intermediates of the ModDown NTTs
//   t0     : slots_q * N   c0 gathered through the automorphism (rotation)
size_t ks_scratch_words(uint32_t n, uint32_t slots_q, uint32_t K, uint32_t parts) {
    const size_t S = slots_q + K;
    return (size_t)n * (slots_q + parts * S + 2 * S + 3 * (size_t)slots_q);
}

// Input load through the automorphism: the key switch of auto(c1) reads
// c1[map[x]] (the reference applies automorphism() first, fhe_host_driver.cpp:342-350).
struct LoadGather {
    const u64* base;
    const uint32_t* map;
    ZField mapz;        // per-entry map addresses (per_z)
    int per_z;
    __device__ __forceinline__ u64 operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x,
                                              const PrimeConst&) const {
        const uint32_t* m = per_z ? (const uint32_t*)mapz.at(z) : map;
        return base[zb.src.at(z) + j.src + __ldg(m + x)];
    }
};

// Epilogue of the input's INTT: stores y_i = [x_i * qHatInv_i]_{q_i}, the
// first factor of ModUp's base conversion (key_switch.cpp:7-60), once per
// input limb instead of once per complementary output limb. job.aux = Q limb i.
struct StoreQhatInv {
    u64* scratch;
    OpTabs t;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst& pc) const {
        const uint32_t part = j.aux / t.alpha, idx = j.aux - part * t.alpha;
        scratch[zb.out.at(z) + j.out + x] =
            mul_shoup(v, __ldg(t.qhat_inv[part] + idx), __ldg(t.qhat_inv_sh[part] + idx), pc.q);
    }
};

// ModUp base conversion as the NTT prologue: job.aux = digit << 16 | k, where
// k is the output's position among the digit's complementary primes. Reads
// y_i = [x_i * qHatInv_i]_{q_i} (StoreQhatInv) and sums y_i * [qHat_i]_p.
struct ModUpLoad {
    const u64* scratch;   // coef region at zb.aux[z]
    OpTabs t;
    uint32_t K;
    uint32_t n;
    __device__ __forceinline__ u64 operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x,
                                              const PrimeConst& pc) const {
        const uint32_t part = j.aux >> 16, k = j.aux & 0xFFFFu;
        const uint32_t start = part * t.alpha;
        const uint32_t size = (part == t.parts - 1) ? t.sizeQl - start : t.alpha;
        const uint32_t row = t.sizeQl - size + K;   // complementary primes of this digit
        const u64 p = pc.q, p2 = p << 1;
        const u64* qm = t.qhat_modp[part];
        const u64* qmsh = t.qhat_modp_sh[part];
        u64 s = 0;
        for (uint32_t i = 0; i < size; ++i) {
            const uint32_t limb = start + i;
            const u64 y = scratch[zb.aux.at(z) + (u64)limb * n + x];            // [x * qHatInv]_{q_i}
            u64 w = mul_shoup_lazy(y, __ldg(qm + i * row + k), __ldg(qmsh + i * row + k), p);
            s += w;
            s = s >= p2 ? s - p2 : s;
        }
        return csub(s, p);
    }
};

struct StoreSlot {   // plain store into scratch
    u64* scratch;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst&) const {
        scratch[zb.out.at(z) + j.out + x] = v;
    }
};

// Inner product with the evaluation key. One thread per (slot, coefficient).
// slot s < sizeQl is Q limb s, slot slots_q + k is special limb k.
__global__ void __launch_bounds__(256) ks_mac_kernel(OpTabs t, uint32_t n, uint32_t slots_q, uint32_t sizeQl,
                                                     uint32_t K, const u64* __restrict__ key, u64 evk_a, u64 evk_b,
                                                     uint32_t key_stride, uint32_t key_pbase,
                                                     const u64* __restrict__ arena, u64* __restrict__ scratch,
                                                     u64 modup_off, u64 ext0_off, u64 ext1_off, u64 t0_off,
                                                     const ZBases zb, const KsFuse f) {
    const uint32_t sidx = blockIdx.y;   // 0..sizeQl+K-1
    const uint32_t z = blockIdx.z;
    const bool isq = sidx < sizeQl;
    const uint32_t slot = isq ? sidx : slots_q + (sidx - sizeQl);
    const uint32_t prime = isq ? sidx : t.p_base + (sidx - sizeQl);
    const uint32_t klimb_in_digit = isq ? sidx : key_pbase + (sidx - sizeQl);
    const PrimeConst pc = t.pt.pc[prime];
    const ModConst mc = modconst_of(pc);
    const u64 S = (u64)slots_q + K;
    const u64 base_scr = zb.mid.at(z);
    const u64* in = arena + zb.src.at(z) + (u64)sidx * n;   // only valid for Q limbs
    const u64 c0_off = f.has_c0 ? f.c0.at(z) : 0;
    const uint32_t* map = f.per_z ? (const uint32_t*)f.mapz.at(z) : f.map;
    const u64 koff = f.per_z ? f.keyz.at(z) : 0;           // this entry's key (per_z)
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
        const uint32_t xs = map ? __ldg(map + x) : x;         // position read through the automorphism
        if (isq && f.has_c0)
            scratch[base_scr + t0_off + (u64)sidx * n + x] = arena[c0_off + (u64)sidx * n + xs];
        Acc128 ab, aa;
        acc_init(ab);
        acc_init(aa);
        for (uint32_t part = 0; part < t.parts; ++part) {
            const uint32_t start = part * t.alpha;
            const uint32_t size = (part == t.parts - 1) ? sizeQl - start : t.alpha;
            u64 d;
            if (isq && sidx >= start && sidx < start + size) d = in[xs];
            else d = scratch[base_scr + modup_off + ((u64)part * S + slot) * n + x];
            const u64 kl = koff + ((u64)part * key_stride + klimb_in_digit) * n + x;
            acc_mad(ab, d, __ldg(key + evk_b + kl));
            acc_mad(aa, d, __ldg(key + evk_a + kl));
        }
        scratch[base_scr + ext0_off + (u64)slot * n + x] = acc_reduce(ab, mc);
        scratch[base_scr + ext1_off + (u64)slot * n + x] = acc_reduce(aa, mc);
    }
}

cudaError_t launch_ks_moddown(int log_n, const OpTabs& t, const LimbJob* jobs_qp, uint32_t slots_q, uint32_t sizeQl,
                              uint32_t K, u64* arena, u64* scratch, uint32_t nz, const ZBases& zb, const KsFuse& f,
                              u64 off_ext0, u64 off_ext1, u64 off_mid, u64 off_t0, cudaStream_t st);   // kswitch_down.cu

cudaError_t launch_key_switch(int log_n, const OpTabs& t, const LimbJob* jobs_qp, const LimbJob* jobs_modup,
                              uint32_t n_modup, uint32_t slots_q, uint32_t sizeQl, uint32_t K, const u64* key,
                              u64 evk_a, u64 evk_b, uint32_t key_stride, uint32_t key_pbase, u64* arena,
                              u64* scratch, uint32_t nz, const ZBases& zb, cudaStream_t st, const KsFuse* fuse) {
    if (nz == 0) return cudaSuccess;
    if (2ull * nz > 65535ull) return cudaErrorInvalidValue;
    KsFuse f{};
    if (fuse) f = *fuse;
    const u64 n = 1ull << log_n;
    const u64 S = (u64)slots_q + K;
    const u64 off_coef = 0;
    const u64 off_modup = off_coef + (u64)slots_q * n;
    const u64 off_ext0 = off_modup + (u64)t.parts * S * n;
    const u64 off_ext1 = off_ext0 + S * n;
    const u64 off_mid = off_ext1 + S * n;
    const u64 off_t0 = off_mid + 2ull * slots_q * n;
    cudaError_t e;

    // 1. INTT of the input's Q limbs -> coef (slot i at coef + i*N)
    {
        ZBases a = zb;
        a.mid = zf_plus(zb.mid, off_coef);
        a.out = a.mid;
        if (f.map || f.per_z)
            e = launch_ntt<true>(log_n, t.pt, jobs_qp, sizeQl, nz, scratch, a,
                                 LoadGather{arena, f.map, f.mapz, f.per_z}, StoreQhatInv{scratch, t}, st);
        else
            e = launch_ntt<true>(log_n, t.pt, jobs_qp, sizeQl, nz, scratch, a, LoadPlain{arena},
                                 StoreQhatInv{scratch, t}, st);
        if (e != cudaSuccess) return e;
    }
    // 2. ModUp: base conversion + NTT for every (digit, complementary limb)
    {
        ZBases a = zb;
        a.aux = zf_plus(zb.mid, off_coef);
        a.mid = zf_plus(zb.mid, off_modup);
        a.out = a.mid;
        ModUpLoad pro{scratch, t, K, (uint32_t)n};
        e = launch_ntt<false>(log_n, t.pt, jobs_modup, n_modup, nz, scratch, a, pro, StoreSlot{scratch}, st);
        if (e != cudaSuccess) return e;
    }
    // 3. inner product with the key
    {
        dim3 grid((uint32_t)((n + 255) / 256), sizeQl + K, nz);
        ks_mac_kernel<<<grid, 256, 0, st>>>(t, (uint32_t)n, slots_q, sizeQl, K, key, evk_a, evk_b, key_stride,
                                            key_pbase, arena, scratch, off_modup, off_ext0, off_ext1, off_t0, zb, f);
        count_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // 4. ModDown of both accumulators
    return launch_ks_moddown(log_n, t, jobs_qp, slots_q, sizeQl, K, arena, scratch, nz, zb, f, off_ext0, off_ext1,
                             off_mid, off_t0, st);
}

}  // namespace afhe

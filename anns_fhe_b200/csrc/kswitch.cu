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
    static constexpr bool kMany = false;
    static constexpr bool kWords = true;
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
        scratch[zb.out.at(z) + j.out + x] = mul_tc(v, t.qhat_inv_tc[part] + 4ull * idx, pc);
    }
};

// ModUp base conversion as the NTT prologue: job.aux = digit << 16 | k, where
// k is the output's position among the digit's complementary primes. Reads
// y_i = [x_i * qHatInv_i]_{q_i} (StoreQhatInv) and sums y_i * [qHat_i]_p.
struct ModUpLoad {
    static constexpr bool kMany = true;
    static constexpr bool kWords = false;
    const u64* scratch;   // coef region at zb.aux[z]
    OpTabs t;
    uint32_t K;
    uint32_t n;
    template <int M>
    __device__ __forceinline__ void many(u64* o, const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 step,
                                         const PrimeConst& pc) const {
        const uint32_t part = j.aux >> 16, k = j.aux & 0xFFFFu;
        const uint32_t start = part * t.alpha;
        const uint32_t size = (part == t.parts - 1) ? t.sizeQl - start : t.alpha;
        const u64* const y = scratch + zb.aux.at(z) + (u64)start * n + x;     // [x * qHatInv]_{q_i}
        bconv<M>(o, size, t.qhat_modp_sp[part] + 4ull * k, t.sizeQl - size + K, pc.q,
                 [&](uint32_t i, uint32_t e) { return y[(u64)i * n + e * step]; });
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
// slot s < sizeQl is Q limb s, slot slots_q + k is special limb k. The operands
// of up to four digits are on their way before the first is used; products of
// residues of primes below 2^50 in doubles, else (also where a key's word is no
// residue) summed in 128 bits and reduced once.
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
        double fb = 0, fa = 0;
        bool words = !pc.fp;                    // something in ab, aa
        constexpr uint32_t D = 4;
        for (uint32_t part0 = 0; part0 < t.parts; part0 += D) {
            u64 d[D], kb[D], ka[D];
#pragma unroll
            for (uint32_t e = 0; e < D; ++e) {
                const uint32_t part = part0 + e;
                if (part >= t.parts) {
                    d[e] = kb[e] = ka[e] = 0;
                    continue;
                }
                const uint32_t start = part * t.alpha;
                const uint32_t size = (part == t.parts - 1) ? sizeQl - start : t.alpha;
                const bool own = isq && sidx >= start && sidx < start + size;
                const u64* const from = own ? in + xs : scratch + base_scr + modup_off + ((u64)part * S + slot) * n + x;
                const u64 kl = koff + ((u64)part * key_stride + klimb_in_digit) * n + x;
                d[e] = *from;
                kb[e] = __ldg(key + evk_b + kl);
                ka[e] = __ldg(key + evk_a + kl);
            }
#pragma unroll
            for (uint32_t e = 0; e < D; ++e) {
                if (part0 + e >= t.parts) break;
                if (pc.fp && d[e] < pc.q && kb[e] < pc.q && ka[e] < pc.q) {
                    const double f = fp_of(d[e]);
                    fb = fp_center(__dadd_rn(fb, fp_mul2(f, fp_of(kb[e]), pc.qd, pc.qi)), pc.qd, pc.qi);
                    fa = fp_center(__dadd_rn(fa, fp_mul2(f, fp_of(ka[e]), pc.qd, pc.qi)), pc.qd, pc.qi);
                } else {
                    words = true;
                    acc_mad(ab, d[e], kb[e]);
                    acc_mad(aa, d[e], ka[e]);
                }
            }
        }
        u64 r0 = pc.fp ? fp_canon(fb, pc.qd) : 0, r1 = pc.fp ? fp_canon(fa, pc.qd) : 0;
        if (words) {
            r0 = add_mod(r0, acc_reduce(ab, mc), pc.q);
            r1 = add_mod(r1, acc_reduce(aa, mc), pc.q);
        }
        scratch[base_scr + ext0_off + (u64)slot * n + x] = r0;
        scratch[base_scr + ext1_off + (u64)slot * n + x] = r1;
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

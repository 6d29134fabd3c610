// kswitch_down.cu -- approx_mod_down of the kernel pipeline's key switch
// (hardware_fpga_model/hls/src/key_switch.cpp:62-163): z' = 2z (ext0 -> ks0),
// 2z + 1 (ext1 -> ks1).
#include "internal.h"

namespace afhe {

// Epilogue of the special limbs' INTT before ModDown: stores
// [x_k * PHatInv_k]_{p_k}, the first factor of the P -> Q base conversion
// (key_switch.cpp:62-163), once per special limb. job.aux = special limb k.
struct StorePhatInv {
    u64* scratch;
    OpTabs t;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst& pc) const {
        scratch[zb.out.at(z) + j.out + x] = mul_tc(v, t.phat_inv_tc + 4ull * j.aux, pc);
    }
};

// ModDown base conversion P -> Q as the NTT prologue (job = Q limb i). Reads
// [x_k * PHatInv_k]_{p_k} (StorePhatInv) and sums it times [PHat_k]_{q_i}.
struct ModDownLoad {
    static constexpr bool kMany = true;
    static constexpr bool kWords = false;
    const u64* scratch;  // ext region at zb.aux[z]
    OpTabs t;
    uint32_t slots_q, K, n;
    template <int M>
    __device__ __forceinline__ void many(u64* o, const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 step,
                                         const PrimeConst& pc) const {
        const u64* const y = scratch + zb.aux.at(z) + (u64)slots_q * n + x;
        bconv<M>(o, K, t.phat_modq_sp + 4ull * j.aux, t.sizeQl, pc.q,
                 [&](uint32_t k, uint32_t e) { return y[(u64)k * n + e * step]; });
    }
};

// ModDown combine as the NTT epilogue: out = (x_Q - y) * P^-1 mod q_i.
// z' = 2z + h: h = 0 writes ks0 (+ gathered c0, + acc0), h = 1 writes ks1 (+ acc1).
struct ModDownStore {
    const u64* scratch;  // ext region at zb.src(z)
    u64* arena;          // outputs
    OpTabs t;
    uint32_t n;
    int has_c0, has_acc;
    ZField t0;           // scratch offset of the gathered c0, per ciphertext
    ZField out0, out1;   // ks0 / ks1 destinations, per ciphertext
    ZField acc0, acc1;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst& pc) const {
        const u64 q = pc.q;
        const uint32_t i = j.aux;
        const uint32_t h = z & 1u, zc = z >> 1;
        const u64 li = (u64)i * n + x;
        u64 xq = scratch[zb.src.at(z) + li];
        u64 d = sub_mod(xq, v, q);
        u64 r = mul_tc(d, t.p_inv_tc + 4ull * i, pc);
        if (h == 0 && has_c0) r = add_mod(r, scratch[t0.at(zc) + li], q);
        if (has_acc) r = add_mod(r, arena[(h ? acc1.at(zc) : acc0.at(zc)) + li], q);
        arena[(h ? out1.at(zc) : out0.at(zc)) + li] = r;
    }
};

cudaError_t launch_ks_moddown(int log_n, const OpTabs& t, const LimbJob* jobs_qp, uint32_t slots_q, uint32_t sizeQl,
                              uint32_t K, u64* arena, u64* scratch, uint32_t nz, const ZBases& zb, const KsFuse& f,
                              u64 off_ext0, u64 off_ext1, u64 off_mid, u64 off_t0, cudaStream_t st) {
    const u64 n = 1ull << log_n;
    {
        ZBases a{};
        a.src = zf_pair(zf_plus(zb.mid, off_ext0), off_ext1 - off_ext0);
        a.aux = a.src;
        a.mid = a.src;
        a.out = a.src;
        // 4a. INTT of the special limbs, in place, times PHatInv
        cudaError_t e = launch_ntt<true>(log_n, t.pt, jobs_qp + slots_q, K, 2 * nz, scratch, a, LoadResidue{{scratch}},
                             StorePhatInv{scratch, t}, st);
        if (e != cudaSuccess) return e;
        // 4b. NTT over Q limbs with base-conversion prologue and ModDown epilogue
        ZBases b = a;
        b.mid = zf_pair(zf_plus(zb.mid, off_mid), (u64)slots_q * n);
        ModDownLoad pro{scratch, t, slots_q, K, (uint32_t)n};
        ModDownStore epi{};
        epi.scratch = scratch;
        epi.arena = arena;
        epi.t = t;
        epi.n = (uint32_t)n;
        epi.has_c0 = f.has_c0;
        epi.has_acc = f.has_acc;
        epi.t0 = zf_plus(zb.mid, off_t0);
        epi.out0 = zb.out;
        epi.out1 = zb.aux;
        epi.acc0 = f.acc0;
        epi.acc1 = f.acc1;
        e = launch_ntt<false>(log_n, t.pt, jobs_qp, sizeQl, 2 * nz, scratch, b, pro, epi, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace afhe

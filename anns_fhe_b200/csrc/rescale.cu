// rescale.cu -- rescale (hardware_fpga_model/hls/src/rescale.cpp:3-72): two
// transforms, with the lift of the dropped limb as the second one's prologue
// and the combine as its epilogue.
#include "internal.h"

namespace afhe {

// ---------------------------------------------------------------------------
// rescale (rescale.cpp:3-72)
//   step 1: INTT of the last limb -> coefficients in scratch
//   step 2: NTT over limbs i < L-1 whose prologue is the centred lift of the
//           last limb times QlQlInvModqlDivqlModq[i], and whose epilogue is
//           a_i * qlInvModq[i] + NTT(...)
// ---------------------------------------------------------------------------
// The lift times the constant as one product: where the coefficient is above
// q_l / 2 (rescale.cpp:50 tie rule), -q_l mod q_i is added to it first (a sum
// below 2^62, which the split product takes as it is).
struct RescaleLoad {
    static constexpr bool kMany = false;
    static constexpr bool kWords = false;
    const u64* scratch;
    const u64* qlql;
    const PrimeConst* pc_last;   // q_l, the prime being dropped
    __device__ __forceinline__ u64 operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x,
                                              const PrimeConst& pc) const {
        const u64 q = pc.q, nq = (u64)0 - q;
        const u64 ql = pc_last->q;
        const u64 minus = q - csub(mul_shoup_lazy(ql, 1, pc.one_sh, q), q);
        const ulonglong2 w = __ldg((const ulonglong2*)(qlql + 4ull * j.aux));
        const ulonglong2 s = __ldg((const ulonglong2*)(qlql + 4ull * j.aux) + 1);
        u64 v = scratch[zb.aux.at(z) + x];                           // last limb coefficient, [0, q_l)
        v += v > (ql >> 1) ? minus : 0;
        return csub(sp_mul(v, w.x, w.y, as_double(s.x), as_double(s.y), nq, sp_start(nq)), q);
    }
};

struct RescaleStore {
    u64* arena;
    const u64* qlinv;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst& pc) const {
        u64 a = arena[zb.src.at(z) + j.src + x];
        if (a >= pc.q) a = reduce128(0, a, modconst_of(pc));        // (a word that is no residue)
        arena[zb.out.at(z) + j.out + x] = add_mod(mul_tc(a, qlinv + 4ull * j.aux, pc), v, pc.q);
    }
};

// The same of the product with a plaintext (pt.at(z): its polynomial), which is
// formed where the transforms read it and written nowhere.
struct LoadProduct {
    static constexpr bool kMany = false;
    static constexpr bool kWords = false;
    const u64* arena;
    ZField pt;
    __device__ __forceinline__ u64 operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x,
                                              const PrimeConst& pc) const {
        return mul_words(arena[zb.src.at(z) + j.src + x], arena[pt.at(z) + j.src + x], pc);
    }
};
struct RescaleProductStore {
    u64* arena;
    const u64* qlinv;
    ZField pt;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst& pc) const {
        const u64 a = mul_words(arena[zb.src.at(z) + j.src + x], arena[pt.at(z) + j.src + x], pc);
        arena[zb.out.at(z) + j.out + x] = add_mod(mul_tc(a, qlinv + 4ull * j.aux, pc), v, pc.q);
    }
};

// zb.src = input poly (arena), zb.out = output poly (arena), zb.mid = scratch
// region of sizeQl * N words per z: words [0, N) hold the last limb's
// coefficients, words [N, sizeQl * N) the step-2 intermediates.
cudaError_t launch_rescale(int log_n, const OpTabs& t, const LimbJob* jobs_q, uint32_t sizeQl, u64* arena,
                           u64* scratch, uint32_t nz, const ZBases& zb_in, cudaStream_t st, const ZField* pt) {
    if (sizeQl < 2 || nz == 0) return cudaSuccess;
    const u64 n = 1ull << log_n;
    const uint32_t last = sizeQl - 1;
    // step 1: INTT(last limb). jobs_q[last] has src = dst = out = last * N,
    // so shifting mid / out back by last * N lands it at scratch + mid(z).
    ZBases z1 = zb_in;
    z1.mid = zf_plus(zb_in.mid, (u64)0 - (u64)last * n);
    z1.out = z1.mid;
    cudaError_t e = pt ? launch_ntt<true>(log_n, t.pt, jobs_q + last, 1, nz, scratch, z1, LoadProduct{arena, *pt},
                                          StorePlain{scratch}, st)
                       : launch_ntt<true>(log_n, t.pt, jobs_q + last, 1, nz, scratch, z1, LoadPlain{arena},
                                          StorePlain{scratch}, st);
    if (e != cudaSuccess) return e;
    // step 2
    ZBases z2 = zb_in;
    z2.aux = zb_in.mid;                      // coefficients of the last limb
    z2.mid = zf_plus(zb_in.mid, n);          // intermediates
    RescaleLoad pro{scratch, t.qlql_sp, t.pt.pc + last};
    if (pt)
        return launch_ntt<false>(log_n, t.pt, jobs_q, last, nz, scratch, z2, pro, RescaleProductStore{arena, t.qlinv_tc, *pt}, st);
    return launch_ntt<false>(log_n, t.pt, jobs_q, last, nz, scratch, z2, pro, RescaleStore{arena, t.qlinv_tc}, st);
}

}  // namespace afhe

// kernels.cu -- CUDA kernels and launchers for the CKKS evaluation core.
//
// Reference functions restated here (paths inside iheydardoost/ANNS_FHE):
//   poly_add / poly_sub / poly_mul      hardware_fpga_model/hls/src/poly_arith.cpp:3-38
//   automorphism                        hardware_fpga_model/hls/src/automorphism.cpp:3-12
//   rescale                             hardware_fpga_model/hls/src/rescale.cpp:3-72
//   fast_bases_conv / approx_mod_down   hardware_fpga_model/hls/src/key_switch.cpp:7-163
//   key_switch                          hardware_fpga_model/hls/src/key_switch.cpp:167-439
// Fusion: the base conversions run as the prologue of the NTT that consumes
// them; the rescale combine (a_i * q_l^-1 + NTT(...)) and the ModDown combine
// ((x_Q - y) * P^-1) run as the NTT epilogue; the evaluation-key inner product
// accumulates all digits of a limb in 128-bit registers and reduces once.
#include <atomic>

#include "internal.h"

namespace afhe {

static std::atomic<uint64_t> g_launches{0};
void count_launches(uint64_t k) { g_launches.fetch_add(k, std::memory_order_relaxed); }
uint64_t launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

static std::atomic<int> g_ntt_plan[17];
int ntt_plan(int log_n) { return log_n >= 0 && log_n <= 16 ? g_ntt_plan[log_n].load(std::memory_order_relaxed) : 0; }
void set_ntt_plan(int log_n, int plan) { g_ntt_plan[log_n].store(plan, std::memory_order_relaxed); }

// ---------------------------------------------------------------------------
// elementwise
// ---------------------------------------------------------------------------
template <int OP>
__global__ void __launch_bounds__(256) elementwise_kernel(const PrimeConst* __restrict__ pc, uint32_t prime0,
                                                          u64* __restrict__ arena, uint32_t n, const ZBases zb) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const PrimeConst p = pc[prime0 + l];
    const u64 off = (u64)l * n;
    const u64* a = arena + zb.src.at(z) + off;
    const u64* b = arena + zb.aux.at(z) + off;
    u64* o = arena + zb.out.at(z) + off;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        u64 x = a[i];
        u64 r;
        if (OP == EW_ADD) r = add_mod(x, b[i], p.q);
        else if (OP == EW_SUB) r = sub_mod(x, b[i], p.q);
        else if (OP == EW_MUL) r = mul_mod(x, b[i], modconst_of(p));
        else r = x;
        o[i] = r;
    }
}

cudaError_t launch_elementwise(ElemOp op, const PrimeConst* pc, uint32_t prime0, u64* arena, uint32_t n,
                               uint32_t limbs, uint32_t nz, const ZBases& zb, cudaStream_t st) {
    if (limbs == 0 || nz == 0) return cudaSuccess;
    dim3 grid((n + 255) / 256, limbs, nz);
    switch (op) {
    case EW_ADD: elementwise_kernel<EW_ADD><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb); break;
    case EW_SUB: elementwise_kernel<EW_SUB><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb); break;
    case EW_MUL: elementwise_kernel<EW_MUL><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb); break;
    default: elementwise_kernel<EW_COPY><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb); break;
    }
    count_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// ciphertext tensor product (fhe_host_driver.cpp:280-286):
//   d0 = a0*b0, d1 = a0*b1 + a1*b0, d2 = a1*b1  (d1 reduced once from 128 bits)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) tensor_kernel(const PrimeConst* __restrict__ pc, u64* __restrict__ arena,
                                                     uint32_t n, const TensorArgs ta) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const ModConst m = modconst_of(pc[l]);
    const u64 off = (u64)l * n;
    const u64* a0 = arena + ta.a0.at(z) + off;
    const u64* a1 = arena + ta.a1.at(z) + off;
    const u64* b0 = arena + ta.b0.at(z) + off;
    const u64* b1 = arena + ta.b1.at(z) + off;
    u64* d0 = arena + ta.d0.at(z) + off;
    u64* d1 = arena + ta.d1.at(z) + off;
    u64* d2 = arena + ta.d2.at(z) + off;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        u64 x0 = a0[i], x1 = a1[i], y0 = b0[i], y1 = b1[i];
        Acc128 c;
        acc_init(c);
        acc_mad(c, x0, y1);
        acc_mad(c, x1, y0);
        d0[i] = mul_mod(x0, y0, m);
        d1[i] = acc_reduce(c, m);
        d2[i] = mul_mod(x1, y1, m);
    }
}

cudaError_t launch_tensor(const PrimeConst* pc, u64* arena, uint32_t n, uint32_t limbs, uint32_t nz,
                          const TensorArgs& ta, cudaStream_t st) {
    if (limbs == 0 || nz == 0) return cudaSuccess;
    dim3 grid((n + 255) / 256, limbs, nz);
    tensor_kernel<<<grid, 256, 0, st>>>(pc, arena, n, ta);
    count_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// automorphism: out[i] = a[map[i]]
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) automorphism_kernel(const uint32_t* __restrict__ map32,
                                                           const u64* __restrict__ map64, u64* __restrict__ arena,
                                                           uint32_t n, const ZBases zb) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const u64 off = (u64)l * n;
    const u64* a = arena + zb.src.at(z) + off;
    u64* o = arena + zb.out.at(z) + off;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t idx;
        if (map32) idx = map32[i];
        else {
            u64 packed = map64[i >> 1];
            idx = (i & 1u) ? (uint32_t)(packed >> 32) : (uint32_t)(packed & 0xFFFFFFFFull);
        }
        o[i] = idx < n ? a[idx] : 0ull;  // out-of-range map entries read nothing
    }
}

cudaError_t launch_automorphism(const uint32_t* map32, const u64* map64, u64* arena, uint32_t n, uint32_t limbs,
                                uint32_t nz, const ZBases& zb, cudaStream_t st) {
    if (limbs == 0 || nz == 0) return cudaSuccess;
    dim3 grid((n + 255) / 256, limbs, nz);
    automorphism_kernel<<<grid, 256, 0, st>>>(map32, map64, arena, n, zb);
    count_launches(1);
    return cudaGetLastError();
}

// Every polynomial of a batch through its own permutation: maps.at(z) is the
// device address of polynomial z's map (N indices, each < N).
__global__ void __launch_bounds__(256) automorphism_z_kernel(const ZField maps, u64* __restrict__ arena, uint32_t n,
                                                            const ZBases zb) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const uint32_t* __restrict__ map = (const uint32_t*)maps.at(z);
    const u64 off = (u64)l * n;
    const u64* a = arena + zb.src.at(z) + off;
    u64* o = arena + zb.out.at(z) + off;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) o[i] = a[__ldg(map + i)];
}

cudaError_t launch_automorphism_z(const ZField& maps, u64* arena, uint32_t n, uint32_t limbs, uint32_t nz,
                                  const ZBases& zb, cudaStream_t st) {
    if (limbs == 0 || nz == 0) return cudaSuccess;
    dim3 grid((n + 255) / 256, limbs, nz);
    automorphism_z_kernel<<<grid, 256, 0, st>>>(maps, arena, n, zb);
    count_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// sums of plaintext-ciphertext products, each plaintext read through its own
// automorphism (the inner products of the diagonal method: a plaintext moved
// by a slot rotation is a permutation of its evaluation-form coefficients)
// ---------------------------------------------------------------------------
AFHE_HD void acc_fold(Acc128& a, const ModConst& m) {
    a.lo = acc_reduce(a, m);
    a.hi = 0;
}

__global__ void __launch_bounds__(256) mac_plain_kernel(const PrimeConst* __restrict__ pc, u64* __restrict__ arena,
                                                        uint32_t n, const MacJob* __restrict__ jobs,
                                                        const MacGroup* __restrict__ groups,
                                                        const MacTerm* __restrict__ terms, uint32_t reduce_every,
                                                        int accumulate) {
    const uint32_t l = blockIdx.y;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const MacJob J = jobs[blockIdx.z];
    const ModConst m = modconst_of(pc[l]);
    const u64 off = (u64)l * n + i;
    Acc128 a0, a1;
    acc_init(a0);
    acc_init(a1);
    uint32_t cnt = 0;
    for (uint32_t g = J.g0; g < J.g1; ++g) {
        const MacGroup G = groups[g];
        const bool unit = G.src0 == kMacUnit;
        const u64 x0 = unit ? 1 : arena[G.src0 + off];
        const u64 x1 = unit ? 0 : arena[G.src1 + off];
        for (uint32_t t = G.t0; t < G.t1; ++t) {
            const MacTerm T = terms[t];
            const uint32_t j = T.map ? __ldg(T.map + i) : i;
            const u64 p = arena[T.pt + (u64)l * n + j];
            acc_mad(a0, p, x0);
            if (!unit) acc_mad(a1, p, x1);
            if (++cnt == reduce_every) {
                acc_fold(a0, m);
                acc_fold(a1, m);
                cnt = 1;
            }
        }
    }
    u64 r0 = acc_reduce(a0, m), r1 = acc_reduce(a1, m);
    if (accumulate) {
        r0 = add_mod(r0, arena[J.out0 + off], m.q);
        r1 = add_mod(r1, arena[J.out1 + off], m.q);
    }
    arena[J.out0 + off] = r0;
    arena[J.out1 + off] = r1;
}

// One coefficient per thread: the nb baby-step ciphertexts' coefficients stay
// in registers while the job's units stream through; a unit's automorphism
// index is loaded once for its nb plaintexts, which lie `stride` words apart.
template <int NB>
__global__ void __launch_bounds__(256) diag_inner_kernel(const PrimeConst* __restrict__ pc, u64* __restrict__ arena,
                                                         uint32_t n, const DiagJob* __restrict__ jobs,
                                                         const u64* __restrict__ srcs,
                                                         const DiagUnit* __restrict__ units, u64 stride,
                                                         uint32_t reduce_every, int accumulate) {
    const uint32_t l = blockIdx.y;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DiagJob J = jobs[blockIdx.z];
    const ModConst m = modconst_of(pc[l]);
    const u64 off = (u64)l * n;
    const u64* s = srcs + (u64)blockIdx.z * 2 * NB;
    u64 x0[NB], x1[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        x0[b] = arena[s[2 * b] + off + i];
        x1[b] = arena[s[2 * b + 1] + off + i];
    }
    Acc128 a0, a1;
    acc_init(a0);
    acc_init(a1);
    uint32_t cnt = 0;
    // the next unit's descriptor and automorphism index are loaded while the
    // current unit's plaintexts are read and multiplied
    DiagUnit Un{};
    uint32_t jn = i;
    if (J.u0 < J.u1) {
        Un = units[J.u0];
        jn = Un.map ? __ldg(Un.map + i) : i;
    }
    for (uint32_t k = J.u0; k < J.u1; ++k) {
        const u64* p = arena + Un.pt + off + jn;
        if (k + 1 < J.u1) {
            Un = units[k + 1];
            jn = Un.map ? __ldg(Un.map + i) : i;
        }
        if (cnt + NB > reduce_every) {
            acc_fold(a0, m);
            acc_fold(a1, m);
            cnt = 1;
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const u64 v = p[(u64)b * stride];
            acc_mad(a0, v, x0[b]);
            acc_mad(a1, v, x1[b]);
        }
        cnt += NB;
    }
    u64 r0 = acc_reduce(a0, m), r1 = acc_reduce(a1, m);
    if (accumulate) {
        r0 = add_mod(r0, arena[J.out0 + off + i], m.q);
        r1 = add_mod(r1, arena[J.out1 + off + i], m.q);
    }
    arena[J.out0 + off + i] = r0;
    arena[J.out1 + off + i] = r1;
}

// The same sums with the plaintexts staged through shared memory: every
// placement map of the launch keeps each 256-coefficient tile within itself
// (a slot rotation by a multiple of D permutes the evaluation form inside
// blocks of N / 2D words), so a CTA copies the tile of all nb plaintexts of
// its next unit with cp.async while it multiplies the current one
// (double-buffered), and gathers from shared memory. One coefficient per
// thread, 256 threads: tile t = coefficients [256 t, 256 t + 256).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

constexpr uint32_t kDiagTile = 256;

// Residues below 2^50: operands split into 25-bit halves, x = x1 2^25 + x0;
// the partial sums x0 y0, x0 y1 + x1 y0, x1 y1 of the products accumulate
// in 64-bit registers by single 32 x 32 + 64 multiply-adds (products of
// halves < 2^50: 4,096 products fit between folds); recombined in 128 bits.
constexpr uint32_t kHalfBits = 25, kHalfMask = (1u << kHalfBits) - 1, kHalfFold = 4096;
__device__ __forceinline__ void mad_wide(u64& acc, uint32_t a, uint32_t b) {
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}
struct Halves {
    u64 s00, s01, s11;
};
__device__ __forceinline__ void halves_mad(Halves& h, uint32_t v0, uint32_t v1, uint32_t x0, uint32_t x1) {
    mad_wide(h.s00, v0, x0);
    mad_wide(h.s01, v0, x1);
    mad_wide(h.s01, v1, x0);
    mad_wide(h.s11, v1, x1);
}
__device__ __forceinline__ u64 halves_reduce(const Halves& h, const ModConst& m) {
    u64 lo = h.s00, hi = 0;
    const u64 t1 = h.s01 << kHalfBits, t2 = h.s11 << (2 * kHalfBits);
    lo += t1;
    hi += (lo < t1 ? 1 : 0) + (h.s01 >> (64 - kHalfBits));
    lo += t2;
    hi += (lo < t2 ? 1 : 0) + (h.s11 >> (64 - 2 * kHalfBits));
    return reduce128(hi, lo, m);
}

template <int NB, bool HALVES>
__global__ void __launch_bounds__(kDiagTile) diag_inner_staged_kernel(
    const PrimeConst* __restrict__ pc, u64* __restrict__ arena, uint32_t n, const DiagJob* __restrict__ jobs,
    const u64* __restrict__ srcs, const DiagUnit* __restrict__ units, u64 stride, uint32_t reduce_every,
    int accumulate) {
    extern __shared__ u64 stage[];          // 2 buffers x NB plaintexts x kDiagTile words
    // jobs vary fastest across the grid: consecutive CTAs are other outputs
    // of the same tile, so outputs that share their baby steps (one query's
    // giant steps) read them from L2
    const uint32_t z = blockIdx.x, l = blockIdx.z, tid = threadIdx.x;
    const uint32_t base = blockIdx.y * kDiagTile, i = base + tid;
    const DiagJob J = jobs[z];
    const ModConst m = modconst_of(pc[l]);
    const u64 off = (u64)l * n;
    const u64* s = srcs + (u64)z * 2 * NB;
    u64 x0[HALVES ? 1 : NB], x1[HALVES ? 1 : NB];
    uint32_t h00[HALVES ? NB : 1], h01[HALVES ? NB : 1], h10[HALVES ? NB : 1], h11[HALVES ? NB : 1];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const u64 y0 = arena[s[2 * b] + off + i], y1 = arena[s[2 * b + 1] + off + i];
        if (HALVES) {
            h00[b] = (uint32_t)y0 & kHalfMask;
            h01[b] = (uint32_t)(y0 >> kHalfBits);
            h10[b] = (uint32_t)y1 & kHalfMask;
            h11[b] = (uint32_t)(y1 >> kHalfBits);
        } else {
            x0[b] = y0;
            x1[b] = y1;
        }
    }
    // unit k's tile of its NB plaintexts into buffer `buf`: NB x 128 chunks of 16 bytes
    auto issue = [&](uint32_t k, uint32_t buf) {
        const u64* g = arena + units[k].pt + off + base;
        u64* d = stage + (size_t)buf * NB * kDiagTile;
        for (uint32_t c = tid; c < NB * (kDiagTile / 2); c += kDiagTile) {
            const uint32_t b = c / (kDiagTile / 2), w = (c % (kDiagTile / 2)) * 2;
            cp_async16(d + b * kDiagTile + w, g + (u64)b * stride + w);
        }
        cp_async_commit();
    };
    Acc128 a0, a1;
    acc_init(a0);
    acc_init(a1);
    Halves c0{0, 0, 0}, c1{0, 0, 0};
    uint32_t cnt = 0;
    if (J.u0 < J.u1) issue(J.u0, 0);
    for (uint32_t k = J.u0; k < J.u1; ++k) {
        const uint32_t buf = (k - J.u0) & 1u;
        const uint32_t* map = units[k].map;
        const uint32_t j = (map ? __ldg(map + i) : i) - base;
        if (k + 1 < J.u1) {
            issue(k + 1, buf ^ 1u);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const u64* t = stage + (size_t)buf * NB * kDiagTile + j;
        if (HALVES) {
            if (cnt + NB > kHalfFold) {
                c0 = Halves{halves_reduce(c0, m), 0, 0};
                c1 = Halves{halves_reduce(c1, m), 0, 0};
                cnt = 1;
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const u64 v = t[b * kDiagTile];
                const uint32_t v0 = (uint32_t)v & kHalfMask, v1 = (uint32_t)(v >> kHalfBits);
                halves_mad(c0, v0, v1, h00[b], h01[b]);
                halves_mad(c1, v0, v1, h10[b], h11[b]);
            }
        } else {
            if (cnt + NB > reduce_every) {
                acc_fold(a0, m);
                acc_fold(a1, m);
                cnt = 1;
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const u64 v = t[b * kDiagTile];
                acc_mad(a0, v, x0[b]);
                acc_mad(a1, v, x1[b]);
            }
        }
        cnt += NB;
        __syncthreads();                    // the buffer is refilled two units later
    }
    u64 r0 = HALVES ? halves_reduce(c0, m) : acc_reduce(a0, m);
    u64 r1 = HALVES ? halves_reduce(c1, m) : acc_reduce(a1, m);
    if (accumulate) {
        r0 = add_mod(r0, arena[J.out0 + off + i], m.q);
        r1 = add_mod(r1, arena[J.out1 + off + i], m.q);
    }
    arena[J.out0 + off + i] = r0;
    arena[J.out1 + off + i] = r1;
}

cudaError_t launch_diag_inner(const PrimeConst* pc, u64* arena, uint32_t n, uint32_t limbs, uint32_t jobs,
                              uint32_t nb, const DiagJob* job, const u64* srcs, const DiagUnit* unit, u64 stride,
                              uint32_t reduce_every, int accumulate, bool staged, bool halves, cudaStream_t st) {
    if (limbs == 0 || jobs == 0) return cudaSuccess;
    if (staged) {
        if (n % kDiagTile) return cudaErrorInvalidValue;
        if (n / kDiagTile > 65535 || limbs > 65535) return cudaErrorInvalidValue;
        dim3 grid(jobs, n / kDiagTile, limbs);
        const size_t smem = 2ull * nb * kDiagTile * sizeof(u64);
#define DIAG_STAGED_H(NBV, H)                                                                                  \
    {                                                                                                          \
        cudaError_t e = cudaFuncSetAttribute(diag_inner_staged_kernel<NBV, H>,                                 \
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);          \
        if (e != cudaSuccess) return e;                                                                        \
        diag_inner_staged_kernel<NBV, H><<<grid, kDiagTile, smem, st>>>(pc, arena, n, job, srcs, unit, stride, \
                                                                        reduce_every, accumulate);             \
    }
#define DIAG_STAGED(NBV)                \
    case NBV:                           \
        if (halves)                     \
            DIAG_STAGED_H(NBV, true)    \
        else                            \
            DIAG_STAGED_H(NBV, false)   \
        break;
        switch (nb) {
            DIAG_STAGED(1)
            DIAG_STAGED(2)
            DIAG_STAGED(4)
            DIAG_STAGED(8)
            DIAG_STAGED(16)
        default: return cudaErrorInvalidValue;
        }
#undef DIAG_STAGED
#undef DIAG_STAGED_H
        count_launches(1);
        return cudaGetLastError();
    }
    dim3 grid((n + 255) / 256, limbs, jobs);
    switch (nb) {
    case 1: diag_inner_kernel<1><<<grid, 256, 0, st>>>(pc, arena, n, job, srcs, unit, stride, reduce_every, accumulate); break;
    case 2: diag_inner_kernel<2><<<grid, 256, 0, st>>>(pc, arena, n, job, srcs, unit, stride, reduce_every, accumulate); break;
    case 4: diag_inner_kernel<4><<<grid, 256, 0, st>>>(pc, arena, n, job, srcs, unit, stride, reduce_every, accumulate); break;
    case 8: diag_inner_kernel<8><<<grid, 256, 0, st>>>(pc, arena, n, job, srcs, unit, stride, reduce_every, accumulate); break;
    case 16: diag_inner_kernel<16><<<grid, 256, 0, st>>>(pc, arena, n, job, srcs, unit, stride, reduce_every, accumulate); break;
    default: return cudaErrorInvalidValue;
    }
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_mac_plain(const PrimeConst* pc, u64* arena, uint32_t n, uint32_t limbs, uint32_t jobs,
                             const MacJob* job, const MacGroup* group, const MacTerm* term, uint32_t reduce_every,
                             int accumulate, cudaStream_t st) {
    if (limbs == 0 || jobs == 0) return cudaSuccess;
    dim3 grid((n + 255) / 256, limbs, jobs);
    mac_plain_kernel<<<grid, 256, 0, st>>>(pc, arena, n, job, group, term, reduce_every, accumulate);
    count_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// plain transforms
// ---------------------------------------------------------------------------
cudaError_t launch_ntt_plain(bool inverse, int log_n, const PrimeTables& pt, const LimbJob* jobs, uint32_t limbs,
                             u64* src_arena, u64* dst_arena, uint32_t nz, const ZBases& zb, cudaStream_t st) {
    LoadPlain pro{src_arena};
    StorePlain epi{dst_arena};
    if (inverse) return launch_ntt<true>(log_n, pt, jobs, limbs, nz, dst_arena, zb, pro, epi, st);
    return launch_ntt<false>(log_n, pt, jobs, limbs, nz, dst_arena, zb, pro, epi, st);
}

// ---------------------------------------------------------------------------
// table preparation
// ---------------------------------------------------------------------------
__global__ void companions_kernel(u64* v, u64* sh, const u64* m, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        u64 mod = m[i];
        if (mod == 0) { sh[i] = 0; continue; }
        u64 w = v[i] % mod;
        v[i] = w;
        sh[i] = shoup_companion(w, mod);
    }
}

cudaError_t launch_companions(u64* v, u64* sh, const u64* m, size_t count, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((count + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    companions_kernel<<<blocks, 256, 0, st>>>(v, sh, m, count);
    count_launches(1);
    return cudaGetLastError();
}

__global__ void twiddles_kernel(const u64* __restrict__ raw, const u64* __restrict__ q, ulonglong2* __restrict__ out2,
                                ulonglong2* __restrict__ out2b, uint32_t rows, int log_n) {
    const size_t total = (size_t)rows << log_n;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i >> log_n;
        const uint32_t j = (uint32_t)(i & ((1u << log_n) - 1));
        const u64 m = q[row];
        u64 o[4];
        transform_constant(raw[i] % m, m, o);
        uint32_t at = 0;                       // j = 0 belongs to no stage
        if (j) {
            const int lg = 31 - __clz((int)j);
            at = tw_place(log_n, log_n - 1 - lg, j - (1u << lg));
        }
        out2[(row << log_n) + at] = make_ulonglong2(o[0], o[1]);
        out2b[(row << log_n) + at] = make_ulonglong2(o[2], o[3]);
    }
}

cudaError_t launch_twiddles(const u64* raw, const u64* q, ulonglong2* out2, ulonglong2* out2b, uint32_t rows, int log_n,
                            cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    const size_t total = (size_t)rows << log_n;
    unsigned blocks = (unsigned)((total + 255) / 256);
    if (blocks > 8192) blocks = 8192;
    twiddles_kernel<<<blocks, 256, 0, st>>>(raw, q, out2, out2b, rows, log_n);
    count_launches(1);
    return cudaGetLastError();
}

__global__ void prime_consts_kernel(PrimeConst* pc, const u64* q, const u64* ninv, const u64* itw, uint32_t n,
                                    uint32_t count) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    PrimeConst c;
    c.q = q[i];
    ModConst m = make_modconst(c.q);
    c.r64 = m.r64;
    c.r64_sh = m.r64_sh;
    c.one_sh = m.one_sh;
    c.ninv = ninv[i] % c.q;
    c.ninv_sh = shoup_companion(c.ninv, c.q);
    c.w1ninv = mul_mod(itw[(u64)i * n + 1] % c.q, c.ninv, m);
    c.w1ninv_sh = shoup_companion(c.w1ninv, c.q);
    set_transform_constants(c);
    pc[i] = c;
}

cudaError_t launch_prime_consts(PrimeConst* pc, const u64* q, const u64* ninv, const u64* itw, uint32_t n,
                                uint32_t count, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    prime_consts_kernel<<<(count + 63) / 64, 64, 0, st>>>(pc, q, ninv, itw, n, count);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace afhe

// kernels.cu -- CUDA kernels and launchers for the CKKS evaluation core: pointwise
// operations, tensor products, automorphisms, sums of plaintext products (the
// diagonal method's among them), plain transforms and the tables' constants.
//
// Reference functions restated here (paths inside iheydardoost/ANNS_FHE):
//   poly_add / poly_sub / poly_mul      hardware_fpga_model/hls/src/poly_arith.cpp:3-38
//   automorphism                        hardware_fpga_model/hls/src/automorphism.cpp:3-12
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
// PER coefficients a thread, 256 apart: the loads of all are on their way
// before the first is used. Products of primes below 2^50 in doubles (10 FP64
// instructions in place of about 95 multiplier cycles for the 128-bit product
// and its reduction). Four a thread, or one in launches of few words, which four in a
// row take longer than the launch itself (products of one limb one after another,
// N = 2^11, us, four / one: 60 bits 4.1 / 3.4, 50 bits 4.1 / 3.3; of 2^17 words 4.1 both).
template <int OP, uint32_t PER, class PC>
__global__ void __launch_bounds__(256) elementwise_kernel(const PC* __restrict__ pc, uint32_t prime0,
                                                          u64* __restrict__ arena, uint32_t n, const ZBases zb) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const PrimeBase p = pc[prime0 + l];
    const uint32_t i0 = blockIdx.x * (256 * PER) + threadIdx.x;
    const u64 off = (u64)l * n + i0;
    const u64* a = arena + zb.src.at(z) + off;
    const u64* b = arena + zb.aux.at(z) + off;
    u64* o = arena + zb.out.at(z) + off;
    u64 x[PER], y[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        const bool in = i0 + 256 * k < n;
        x[k] = in ? a[256 * k] : 0;
        y[k] = OP != EW_COPY && in ? b[256 * k] : 0;
    }
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        u64 r = x[k];
        if (OP == EW_ADD) r = add_mod(x[k], y[k], p.q);
        else if (OP == EW_SUB) r = sub_mod(x[k], y[k], p.q);
        else if (OP == EW_MUL) r = mul_words(x[k], y[k], p);
        if (i0 + 256 * k < n) o[256 * k] = r;
    }
}

constexpr u64 kEwFew = 1u << 16;     // words
template <int OP, class PC>
void launch_ew(bool few, const PC* pc, uint32_t prime0, u64* arena, uint32_t n, uint32_t limbs, uint32_t nz,
               const ZBases& zb, cudaStream_t st) {
    const uint32_t per = few ? 256 : 256 * 4;
    const dim3 grid((n + per - 1) / per, limbs, nz);
    if (few) elementwise_kernel<OP, 1, PC><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb);
    else elementwise_kernel<OP, 4, PC><<<grid, 256, 0, st>>>(pc, prime0, arena, n, zb);
}

template <class PC>
cudaError_t launch_elementwise(ElemOp op, const PC* pc, uint32_t prime0, u64* arena, uint32_t n,
                               uint32_t limbs, uint32_t nz, const ZBases& zb, cudaStream_t st) {
    if (limbs == 0 || nz == 0) return cudaSuccess;
    const bool few = (u64)n * limbs * nz <= kEwFew;
    switch (op) {
    case EW_ADD: launch_ew<EW_ADD>(few, pc, prime0, arena, n, limbs, nz, zb, st); break;
    case EW_SUB: launch_ew<EW_SUB>(few, pc, prime0, arena, n, limbs, nz, zb, st); break;
    case EW_MUL: launch_ew<EW_MUL>(few, pc, prime0, arena, n, limbs, nz, zb, st); break;
    default: launch_ew<EW_COPY>(few, pc, prime0, arena, n, limbs, nz, zb, st); break;
    }
    count_launches(1);
    return cudaGetLastError();
}
template cudaError_t launch_elementwise(ElemOp, const PrimeConst*, uint32_t, u64*, uint32_t, uint32_t, uint32_t,
                                        const ZBases&, cudaStream_t);
template cudaError_t launch_elementwise(ElemOp, const PrimeBase*, uint32_t, u64*, uint32_t, uint32_t, uint32_t,
                                        const ZBases&, cudaStream_t);

// ---------------------------------------------------------------------------
// ciphertext tensor product (fhe_host_driver.cpp:280-286):
//   d0 = a0*b0, d1 = a0*b1 + a1*b0, d2 = a1*b1  (d1 reduced once from 128 bits)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) tensor_kernel(const PrimeConst* __restrict__ pc, u64* __restrict__ arena,
                                                     uint32_t n, const TensorArgs ta) {
    const uint32_t l = blockIdx.y, z = blockIdx.z;
    const PrimeConst p = pc[l];
    const ModConst m = modconst_of(p);
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
        if (p.fp && x0 < p.q && x1 < p.q && y0 < p.q && y1 < p.q) {
            const double f0 = fp_of(x0), f1 = fp_of(x1), g0 = fp_of(y0), g1 = fp_of(y1);
            const double c = __dadd_rn(fp_mul2(f0, g1, p.qd, p.qi), fp_mul2(f1, g0, p.qd, p.qi));
            d0[i] = fp_canon(fp_mul2(f0, g0, p.qd, p.qi), p.qd);
            d1[i] = fp_canon(fp_center(c, p.qd, p.qi), p.qd);
            d2[i] = fp_canon(fp_mul2(f1, g1, p.qd, p.qi), p.qd);
            continue;
        }
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

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

constexpr uint32_t kDiagTile = 256, kDiagUnits = 128;

// Residues below 2^50: operands split into 25-bit halves, x = x1 2^25 + x0;
// the partial sums x0 y0, x0 y1 + x1 y0, x1 y1 of the products accumulate
// in 64-bit registers by single 32 x 32 + 64 multiply-adds (products of
// halves below 2^57: room for 32 of the middle ones, used for at most 16 of
// them twice); recombined in 128 bits.
constexpr uint32_t kHalfBits = 25, kHalfMask = (1u << kHalfBits) - 1, kWordBits = 2 * kHalfBits;
struct Halves {
    u64 s00, s01, s11;
};
__device__ __forceinline__ void halves_mad(Halves& h, uint32_t v0, uint32_t v1, u64 x) {
    const uint32_t x0 = (uint32_t)x & kHalfMask, x1 = (uint32_t)(x >> kHalfBits);
    h.s00 = mad_wide_u32(v0, x0, h.s00);
    h.s01 = mad_wide_u32(v0, x1, h.s01);
    h.s01 = mad_wide_u32(v1, x0, h.s01);
    h.s11 = mad_wide_u32(v1, x1, h.s11);
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

// The diagonal method's inner products, out = sum over units u, baby steps b of
// plaintext(u, b) x(b). Every unit of an output meets the same baby steps, so
// a thread first adds up its coefficient of the units' plaintexts (a sum for
// each of the nb baby steps) and then multiplies: nb products an output instead
// of nb times its units. The sums hold for every output of
// a group (results of other baby steps with the same units: queries that scan
// the same list), so a group's plaintexts are read once too; what is left is
// the reading of each output's 2 nb coefficients, from L2 where the outputs of
// neighbouring CTAs share their baby steps.
// HALVES: primes below 2^50; sums of up to kDiagUnits residues are below 2^57, a
// 25-bit half and a 32-bit one, and multiply as they are. Else the sums have
// 96 bits and are reduced once. Words that are no residues: ANY looks at each and
// reduces those from 2^50 on; without it (the shared-memory form, where that
// look costs 10% of the kernel) plaintexts may be below 2^57 and baby steps
// below 2^53. One coefficient per thread, tile t =
// coefficients [256 t, 256 t + 256); groups vary fastest across the grid, so
// consecutive CTAs are other groups of the same tile.
template <int NB, bool HALVES>
struct DiagSums {
    u64 p[NB];
    uint32_t hi[HALVES ? 1 : NB];
    __device__ __forceinline__ DiagSums() {
#pragma unroll
        for (int b = 0; b < NB; ++b) p[b] = 0;
#pragma unroll
        for (int b = 0; b < (HALVES ? 1 : NB); ++b) hi[b] = 0;
    }
    // the array moves on by one, `first` to its end: a loop over it with one copy
    // of its body and no more registers
    __device__ __forceinline__ void turn(u64 first) {
#pragma unroll
        for (int c = 0; c + 1 < NB; ++c) p[c] = p[c + 1];
        p[NB - 1] = first;
    }
    // unit k's plaintexts, `stride` words apart
    template <bool ANY>
    __device__ __forceinline__ void add(uint32_t k, const u64* t, u64 stride, const ModConst& m) {
        uint32_t high = 0;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const u64 v = t[b * stride];
            p[b] += v;
            if (HALVES && ANY) high |= (uint32_t)(v >> 32);
            if (!HALVES) hi[b] += p[b] < v ? 1u : 0u;
        }
        if (HALVES && ANY && high >> (kWordBits - 32)) {     // (words that are no residues)
#pragma unroll 1
            for (int b = 0; b < NB; ++b) {
                const u64 v = t[b * stride];
                turn(p[0] + reduce128(0, v, m) - v);
            }
        }
        if (HALVES && k % (kDiagUnits - 1) == kDiagUnits - 2) {
#pragma unroll 1
            for (int b = 0; b < NB; ++b) turn(reduce128(0, p[0], m));
        }
    }
    // after the last unit: residues, or their halves side by side
    __device__ __forceinline__ void close(const ModConst& m) {
        if (HALVES) {
            uint32_t high = 0;
#pragma unroll
            for (int b = 0; b < NB; ++b) high |= (uint32_t)(p[b] >> 32);
            if (high >> kHalfBits) {                    // a sum from 2^57 on (words that are no residues)
#pragma unroll 1
                for (int b = 0; b < NB; ++b) turn(reduce128(0, p[0], m));
            }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
            p[b] = HALVES ? (p[b] >> kHalfBits << 32 | ((uint32_t)p[b] & kHalfMask)) : reduce128(hi[HALVES ? 0 : b], p[b], m);
    }
    template <bool ANY, typename X>
    __device__ __forceinline__ u64 times(X&& x, const ModConst& m) {
        if (HALVES) {
            Halves c{0, 0, 0};
            uint32_t high = 0;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const u64 v = x(b);
                if (ANY) high |= (uint32_t)(v >> 32);
                halves_mad(c, (uint32_t)p[b], (uint32_t)(p[b] >> 32), v);
            }
            if (ANY && high >> (kWordBits - 32)) {      // (words that are no residues)
                c = Halves{0, 0, 0};
#pragma unroll 1
                for (int b = 0; b < NB; ++b) {
                    halves_mad(c, (uint32_t)p[0], (uint32_t)(p[0] >> 32), reduce128(0, x(b), m));
                    turn(p[0]);
                }
            }
            return halves_reduce(c, m);
        }
        Acc128 a;
        acc_init(a);
#pragma unroll
        for (int b = 0; b < NB; ++b) acc_mad(a, p[b], x(b));
        return acc_reduce(a, m);
    }
};

// Plaintexts and baby steps straight from global memory: any placement map,
// any alignment.
template <int NB, bool HALVES>
__global__ void __launch_bounds__(kDiagTile) diag_inner_kernel(
    const PrimeConst* __restrict__ pc, u64* __restrict__ arena, uint32_t n, const DiagGroup* __restrict__ groups,
    const DiagJob* __restrict__ jobs, const u64* __restrict__ srcs, const DiagUnit* __restrict__ units, u64 stride,
    int accumulate) {
    const uint32_t l = blockIdx.z, i = blockIdx.y * kDiagTile + threadIdx.x;
    if (i >= n) return;
    const DiagGroup G = groups[blockIdx.x];
    const ModConst m = modconst_of(pc[l]);
    arena += (u64)l * n;
    DiagSums<NB, HALVES> sums;
    const DiagJob J = jobs[G.first];
    for (uint32_t k = J.u0; k < J.u1; ++k) {
        const DiagUnit U = units[k];
        sums.template add<true>(k - J.u0, arena + U.pt + J.add + (U.map ? __ldg(U.map + i) : i), stride, m);
    }
    sums.close(m);
    for (uint32_t z = G.first; z < G.first + G.count; ++z) {
        const u64* s = srcs + 2ull * jobs[z].s;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            u64* out = arena + (h ? jobs[z].out1 : jobs[z].out0) + i;
            const u64 r = sums.template times<true>([&](int b) { return arena[s[2 * b + h] + i]; }, m);
            *out = accumulate ? add_mod(r, *out, m.q) : r;
        }
    }
}

// Primes below 2^50, eight baby steps or more, and every placement map of the
// launch keeps each 256-coefficient tile within itself (a slot rotation by a multiple of D permutes the evaluation form
// inside blocks of N / 2D words): tiles of nb rows, a unit's plaintexts or one
// half of an output's baby steps, come by cp.async into one of two buffers
// while the other is worked on. 64 KB a CTA at nb = 16, three on an SM.
// 480 outputs of 9 units at nb = 16, N = 2^15, two limbs: 43 GB through L2, of
// which 9.5 GB from HBM, in 3.3 ms (7.0 ms with a product for each plaintext
// word); L2 at 56% and the issue slots at 54% of their peaks. Measured and
// slower: four buffers of eight rows (3.7 ms: the instructions of a deeper
// ring), the products with a baby step for each unit in double precision
// (9.0 ms).
template <int NB>
__global__ void __launch_bounds__(kDiagTile, 3) diag_inner_staged_kernel(
    const PrimeConst* __restrict__ pc, u64* __restrict__ arena, uint32_t n, const DiagGroup* __restrict__ groups,
    const DiagJob* __restrict__ jobs, const u64* __restrict__ srcs, const DiagUnit* __restrict__ units, u64 stride,
    int accumulate) {
    extern __shared__ __align__(16) u64 stage[];          // 2 buffers x NB rows x kDiagTile words
    __shared__ u64 from[2][2 * NB];         // an output's baby steps, one output ahead
    const uint32_t l = blockIdx.z, tid = threadIdx.x;
    const DiagGroup G = groups[blockIdx.x];
    const ModConst m = modconst_of(pc[l]);
    const uint32_t base = blockIdx.y * kDiagTile, i = base + tid;
    arena += (u64)l * n + base;
    const DiagJob J = jobs[G.first];
    const uint32_t nu = J.u1 - J.u0, items = nu + 2 * G.count;
    units += J.u0;
    if (tid < 2 * NB) from[0][tid] = srcs[2ull * J.s + tid];
    // thread t copies words [2 (t % 128), + 2) of rows t / 128, t / 128 + 2, ...
    const uint32_t row = tid / (kDiagTile / 2), col = tid % (kDiagTile / 2) * 2;
    const u64 first = J.add + row * stride + col;
    const u64 step = 2 * stride;
    auto issue_unit = [&](uint32_t k, u64 pt) {
        const u64* g = arena + (first + pt);
        u64* d = stage + ((k & 1u) * NB + row) * kDiagTile + col;
#pragma unroll
        for (uint32_t r = 0; r < NB / 2; ++r, g += step) cp_async16(d + 2 * r * kDiagTile, g);
        cp_async_commit();
    };
    auto issue_baby = [&](uint32_t k) {
        const uint32_t e = k - nu;
        const u64* f = &from[e >> 1 & 1u][2 * row + (e & 1u)];
        u64* d = stage + ((k & 1u) * NB + row) * kDiagTile + col;
#pragma unroll
        for (uint32_t r = 0; r < NB / 2; ++r) cp_async16(d + 2 * r * kDiagTile, arena + f[4 * r] + col);
        cp_async_commit();
    };
    // the next unit's descriptor and automorphism index are loaded while the
    // current unit is added
    DiagUnit U{0, nullptr}, V{0, nullptr};
    uint32_t j = tid, jn = tid;
    if (nu) U = units[0];
    if (nu > 1) V = units[1];
    if (nu) {
        issue_unit(0, U.pt);
        if (U.map) j = __ldg(U.map + i) - base;
    } else {
        __syncthreads();
        issue_baby(0);
    }
    DiagSums<NB, true> sums;
    for (uint32_t k = 0; k < nu; ++k) {
        cp_async_wait<0>();
        __syncthreads();                    // item k is here, the other buffer free
        if (k + 1 < nu) {
            issue_unit(k + 1, V.pt);
            jn = V.map ? __ldg(V.map + i) - base : tid;
            if (k + 2 < nu) V = units[k + 2];
        } else {
            issue_baby(nu);
        }
        sums.template add<false>(k, stage + (k & 1u) * NB * kDiagTile + j, kDiagTile, m);
        j = jn;
    }
    sums.close(m);
    for (uint32_t k = nu; k < items; ++k) {
        const uint32_t e = k - nu, z = G.first + (e >> 1);
        cp_async_wait<0>();
        __syncthreads();
        if (k + 1 < items) issue_baby(k + 1);
        if (!(e & 1u) && z + 1 < G.first + G.count && tid < 2 * NB) from[~(e >> 1) & 1u][tid] = srcs[2ull * jobs[z + 1].s + tid];
        u64* out = arena + ((e & 1u) ? jobs[z].out1 : jobs[z].out0) + tid;
        const u64* t = stage + (k & 1u) * NB * kDiagTile + tid;
        const u64 r = sums.template times<false>([&](int b) { return t[b * kDiagTile]; }, m);
        *out = accumulate ? add_mod(r, *out, m.q) : r;
    }
}

// Up to three units an output, and no plaintexts shared between outputs (or one
// unit): the sums above would only put the plaintexts' loads before the baby
// steps'. Four baby steps at a time with all their loads in flight, products in 128
// bits (they fit: 48 of below 2^61 squared; 25-bit halves are slower, 292 against
// 253 us for 64 outputs of one shared unit at nb = 16, N = 2^15, two limbs). Any
// placement, any alignment, any words. 64 outputs of one unit each at nb = 8, 60-bit
// primes: 146 us (209 through the sums).
template <int NB, int NU>
__global__ void __launch_bounds__(kDiagTile) diag_inner_few_kernel(
    const PrimeConst* __restrict__ pc, u64* __restrict__ arena, uint32_t n, const DiagJob* __restrict__ jobs,
    const u64* __restrict__ srcs, const DiagUnit* __restrict__ units, u64 stride, int accumulate) {
    constexpr int C = NB < 4 ? NB : 4;
    const uint32_t l = blockIdx.z, i = blockIdx.y * kDiagTile + threadIdx.x;
    if (i >= n) return;
    const DiagJob J = jobs[blockIdx.x];
    const ModConst m = modconst_of(pc[l]);
    arena += (u64)l * n;
    const u64* pt[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        const DiagUnit U = units[J.u0 + u];
        pt[u] = arena + (U.pt + J.add + (U.map ? __ldg(U.map + i) : i));
    }
    srcs += 2ull * J.s;
    Acc128 a0, a1;
    acc_init(a0);
    acc_init(a1);
    u64 high = 0;
#pragma unroll 2
    for (int b = 0; b < NB; b += C) {
        u64 p[C], x0[C], x1[C];
#pragma unroll
        for (int e = 0; e < C; ++e) {
            x0[e] = arena[srcs[2 * (b + e)] + i];
            x1[e] = arena[srcs[2 * (b + e) + 1] + i];
            p[e] = 0;
        }
#pragma unroll
        for (int u = 0; u < NU; ++u)
#pragma unroll
            for (int e = 0; e < C; ++e) {
                const u64 v = pt[u][(b + e) * stride];
                high |= v;
                p[e] += v;
            }
#pragma unroll
        for (int e = 0; e < C; ++e) {
            high |= x0[e] | x1[e];
            acc_mad(a0, p[e], x0[e]);
            acc_mad(a1, p[e], x1[e]);
        }
    }
    if (high >> 61) {                       // (words that are no residues)
        acc_init(a0);
        acc_init(a1);
#pragma unroll 1
        for (int b = 0; b < NB; ++b) {
            u64 p = 0;
            for (int u = 0; u < NU; ++u) p += reduce128(0, pt[u][b * stride], m);
            acc_mad(a0, p, reduce128(0, arena[srcs[2 * b] + i], m));
            acc_mad(a1, p, reduce128(0, arena[srcs[2 * b + 1] + i], m));
        }
    }
    u64 r0 = acc_reduce(a0, m), r1 = acc_reduce(a1, m);
    if (accumulate) {
        r0 = add_mod(r0, arena[J.out0 + i], m.q);
        r1 = add_mod(r1, arena[J.out1 + i], m.q);
    }
    arena[J.out0 + i] = r0;
    arena[J.out1 + i] = r1;
}

template <int NB, bool HALVES>
cudaError_t launch_diag(const PrimeConst* pc, u64* arena, uint32_t n, uint32_t limbs, uint32_t groups,
                        const DiagGroup* group, const DiagJob* job, const u64* srcs, const DiagUnit* unit, u64 stride,
                        int accumulate, bool staged, uint32_t few, cudaStream_t st) {
    const dim3 grid(groups, (n + kDiagTile - 1) / kDiagTile, limbs);
    if (few) {
        auto kern = few == 1 ? diag_inner_few_kernel<NB, 1> : few == 2 ? diag_inner_few_kernel<NB, 2> : diag_inner_few_kernel<NB, 3>;
        kern<<<grid, kDiagTile, 0, st>>>(pc, arena, n, job, srcs, unit, stride, accumulate);
    } else if (staged) {
        if constexpr (HALVES && NB >= 8) {
            const size_t smem = 2ull * NB * kDiagTile * sizeof(u64);
            auto kern = diag_inner_staged_kernel<NB>;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            kern<<<grid, kDiagTile, smem, st>>>(pc, arena, n, group, job, srcs, unit, stride, accumulate);
        } else {
            return cudaErrorInvalidValue;
        }
    } else {
        diag_inner_kernel<NB, HALVES><<<grid, kDiagTile, 0, st>>>(pc, arena, n, group, job, srcs, unit, stride, accumulate);
    }
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_diag_inner(const PrimeConst* pc, u64* arena, uint32_t n, uint32_t limbs, uint32_t groups,
                              uint32_t nb, const DiagGroup* group, const DiagJob* job, const u64* srcs,
                              const DiagUnit* unit, u64 stride, int accumulate, bool staged, bool halves, uint32_t few,
                              cudaStream_t st) {
    if (limbs == 0 || groups == 0) return cudaSuccess;
    if (limbs > 65535 || (staged && n % kDiagTile) || few > 3) return cudaErrorInvalidValue;
    switch (nb) {
    case 1:
        return halves ? launch_diag<1, true>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st)
                      : launch_diag<1, false>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st);
    case 2:
        return halves ? launch_diag<2, true>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st)
                      : launch_diag<2, false>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st);
    case 4:
        return halves ? launch_diag<4, true>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st)
                      : launch_diag<4, false>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st);
    case 8:
        return halves ? launch_diag<8, true>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st)
                      : launch_diag<8, false>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st);
    case 16:
        return halves ? launch_diag<16, true>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st)
                      : launch_diag<16, false>(pc, arena, n, limbs, groups, group, job, srcs, unit, stride, accumulate, staged, few, st);
    default: return cudaErrorInvalidValue;
    }
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
__global__ void table_constants_kernel(const u64* __restrict__ v, const u64* __restrict__ m, u64* __restrict__ sp,
                                       u64* __restrict__ tc, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const u64 mod = m[i];
        if (mod == 0) continue;
        const u64 w = v[i] % mod;
        split_constant(w, mod, sp + 4 * i);
        transform_constant(w, mod, tc + 4 * i);
    }
}

cudaError_t launch_table_constants(const u64* v, const u64* m, u64* sp, u64* tc, size_t count, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((count + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    table_constants_kernel<<<blocks, 256, 0, st>>>(v, m, sp, tc, count);
    count_launches(1);
    return cudaGetLastError();
}

__global__ void twiddles_kernel(const u64* __restrict__ raw, const u64* __restrict__ q, ulonglong2* __restrict__ out2,
                                ulonglong2* __restrict__ out2b, uint32_t first_b, uint32_t rows, int log_n) {
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
        if (m >= kFpLimit) out2b[((row - first_b) << log_n) + at] = make_ulonglong2(o[2], o[3]);
    }
}

cudaError_t launch_twiddles(const u64* raw, const u64* q, ulonglong2* out2, ulonglong2* out2b, uint32_t first_b,
                            uint32_t rows, int log_n, cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    const size_t total = (size_t)rows << log_n;
    unsigned blocks = (unsigned)((total + 255) / 256);
    if (blocks > 8192) blocks = 8192;
    twiddles_kernel<<<blocks, 256, 0, st>>>(raw, q, out2, out2b, first_b, rows, log_n);
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
    c.w1ninv = mul_mod(itw[(u64)i * n + 1] % c.q, c.ninv, m);
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

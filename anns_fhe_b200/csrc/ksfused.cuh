// ksfused.cuh -- the whole hybrid key switch in one kernel, N = 2^10 .. 2^16.
//
// Same arithmetic as launch_key_switch (key_switch.cpp:167-439 restated:
// INTT of the input's limbs, fast_bases_conv to each digit's complementary
// primes, NTT, inner product with evk_a / evk_b, approx_mod_down), but one
// polynomial is carried through every step by one CTA (N <= 2^12) or by a
// thread-block cluster of CL CTAs, each holding a slice of the limb being
// transformed (2^12 values and CL = 2, 4, 8 at N = 2^13, 2^14, 2^15; 2^13
// values and CL = 8 at N = 2^16), sixteen values per thread (or eight, see launch_fused):
//
//   phase 0  coef[i] = INTT(in[i]) * qHatInv_i for the input's Q limbs -> lane scratch
//   phase 1  for every special slot k: per digit BConv(coef) + NTT and the
//            products with the key's two halves, summed over the digits; INTT
//            of both sums times PHatInv -> lane scratch
//   phase 2  for every Q limb i: the sums as above (the limb's own digit is
//            the input itself), then for each half BConv of the special limbs
//            to q_i, NTT, (sum - that) * P^-1, plus the fused extras (c0
//            through the automorphism, accumulate), and the store
//
// What bounds it: the multiply and FP64 pipes (the transforms' butterflies),
// then barriers. So:
//   * every product takes its prime's arithmetic of ntt.cuh (FP64 below 2^50,
//     split 32-bit halves above), the base conversions and the constants too;
//     the constants qHatInv and PHatInv are folded into the last inverse
//     stage's N^-1;
//   * the stages across a cluster read and write no shared memory of their
//     own: a forward transform computes its inputs (base conversions read the
//     lane scratch) in columns of CL values, transforms them in registers and
//     scatters them through distributed shared memory; an inverse transform
//     gathers columns from it and stores its results straight to the scratch.
//     Two cluster barriers per slot;
//   * the last forward round (eight adjacent values per thread), the products
//     with the key and the first inverse round run on the same registers;
//   * rounds exchange values within the CTA, 64 or 8 threads, and only those wait
//     for one another.
//
// Shared memory: three padded slices (W for transforms, A0 / A1 for the two
// sums), or two with a single digit (W is A0): 104 or 70 KB per CTA at 2^12 values,
// two CTAs per SM.
//
// The key limbs every CTA of a launch reads are the same, so they come from
// L2. A registered key comes as a prepared copy (key_prep_kernel): pairs in
// the form its prime multiplies by, and in the order the threads read them.
//
// In place is safe: input limb i and the gathered c0 limb i are read at the
// start of slot i of phase 2, and output limb i is written after at least one
// barrier over every CTA of the polynomial that follows those reads.
#pragma once
#include <cooperative_groups.h>

#include "internal.h"

namespace cg = cooperative_groups;

namespace afhe {

namespace ksf {

struct KsFusedArgs {
    // entry z runs at level lvz.at(z) with the tables lvtabs[level] (device
    // copy of the context's per-level tables); lvz unused: all at sizeQl
    const OpTabs* lvtabs;
    ZField lvz;
    int mixed;
    uint32_t sizeQl, K;
    const u64* key;
    u64 evk_a, evk_b;
    uint32_t key_stride, key_pbase;
    u64* arena;
    u64* scratch;
    ZField in, out0, out1, mid;
    KsFuse f;
    const ulonglong2* prep;   // prepared key (evk_a digits, then evk_b digits), or null
    u64 prep_b;               // offset of the evk_b digits in prep
};

// The parts of a slot are functions of their own; inlined unless said otherwise.
#ifndef AFHE_KS_FN
#define AFHE_KS_FN __forceinline__
#endif

// log2 of the values a CTA holds, at ring degree 2^log_n
inline constexpr int slice_bits(int log_n) { return log_n <= 12 ? log_n : (log_n == 16 ? 13 : 12); }

template <int LOGQ, int LOGCL, uint32_t E>
struct Geo {
    static constexpr int LOGN = LOGQ + LOGCL;
    static constexpr uint32_t QN = 1u << LOGQ;
    static constexpr uint32_t CL = 1u << LOGCL;
    static constexpr uint32_t KG = E / 8;             // groups of the rounds' eight values a thread
    static constexpr uint32_t T = QN / E;             // threads
    static constexpr uint32_t PER = QN / CL;          // columns per CTA
    static constexpr uint32_t CPT = E / CL;           // columns per thread
    static constexpr uint32_t PADQ = QN + QN / 16;
    static_assert(CL <= 8 && PER == T * CPT, "a thread's columns hold its values");
    __device__ __forceinline__ static uint32_t rank() {
        if constexpr (LOGCL == 0) return 0;
        else return cg::this_cluster().block_rank();
    }
    // A barrier over the polynomial's CTAs in two halves: what a CTA did to any
    // slice before its arrive is seen after the wait. They alternate strictly.
    __device__ __forceinline__ static void arrive() {
        if constexpr (LOGCL > 0) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    }
    __device__ __forceinline__ static void wait() {
        if constexpr (LOGCL == 0) __syncthreads();
        else asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
    __device__ __forceinline__ static void sync_all() {
        arrive();
        wait();
    }
    // position i < E of this thread's columns: value k = i % CL of column
    // i / CL; global index and index in the slice of CTA k
    __device__ __forceinline__ static uint32_t column(uint32_t i) {
        return rank() * PER + threadIdx.x + (i >> LOGCL) * T;
    }
    __device__ __forceinline__ static u64 column_x(uint32_t i) {
        return (u64)(rank() * PER + threadIdx.x) + ((i & (CL - 1)) * QN + (i >> LOGCL) * T);
    }
    // position i of this thread in a pass over the CTA's own slice, and where
    // it lies in shared memory
    __device__ __forceinline__ static u64 lpos(uint32_t i) { return (u64)threadIdx.x + i * T; }
    __device__ __forceinline__ static uint32_t spos(uint32_t i) { return padix(threadIdx.x) + padix(i * T); }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ u64 ld_cluster(uint32_t addr) {
    u64 v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, u64 v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

// The threads that exchange values between the rounds at bits RB and RB - 3:
// 2^RB consecutive ones (the round at RB writes a block of 2^RB values from
// 2^RB consecutive groups, and the round below reads that block).
template <int RB, uint32_t T>
__device__ __forceinline__ void sync_round() {
    constexpr uint32_t n = 1u << RB;
    if constexpr (n >= T) {
        __syncthreads();
    } else if constexpr (n <= 32) {
        __syncwarp();
    } else {
        static_assert(RB == 6 && T <= 512, "named barriers 1 to 8");
        asm volatile("bar.sync %0, %1;\n" ::"r"(1 + threadIdx.x / n), "r"(n) : "memory");
    }
}

template <class A, bool INV, int LOGQ, int RB, int K, int LOGN, uint32_t E>
struct KsRound {
    typedef NttRound<A, INV, LOGN, 0, LOGQ, 0, false, RB, K, E> R;
};

// Forward rounds from the top of the slice down to bit 3: on entry the slices
// are written and visible, on return this thread's groups of adjacent values are.
template <class A, int LOGQ, int LOGCL, uint32_t E, int NB, int I = 0>
__device__ __forceinline__ void fwd_rounds(u64* const (&bufs)[NB], const TwRow& tw, const typename A::C& c) {
    using G = Geo<LOGQ, LOGCL, E>;
    typedef Rounds<false, LOGQ> R;
    if constexpr (I < R::NR - 1) {
        KsRound<A, false, LOGQ, R::rb(I), R::k(I), G::LOGN, E>::R::template run_n<NB>(bufs, tw, c, nullptr, G::rank(),
                                                                                    I > 0 || LOGCL > 0 ? kEarlier : kResidues, false);
        sync_round<R::rb(I), G::T>();
        fwd_rounds<A, LOGQ, LOGCL, E, NB, I + 1>(bufs, tw, c);
    }
}
// Inverse rounds from bit 3 up: on entry every thread has stored its groups of
// adjacent values; without a cluster fin holds the constants of the transform's
// last stage and the results are canonical residues.
template <class A, int LOGQ, int LOGCL, uint32_t E, int NB, int I = 1>
__device__ __forceinline__ void inv_rounds(u64* const (&bufs)[NB], const TwRow& tw, const typename A::C& c,
                                           const u64* fin) {
    using G = Geo<LOGQ, LOGCL, E>;
    typedef Rounds<true, LOGQ> R;
    if constexpr (I < R::NR) {
        sync_round<R::rb(I), G::T>();
        KsRound<A, true, LOGQ, R::rb(I), R::k(I), G::LOGN, E>::R::template run_n<NB>(bufs, tw, c, fin, G::rank(), kEarlier,
                                                                                LOGCL == 0 && I == R::NR - 1);
        inv_rounds<A, LOGQ, LOGCL, E, NB, I + 1>(bufs, tw, c, fin);
    }
}
template <class A, int LOGQ, int LOGCL, uint32_t E, int NB>
__device__ AFHE_KS_FN void fwd_rounds_call(u64* b0, u64* b1, const PrimeTables* pt, uint32_t prime) {
    const TwRow tw = tw_row<false>(*pt, prime, LOGQ + LOGCL);
    const typename A::C c = A::consts(pt->pc[prime]);
    if constexpr (NB == 2) {
        u64* const two[2] = {b0, b1};
        fwd_rounds<A, LOGQ, LOGCL, E, 2>(two, tw, c);
    } else {
        u64* const one[1] = {b0};
        fwd_rounds<A, LOGQ, LOGCL, E, 1>(one, tw, c);
    }
}
template <class A, int LOGQ, int LOGCL, uint32_t E, int NB>
__device__ AFHE_KS_FN void inv_rounds_call(u64* b0, u64* b1, const PrimeTables* pt, uint32_t prime, const u64* fin) {
    const TwRow tw = tw_row<true>(*pt, prime, LOGQ + LOGCL);
    const typename A::C c = A::consts(pt->pc[prime]);
    if constexpr (NB == 2) {
        u64* const two[2] = {b0, b1};
        inv_rounds<A, LOGQ, LOGCL, E, 2>(two, tw, c, fin);
    } else {
        u64* const one[1] = {b0};
        inv_rounds<A, LOGQ, LOGCL, E, 1>(one, tw, c, fin);
    }
}

// twiddles of the stages across a cluster (bits LOGQ and up): the same for
// every column, at places known at compile time
template <int LOGQ, int LOGN>
struct TwCross {
    TwRow row;
    __device__ __forceinline__ ulonglong2 first(int s, uint32_t m) const { return __ldg(row.a + tw_place(LOGN, LOGQ + s, m)); }
    __device__ __forceinline__ ulonglong2 second(int s, uint32_t m) const { return __ldg(row.b + tw_place(LOGN, LOGQ + s, m)); }
};

// Eight of this thread's positions (8 g .. 8 g + 7: columns over the cluster, or
// its own slice) as the inputs of a forward transform: the stages across the
// cluster in registers, then the values to their slices' W. A barrier over
// the polynomial's CTAs (sync_all) has to follow the last group.
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void fwd_enter(typename A::V* v, uint32_t g, u64* W, const TwRow& tw,
                                          const typename A::C& c) {
    using G = Geo<LOGQ, LOGCL, E>;
    if constexpr (LOGCL == 0) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) W[G::spos(8 * g + i)] = A::store(v[i]);
    } else {
        const TwCross<LOGQ, G::LOGN> cross{tw};
        const uint32_t base = smem_u32(W);
#pragma unroll
        for (uint32_t q = 0; q < 8 / G::CL; ++q) {
            fwd_stages<A, LOGCL>(v + q * G::CL, cross, c, kResidues);
            const uint32_t at = 8 * padix(G::column(8 * g + q * G::CL));
#pragma unroll
            for (uint32_t k = 0; k < G::CL; ++k) st_cluster(map_rank(base, k) + at, A::store(v[q * G::CL + k]));
        }
    }
}

// The end of an inverse transform, for eight positions: inv_gather reads them
// (columns of every CTA's slice of buf), inv_leave runs the stages across the
// cluster; v[i] = the canonical residue at column_x(8 g + i) (at this thread's
// lpos(8 g + i) without a cluster).
template <int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void inv_gather(u64* v, uint32_t g, const u64* buf) {
    using G = Geo<LOGQ, LOGCL, E>;
    if constexpr (LOGCL == 0) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) v[i] = buf[G::spos(8 * g + i)];
    } else {
        const uint32_t base = smem_u32(buf);
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i)
            v[i] = ld_cluster(map_rank(base, i & (G::CL - 1)) + 8 * padix(G::column(8 * g + i)));
    }
}
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void inv_leave(u64* v, const TwRow& tw, const typename A::C& c, const u64* fin) {
    using G = Geo<LOGQ, LOGCL, E>;
    if constexpr (LOGCL > 0) {
        const TwCross<LOGQ, G::LOGN> cross{tw};
#pragma unroll
        for (uint32_t q = 0; q < 8 / G::CL; ++q) {
            typename A::V x[G::CL];
#pragma unroll
            for (uint32_t k = 0; k < G::CL; ++k) x[k] = A::load(v[q * G::CL + k]);
            inv_stages<A, LOGCL>(x, cross, c, true, fin);
#pragma unroll
            for (uint32_t k = 0; k < G::CL; ++k) v[q * G::CL + k] = A::canon_inv(x[k], c);
        }
    }
}
template <int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ u64 leave_x(uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    return LOGCL ? G::column_x(i) : (u64)threadIdx.x + i * G::T;
}

// The eight adjacent values of this thread's group g (at 8 (threadIdx.x + g T)
// in the slice) through the last forward round.
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void fwd_last(typename A::V* v, uint32_t g, const u64* W, const TwRow& tw,
                                         const typename A::C& c) {
    using G = Geo<LOGQ, LOGCL, E>;
    typedef typename KsRound<A, false, LOGQ, 0, 3, G::LOGN, E>::R R;
    const typename R::Group gr = R::group(g, G::rank());
    const u64* const sp = W + padix(gr.base_e);
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) v[j] = A::load(sp[j]);
    R::run_regs(v, tw, gr.blk, c, nullptr, kEarlier, false);
}
// The first inverse round on eight adjacent values, stored to buf.
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void inv_first(typename A::V* v, uint32_t g, u64* buf, const TwRow& tw,
                                          const typename A::C& c) {
    using G = Geo<LOGQ, LOGCL, E>;
    typedef typename KsRound<A, true, LOGQ, 0, 3, G::LOGN, E>::R R;
    const typename R::Group gr = R::group(g, G::rank());
    R::run_regs(v, tw, gr.blk, c, nullptr, kEarlier, false);
    u64* const sp = buf + padix(gr.base_e);
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) sp[j] = A::store(v[j]);
}
// this thread's group g of eight adjacent values, as an offset in a slice
template <int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ uint32_t adjacent(uint32_t g) {
    return padix(8 * (threadIdx.x + g * Geo<LOGQ, LOGCL, E>::T));
}

// gathered position of x: the automorphism's source index, or x itself
__device__ __forceinline__ uint32_t gpos(const uint32_t* map, uint32_t x) { return map ? __ldg(map + x) : x; }

// This entry's rotation (automorphism map, key offset, prepared key).
struct EntryKey {
    const uint32_t* map;
    u64 koff;
    const ulonglong2* prep;
};

__device__ __forceinline__ EntryKey entry_key(const KsFusedArgs& a, uint32_t z) {
    EntryKey k;
    if (a.f.per_z) {
        k.map = (const uint32_t*)a.f.mapz.at(z);
        k.koff = a.f.keyz.at(z);
        k.prep = a.prep ? (const ulonglong2*)a.f.prepz.at(z) : nullptr;
    } else {
        k.map = a.f.map;
        k.koff = 0;
        k.prep = a.prep;
    }
    return k;
}

// Products with key words and the sums of them, per arithmetic. key(): the
// prepared pair times any lazy value; raw(): an unprepared key word; add():
// keeps a sum of products in the range the inverse transform and the ModDown
// combine take (ArFp: within 1/2; ArSp: below q (1 + 2^-17)).
template <class A>
struct KeyMul;
template <>
struct KeyMul<ArFp> {
    static __device__ __forceinline__ double key(double d, const ulonglong2& k, const ArFp::C& c) {
        return fp_mul(d, as_double(k.x), as_double(k.y), c.q);
    }
    static __device__ __forceinline__ double raw(double d, u64 k, const ArFp::C& c, const ModConst& m) {
        return fp_of(mul_mod(ArFp::canon(d, c), k, m));
    }
    static __device__ __forceinline__ double add(double a, double b, const ArFp::C& c) {
        return fp_center(__dadd_rn(a, b), c.q, c.qi);
    }
};
template <>
struct KeyMul<ArSp> {
    static __device__ __forceinline__ u64 key(u64 d, const ulonglong2& k, const ArSp::C& c) {
        return csub(mul_shoup_lazy(d, k.x, k.y, c.q), c.q);
    }
    static __device__ __forceinline__ u64 raw(u64 d, u64 k, const ArSp::C& c, const ModConst& m) {
        return mul_mod(ArSp::canon(d, c), k, m);
    }
    static __device__ __forceinline__ u64 add(u64 a, u64 b, const ArSp::C& c) { return csub(a + b, c.q); }
};

// Base conversion at this thread's positions 8 g .. 8 g + 7: sum over i < size
// of y_i w_i mod q, y_i = src[i stride N + x] (values this thread stored), w_i =
// split constants at tab + 4 i row (any q < 2^61). The products' low words are
// summed mod 2^64 and the quotient by q in doubles rounded down (sp_mul's form
// for a sum), so one reduction serves the whole sum: t in [0, q (1 + 2^-6)).
template <int LOGQ, int LOGCL, uint32_t E>
__device__ __forceinline__ void bconv8(u64* t, uint32_t g, const u64* src, uint32_t stride, uint32_t size,
                                       const u64* __restrict__ tab, uint32_t row, u64 q) {
    using G = Geo<LOGQ, LOGCL, E>;
    const u64 nq = (u64)0 - q;
    double m[8];
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) {
        t[e] = 0;
        m[e] = 0;
    }
    // the next limb's values are on their way while this one's are used
    u64 v[8];
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) v[e] = src[leave_x<LOGQ, LOGCL, E>(8 * g + e)];
#pragma unroll 1
    for (uint32_t i = 0; i < size; ++i) {
        const ulonglong2 w = __ldg((const ulonglong2*)(tab + 4ull * i * row));
        const ulonglong2 s = __ldg((const ulonglong2*)(tab + 4ull * i * row) + 1);
        const double s0 = as_double(s.x), s1 = as_double(s.y);
        const u64* const y = src + ((u64)((i + 1 < size ? i + 1 : i) * stride) << G::LOGN);
        u64 nv[8];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) nv[e] = y[leave_x<LOGQ, LOGCL, E>(8 * g + e)];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) {
            const uint32_t a0 = (uint32_t)v[e], a1 = (uint32_t)(v[e] >> 32);
            m[e] = __fma_rd(__hiloint2double(0, (int)a0), s0, __fma_rd(__hiloint2double(0, (int)a1), s1, m[e]));
            u64 x = mad_wide_u32(a0, (uint32_t)w.x, t[e]);
            x = mad_wide_u32(a1, (uint32_t)w.y, x);
            uint32_t xh = (uint32_t)(x >> 32) + a0 * (uint32_t)(w.x >> 32);
            xh += a1 * (uint32_t)(w.y >> 32);
            t[e] = ((u64)xh << 32) | (uint32_t)x;
            v[e] = nv[e];
        }
    }
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) {
        const double c = __dadd_rd(m[e], kSpRound);
        const uint32_t cl = (uint32_t)__double2loint(c), ch = (uint32_t)__double2hiint(c) - kSpHigh;
        const u64 x = mad_wide_u32(cl, (uint32_t)nq, t[e]);
        uint32_t xh = (uint32_t)(x >> 32) + cl * (uint32_t)(nq >> 32);
        xh += ch * (uint32_t)nq;
        t[e] = ((u64)xh << 32) | (uint32_t)x;
    }
}
// its result as a forward transform's input
__device__ __forceinline__ double bconv_value(u64 t, const ArFp::C&) { return fp_of(t); }
__device__ __forceinline__ u64 bconv_value(u64 t, const ArSp::C&) { return t; }

// The entry a cluster works on. Only its level and table pointer are held;
// the rest is read again where it is used (registers).
template <int LOGQ, int LOGCL, uint32_t E, bool SINGLE>
struct Slot {
    using G = Geo<LOGQ, LOGCL, E>;
    const KsFusedArgs& a;
    const OpTabs* tp;
    uint32_t l;
    __device__ __forceinline__ uint32_t z() const { return blockIdx.x >> LOGCL; }
    __device__ __forceinline__ const OpTabs& t() const { return *tp; }
    __device__ __forceinline__ const PrimeTables* pt() const { return &tp->pt; }
    // 0: W, 1: A0, 2: A1; SINGLE: W is A0
    __device__ __forceinline__ u64* buf(uint32_t i) const {
        extern __shared__ u64 smem[];
        return smem + (SINGLE && i ? i - 1 : i) * G::PADQ;
    }
    __device__ __forceinline__ const u64* in() const { return a.arena + a.in.at(z()); }
    // l limbs of coefficients, then the 2K sums'
    __device__ __forceinline__ u64* coef(uint32_t limb) const {
        return a.scratch + a.mid.at(z()) + ((u64)limb << G::LOGN);
    }
};

// Base conversion of a digit (`size` limbs of coefficients at src, `stride`
// limbs apart; constants at tab, `row` entries apart) into a forward transform
// of prime `prime` in slice W, after the wait that an earlier arrive belongs to
// (wait; not for the second half of a pair).
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ AFHE_KS_FN void convert_enter(const u64* src, uint32_t stride, uint32_t size, const u64* tab, uint32_t row,
                                           u64* W, const PrimeTables* pt, uint32_t prime, bool wait) {
    using G = Geo<LOGQ, LOGCL, E>;
    const PrimeConst* const pcp = pt->pc + prime;
    const typename A::C c = A::consts(*pcp);
    const TwRow tw = tw_row<false>(*pt, prime, G::LOGN);
#pragma unroll 1
    for (uint32_t g = 0; g < G::KG; ++g) {
        u64 b[8];
        bconv8<LOGQ, LOGCL, E>(b, g, src, stride, size, tab, row, pcp->q);
        typename A::V v[8];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) v[e] = bconv_value(b[e], c);
        if (wait && g == 0) G::wait();
        fwd_enter<A, LOGQ, LOGCL, E>(v, g, W, tw, c);
    }
}

// The last forward round of a digit in slice W and its products with the key's
// halves (digit's key limb at offset kofs), on groups of eight adjacent
// positions. Sums go to A0 / A1 (first: nothing there yet), or, with inverse on
// the last digit, straight through the first inverse round.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
__device__ AFHE_KS_FN void last_products(const Slot<LOGQ, LOGCL, E, SINGLE> S, uint32_t prime, u64 kofs, bool first,
                                           bool inverse) {
    using G = Geo<LOGQ, LOGCL, E>;
    constexpr int LOGN = G::LOGN;
    const PrimeConst* const pcp = S.pt()->pc + prime;
    const typename A::C c = A::consts(*pcp);
    const EntryKey ek = entry_key(S.a, S.z());
#pragma unroll 1
    for (uint32_t g = 0; g < G::KG; ++g) {
        typename A::V v[8];
        fwd_last<A, LOGQ, LOGCL, E>(v, g, S.buf(0), tw_row<false>(*S.pt(), prime, LOGN), c);
        const ulonglong2* const kp = ek.prep + kofs + threadIdx.x + g * G::T;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            u64* const Ah = S.buf(1 + h) + adjacent<LOGQ, LOGCL, E>(g);
            typename A::V p[8];
            if (PREP) {
                const ulonglong2* const kh = kp + (h ? 0 : S.a.prep_b);
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) p[e] = KeyMul<A>::key(v[e], __ldg(kh + e * (G::QN / 8)), c);
            } else {
                const ModConst mc = modconst_of(*pcp);
                const u64* const rp = S.a.key + ek.koff + (h ? S.a.evk_a : S.a.evk_b) + kofs +
                                      8 * (threadIdx.x + g * G::T);
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) p[e] = KeyMul<A>::raw(v[e], __ldg(rp + e), c, mc);
            }
            if (!SINGLE && !first) {
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) p[e] = KeyMul<A>::add(p[e], A::load(Ah[e]), c);
            }
            if (SINGLE || inverse) {
                inv_first<A, LOGQ, LOGCL, E>(p, g, S.buf(1 + h), tw_row<true>(*S.pt(), prime, LOGN), c);
            } else {
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) Ah[e] = A::store(p[e]);
            }
        }
    }
}

// One digit's contribution to a slot it does not own (Q limb s < l, or special
// limb s - l): BConv of the digit's coefficients, NTT, products. Enters with an
// arrive that its first store to other CTAs' slices waits for, and leaves with
// one where W is read last (not with inverse).
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
__device__ __forceinline__ void digit_slot(const Slot<LOGQ, LOGCL, E, SINGLE>& S, uint32_t s, uint32_t j, bool first,
                                           bool inverse) {
    using G = Geo<LOGQ, LOGCL, E>;
    const OpTabs& t = S.t();
    const uint32_t l = S.l, K = S.a.K;
    const bool isq = s < l;
    const uint32_t prime = isq ? s : t.p_base + (s - l);
    const uint32_t start = j * t.alpha, size = (j == t.parts - 1) ? l - start : t.alpha;
    const uint32_t kpos = isq ? (s < start ? s : s - size) : (l - size) + (s - l);
    convert_enter<A, LOGQ, LOGCL, E>(S.coef(start), 1, size, t.qhat_modp_sp[j] + 4ull * kpos, l - size + K, S.buf(0), S.pt(),
                                  prime, true);
    G::sync_all();
    fwd_rounds_call<A, LOGQ, LOGCL, E, 1>(S.buf(0), nullptr, S.pt(), prime);
    const uint32_t klimb = isq ? s : S.a.key_pbase + (s - l);
    last_products<A, LOGQ, LOGCL, E, PREP>(S, prime, (((u64)j * S.a.key_stride + klimb) << G::LOGN) + G::rank() * G::QN,
                                        first, inverse);
    if (!(SINGLE || inverse)) G::arrive();
}

// Phase 0, limb i: coef[i] = INTT(input through the automorphism) * qHatInv.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool SINGLE>
__device__ AFHE_KS_FN void input_limb(const Slot<LOGQ, LOGCL, E, SINGLE> S, uint32_t i, u64* buf) {
    using G = Geo<LOGQ, LOGCL, E>;
    constexpr int LOGN = G::LOGN;
    const u64* src = S.in() + ((u64)i << LOGN);
    {
        const uint32_t* const map = entry_key(S.a, S.z()).map;
        uint32_t g[E];
        u64 x[E];
#pragma unroll
        for (uint32_t e = 0; e < E; ++e) g[e] = gpos(map, G::rank() * G::QN + (uint32_t)G::lpos(e));
#pragma unroll
        for (uint32_t e = 0; e < E; ++e) x[e] = src[g[e]];
        residues<E, A::kSecond>(x, S.pt()->pc[i]);
#pragma unroll
        for (uint32_t e = 0; e < E; ++e) buf[G::spos(e)] = A::store(A::of(x[e]));
    }
    __syncthreads();
    const typename A::C c = A::consts(S.pt()->pc[i]);
    const TwRow tw = tw_row<true>(*S.pt(), i, LOGN);
    const u64* const fin = S.t().fin_q + 8ull * i;
#pragma unroll 1
    for (uint32_t g = 0; g < G::KG; ++g) {
        typename A::V v[8];
        const u64* const sp = buf + adjacent<LOGQ, LOGCL, E>(g);
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) v[e] = A::load(sp[e]);
        inv_first<A, LOGQ, LOGCL, E>(v, g, buf, tw, c);
    }
    inv_rounds_call<A, LOGQ, LOGCL, E, 1>(buf, nullptr, S.pt(), i, fin);
    G::sync_all();
    u64* const dst = S.coef(i);
    u64 v[E];
#pragma unroll
    for (uint32_t g = 0; g < G::KG; ++g) inv_gather<LOGQ, LOGCL, E>(v + 8 * g, g, buf);
#pragma unroll
    for (uint32_t g = 0; g < G::KG; ++g) {
        inv_leave<A, LOGQ, LOGCL, E>(v + 8 * g, tw, c, fin);
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) dst[leave_x<LOGQ, LOGCL, E>(8 * g + e)] = v[8 * g + e];
    }
}

// The end of both sums' inverse transforms at special slot k, to the scratch.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool SINGLE>
__device__ AFHE_KS_FN void leave_sums(const Slot<LOGQ, LOGCL, E, SINGLE> S, uint32_t k, const u64* fin) {
    using G = Geo<LOGQ, LOGCL, E>;
    const uint32_t prime = S.t().p_base + k;
    const typename A::C c = A::consts(S.pt()->pc[prime]);
    const TwRow tw = tw_row<true>(*S.pt(), prime, G::LOGN);
    // the next eight positions are on their way while these are transformed
    u64 v[8], nv[8];
    inv_gather<LOGQ, LOGCL, E>(v, 0, S.buf(1));
#pragma unroll 1
    for (uint32_t g = 0; g < 2 * G::KG; ++g) {
        if (g + 1 < 2 * G::KG) inv_gather<LOGQ, LOGCL, E>(nv, (g + 1) >> 1, S.buf(1 + ((g + 1) & 1)));
        inv_leave<A, LOGQ, LOGCL, E>(v, tw, c, fin);
        u64* const dst = S.coef(S.l + 2 * k + (g & 1));
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) {
            dst[leave_x<LOGQ, LOGCL, E>(8 * (g >> 1) + e)] = v[e];
            v[e] = nv[e];
        }
    }
}

// Phase 1, special slot k: both sums' coefficients times PHatInv -> scratch.
// Enters and leaves with an arrive (see digit_slot).
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
__device__ __forceinline__ void special_slot(const Slot<LOGQ, LOGCL, E, SINGLE>& S, uint32_t k) {
    using G = Geo<LOGQ, LOGCL, E>;
    const OpTabs& t = S.t();
    const uint32_t prime = t.p_base + k;
    if (SINGLE) {
        digit_slot<A, LOGQ, LOGCL, E, PREP>(S, S.l + k, 0, true, true);
    } else {
#pragma unroll 1
        for (uint32_t j = 0; j < t.parts; ++j)
            digit_slot<A, LOGQ, LOGCL, E, PREP>(S, S.l + k, j, j == 0, j + 1 == t.parts);
    }
    const u64* const fin = t.fin_p + 8ull * k;
    inv_rounds_call<A, LOGQ, LOGCL, E, 2>(S.buf(1), S.buf(2), S.pt(), prime, fin);
    G::sync_all();
    leave_sums<A, LOGQ, LOGCL, E>(S, k, fin);
    G::arrive();
}

// The ModDown combine at one position: (sum - y) P^-1, plus acc, canonical.
__device__ __forceinline__ u64 moddown_value(double s, double y, const ulonglong2& pinv, const ulonglong2&,
                                             const ArFp::C& c, bool has_acc, u64 acc, u64 q) {
    const u64 r = fp_canon(fp_mul(__dadd_rn(s, -y), as_double(pinv.x), as_double(pinv.y), c.q), c.q);
    return has_acc ? add_mod(r, acc, q) : r;
}
__device__ __forceinline__ u64 moddown_value(u64 s, u64 y, const ulonglong2& pinv, const ulonglong2& pinv2,
                                             const ArSp::C& c, bool has_acc, u64 acc, u64 q) {
    const u64 d = s + 4 * q - csub(y, 3 * q);       // s below q (1 + 2^-6), y below 6.5q
    u64 r = csub(ArSp::mul(d, pinv, pinv2, c), q);
    if (has_acc) r = add_mod(r, acc, q);
    return r;
}

// The input's own digit at Q limb i: the products of the input with the key's
// halves, c0 joining the first as c0 P (it comes out of the product with P^-1).
// OwnGather reads input and c0 at lpos(e0) .. lpos(e0 + 7) through the
// automorphism, own_products makes the products of four of them.
template <class A, int LOGQ, int LOGCL, uint32_t E>
struct OwnGather {
    u64 d[8], cv[8];
    template <bool SINGLE>
    __device__ __forceinline__ void load(const Slot<LOGQ, LOGCL, E, SINGLE>& S, const EntryKey& ek, uint32_t i,
                                         uint32_t e0) {
        using G = Geo<LOGQ, LOGCL, E>;
        const KsFusedArgs& a = S.a;
        const u64* const src = S.in() + ((u64)i << G::LOGN);
        const u64* const cb = a.arena + (a.f.has_c0 ? a.f.c0.at(S.z()) : 0) + ((u64)i << G::LOGN);
        uint32_t g[8];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) g[e] = gpos(ek.map, G::rank() * G::QN + (uint32_t)G::lpos(e0 + e));
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) {
            d[e] = src[g[e]];
            cv[e] = a.f.has_c0 ? cb[g[e]] : 0;
        }
        if (!A::kSecond) {              // (split and 128-bit products take any word)
            residues<8, false>(d, S.pt()->pc[i]);
            residues<8, false>(cv, S.pt()->pc[i]);
        }
    }
};
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
__device__ __forceinline__ void own_products(const Slot<LOGQ, LOGCL, E, SINGLE>& S, const EntryKey& ek, uint32_t i,
                                             uint32_t e0, const u64* d, const u64* cv, typename A::V* p0,
                                             typename A::V* p1, const typename A::C& c) {
    using G = Geo<LOGQ, LOGCL, E>;
    const KsFusedArgs& a = S.a;
    const OpTabs& t = S.t();
    const u64 kofs = ((((u64)(i / t.alpha) * a.key_stride + i) << G::LOGN) + G::rank() * G::QN) + threadIdx.x;
    if (PREP) {
        const ulonglong2* const kp = ek.prep + kofs;
        ulonglong2 kb[4], ka[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            kb[e] = __ldg(kp + a.prep_b + (e0 + e) * G::T);
            ka[e] = __ldg(kp + (e0 + e) * G::T);
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            p0[e] = KeyMul<A>::key(A::of(d[e]), kb[e], c);
            p1[e] = KeyMul<A>::key(A::of(d[e]), ka[e], c);
        }
    } else {
        const ModConst mc = modconst_of(S.pt()->pc[i]);
        const u64* const key = a.key + ek.koff + kofs;
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            p0[e] = A::of(mul_mod(d[e], __ldg(key + a.evk_b + (e0 + e) * G::T), mc));
            p1[e] = A::of(mul_mod(d[e], __ldg(key + a.evk_a + (e0 + e) * G::T), mc));
        }
    }
    if (a.f.has_c0) {
        const ulonglong2* const pm = (const ulonglong2*)(t.p_mod_q + 4ull * i);
        const ulonglong2 pm0 = __ldg(pm), pm1 = A::kSecond ? __ldg(pm + 1) : ulonglong2{};
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) p0[e] = KeyMul<A>::add(p0[e], A::mul(A::of(cv[e]), pm0, pm1, c), c);
    }
}

// BConv of the special limbs of sum h to q_i (approx_mod_down's
// fast_bases_conv) into a forward transform.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool SINGLE>
__device__ __forceinline__ void moddown_enter(const Slot<LOGQ, LOGCL, E, SINGLE>& S, uint32_t i, uint32_t h, u64* W,
                                              bool wait) {
    convert_enter<A, LOGQ, LOGCL, E>(S.coef(S.l + h), 2, S.a.K, S.t().phat_modq_sp + 4ull * i, S.l, W, S.pt(), i, wait);
}
// the last round of a buffer, back in place
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ AFHE_KS_FN void fwd_finish(u64* W, const PrimeTables* pt, uint32_t prime) {
    const TwRow tw = tw_row<false>(*pt, prime, LOGQ + LOGCL);
    const typename A::C c = A::consts(pt->pc[prime]);
#pragma unroll 1
    for (uint32_t g = 0; g < Geo<LOGQ, LOGCL, E>::KG; ++g) {
        typename A::V v[8];
        fwd_last<A, LOGQ, LOGCL, E>(v, g, W, tw, c);
        u64* const sp = W + adjacent<LOGQ, LOGCL, E>(g);
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) sp[e] = A::store(v[e]);
    }
}

// The own digit's products at Q limb i, to A0 / A1.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP>
__device__ AFHE_KS_FN void own_sums(const Slot<LOGQ, LOGCL, E, false> S, uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    const typename A::C c = A::consts(S.pt()->pc[i]);
    const EntryKey ek = entry_key(S.a, S.z());
#pragma unroll 1
    for (uint32_t e0 = 0; e0 < E; e0 += 8) {
        OwnGather<A, LOGQ, LOGCL, E> og;
        og.load(S, ek, i, e0);
#pragma unroll
        for (uint32_t f = 0; f < 8; f += 4) {
            typename A::V p0[4], p1[4];
            own_products<A, LOGQ, LOGCL, E, PREP>(S, ek, i, e0 + f, og.d + f, og.cv + f, p0, p1, c);
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) {
                S.buf(1)[G::spos(e0 + f + e)] = A::store(p0[e]);
                S.buf(2)[G::spos(e0 + f + e)] = A::store(p1[e]);
            }
        }
    }
}
// ModDown combine of half h at Q limb i, to the output.
template <class A, int LOGQ, int LOGCL, uint32_t E>
__device__ AFHE_KS_FN void combine_half(const Slot<LOGQ, LOGCL, E, false> S, uint32_t i, uint32_t h) {
    using G = Geo<LOGQ, LOGCL, E>;
    const KsFusedArgs& a = S.a;
    const typename A::C c = A::consts(S.pt()->pc[i]);
    const u64 q = S.pt()->pc[i].q;
    const u64 x0 = ((u64)i << G::LOGN) + G::rank() * G::QN + threadIdx.x;
    u64* const out = a.arena + (h ? a.out1 : a.out0).at(S.z()) + x0;
    const u64* const acc = a.arena + (a.f.has_acc ? (h ? a.f.acc1 : a.f.acc0).at(S.z()) + x0 : 0);
    const ulonglong2* const pi = (const ulonglong2*)(S.t().p_inv_tc + 4ull * i);
    const ulonglong2 pi0 = __ldg(pi), pi1 = A::kSecond ? __ldg(pi + 1) : ulonglong2{};
#pragma unroll 1
    for (uint32_t e0 = 0; e0 < E; e0 += 8) {
        u64 ex[8];
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) ex[e] = a.f.has_acc ? acc[(e0 + e) * G::T] : 0;
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e)
            out[(e0 + e) * G::T] = moddown_value(A::load(S.buf(1 + h)[G::spos(e0 + e)]),
                                                 A::load(S.buf(0)[G::spos(e0 + e)]), pi0, pi1, c, a.f.has_acc != 0,
                                                 ex[e], q);
    }
}

// Phase 2, Q limb i. Enters and leaves with an arrive (see digit_slot).
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP>
__device__ __forceinline__ void output_limb(const Slot<LOGQ, LOGCL, E, false>& S, uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    const uint32_t own = i / S.t().alpha, parts = S.t().parts;
    own_sums<A, LOGQ, LOGCL, E, PREP>(S, i);
    // (the barriers of the next transform come before the sums are read)
#pragma unroll 1
    for (uint32_t j = 0; j < parts; ++j)
        if (j != own) digit_slot<A, LOGQ, LOGCL, E, PREP>(S, i, j, false, false);
#pragma unroll 1
    for (uint32_t h = 0; h < 2; ++h) {
        moddown_enter<A, LOGQ, LOGCL, E>(S, i, h, S.buf(0), true);
        G::sync_all();
        fwd_rounds_call<A, LOGQ, LOGCL, E, 1>(S.buf(0), nullptr, S.pt(), i);
        fwd_finish<A, LOGQ, LOGCL, E>(S.buf(0), S.pt(), i);
        __syncthreads();
        combine_half<A, LOGQ, LOGCL, E>(S, i, h);
        G::arrive();
    }
}

// The combine of both halves with a single digit: the limb's own products are
// formed here (input and c0 gathered once), the results stay in the slices.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP>
__device__ AFHE_KS_FN void combine_both(const Slot<LOGQ, LOGCL, E, true> S, uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    const typename A::C c = A::consts(S.pt()->pc[i]);
    const u64 q = S.pt()->pc[i].q;
    const EntryKey ek = entry_key(S.a, S.z());
    const ulonglong2* const pi = (const ulonglong2*)(S.t().p_inv_tc + 4ull * i);
    const ulonglong2 pi0 = __ldg(pi), pi1 = A::kSecond ? __ldg(pi + 1) : ulonglong2{};
#pragma unroll 1
    for (uint32_t e0 = 0; e0 < E; e0 += 8) {
        OwnGather<A, LOGQ, LOGCL, E> og;
        og.load(S, ek, i, e0);
#pragma unroll
        for (uint32_t f = 0; f < 8; f += 4) {
            typename A::V p0[4], p1[4];
            own_products<A, LOGQ, LOGCL, E, PREP>(S, ek, i, e0 + f, og.d + f, og.cv + f, p0, p1, c);
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) {
                u64& r0 = S.buf(1)[G::spos(e0 + f + e)];
                u64& r1 = S.buf(2)[G::spos(e0 + f + e)];
                r0 = moddown_value(p0[e], A::load(r0), pi0, pi1, c, false, 0, q);
                r1 = moddown_value(p1[e], A::load(r1), pi0, pi1, c, false, 0, q);
            }
        }
    }
}
template <int LOGQ, int LOGCL, uint32_t E>
__device__ AFHE_KS_FN void store_both(const Slot<LOGQ, LOGCL, E, true> S, uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    const KsFusedArgs& a = S.a;
    const u64 q = S.pt()->pc[i].q;
    const u64 x0 = ((u64)i << G::LOGN) + G::rank() * G::QN + threadIdx.x;
#pragma unroll 1
    for (uint32_t h = 0; h < 2; ++h) {
        u64* const out = a.arena + (h ? a.out1 : a.out0).at(S.z()) + x0;
        const u64* const acc = a.arena + (a.f.has_acc ? (h ? a.f.acc1 : a.f.acc0).at(S.z()) + x0 : 0);
#pragma unroll 1
        for (uint32_t e0 = 0; e0 < E; e0 += 8) {
            u64 ex[8];
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e) ex[e] = a.f.has_acc ? acc[(e0 + e) * G::T] : 0;
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e) {
                const u64 r = S.buf(1 + h)[G::spos(e0 + e)];
                out[(e0 + e) * G::T] = a.f.has_acc ? add_mod(r, ex[e], q) : r;
            }
        }
    }
}

// Phase 2 with a single digit: both halves' transforms side by side in the two
// slices. The outputs wait in the slices for a barrier over the polynomial's
// CTAs, since they may lie where another CTA gathers from.
template <class A, int LOGQ, int LOGCL, uint32_t E, bool PREP>
__device__ __forceinline__ void output_limb(const Slot<LOGQ, LOGCL, E, true>& S, uint32_t i) {
    using G = Geo<LOGQ, LOGCL, E>;
    moddown_enter<A, LOGQ, LOGCL, E>(S, i, 0, S.buf(1), true);
    moddown_enter<A, LOGQ, LOGCL, E>(S, i, 1, S.buf(2), false);
    G::sync_all();
    fwd_rounds_call<A, LOGQ, LOGCL, E, 2>(S.buf(1), S.buf(2), S.pt(), i);
    fwd_finish<A, LOGQ, LOGCL, E>(S.buf(1), S.pt(), i);
    fwd_finish<A, LOGQ, LOGCL, E>(S.buf(2), S.pt(), i);
    __syncthreads();
    combine_both<A, LOGQ, LOGCL, E, PREP>(S, i);
    G::sync_all();
    store_both(S, i);
    G::arrive();
}

// SINGLE (one digit at every entry's level): two slices instead of three, which
// leaves the L1 cache another 70 KB. Two CTAs per SM either way (128 registers a
// thread): three of SINGLE's would fit the shared memory, but at 80 registers
// the split arithmetic spills and the L1 that is left no longer holds the
// twiddles (N = 2^15, 2 + 4 limbs, 240 ciphertexts: 2.87 ms against 2.34).
inline constexpr int ks_min_ctas(uint32_t threads) { return (int)(512u / threads); }

template <int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
__global__ void __launch_bounds__(Geo<LOGQ, LOGCL, E>::T, ks_min_ctas(Geo<LOGQ, LOGCL, E>::T))
    ks_fused_kernel(const __grid_constant__ KsFusedArgs a) {
    using G = Geo<LOGQ, LOGCL, E>;
    const uint32_t l = a.mixed ? (uint32_t)a.lvz.at(blockIdx.x >> LOGCL) : a.sizeQl;
    const Slot<LOGQ, LOGCL, E, SINGLE> S{a, a.lvtabs + l, l};
    const OpTabs& t = S.t();
    // limbs alternate between two slices: a limb's gather from every CTA may
    // still run while the next one is loaded
#pragma unroll 1
    for (uint32_t i = 0; i < l; ++i) {
        u64* const buf = S.buf(1 + (i & 1));
        if (S.pt()->pc[i].fp) input_limb<ArFp, LOGQ, LOGCL, E>(S, i, buf);
        else input_limb<ArSp, LOGQ, LOGCL, E>(S, i, buf);
    }
    G::arrive();
    // a thread reads back only the coefficients it stored itself
#pragma unroll 1
    for (uint32_t k = 0; k < a.K; ++k) {
        if (S.pt()->pc[t.p_base + k].fp) special_slot<ArFp, LOGQ, LOGCL, E, PREP>(S, k);
        else special_slot<ArSp, LOGQ, LOGCL, E, PREP>(S, k);
    }
    if constexpr (!SINGLE) {        // A0 / A1 are written before the next wait: the last gathers from them
        G::wait();
        G::arrive();
    }
#pragma unroll 1
    for (uint32_t i = 0; i < l; ++i) {
        if (S.pt()->pc[i].fp) output_limb<ArFp, LOGQ, LOGCL, E, PREP>(S, i);
        else output_limb<ArSp, LOGQ, LOGCL, E, PREP>(S, i);
    }
    G::wait();
}

template <int LOGQ, bool SINGLE>
constexpr size_t fused_smem() { return (SINGLE ? 2ull : 3ull) * ((1u << LOGQ) + (1u << LOGQ) / 16) * sizeof(u64); }

template <int LOGQ, int LOGCL, uint32_t E, bool PREP, bool SINGLE>
cudaError_t launch_fused_v(const KsFusedArgs& a, uint32_t nz, cudaStream_t st) {
    constexpr uint32_t T = Geo<LOGQ, LOGCL, E>::T;
    auto kern = ks_fused_kernel<LOGQ, LOGCL, E, PREP, SINGLE>;
    constexpr size_t smem = fused_smem<LOGQ, SINGLE>();
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if constexpr (LOGCL == 0) {
        kern<<<nz, T, smem, st>>>(a);
    } else {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(nz << LOGCL, 1, 1);
        cfg.blockDim = dim3(T, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << LOGCL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, a);
        if (e != cudaSuccess) return e;
    }
    count_launches(1);
    return cudaGetLastError();
}

// Values per thread: sixteen. Where one CTA carries a ciphertext, eight in launches of
// up to half a wave: as many CTAs as fit at once then have twice the threads, and a
// thread half the chain (rotations, us, 16 / 8: N = 2^10, three digits, 120: 120 / 65;
// N = 2^11, two, 74: 88 / 56; N = 2^12, three, 148: 189 / 135; past half a wave, N =
// 2^12, 260: 261 / 304, N = 2^11, two, 592: 150 / 160).
template <int LOGQ, int LOGCL, bool PREP, bool SINGLE>
cudaError_t launch_fused(const KsFusedArgs& a, uint32_t nz, cudaStream_t st) {
    if constexpr (LOGCL == 0) {
        if (2 * nz <= (uint32_t)key_switch_fused_capacity(LOGQ)) return launch_fused_v<LOGQ, LOGCL, 8, PREP, SINGLE>(a, nz, st);
    }
    return launch_fused_v<LOGQ, LOGCL, 16, PREP, SINGLE>(a, nz, st);
}

// Launches by ring degree, one source file each (ksfused_single.cu, _multi.cu,
// _raw.cu): prepared keys with one digit, prepared keys, unprepared keys.
cudaError_t launch_single(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st);
cudaError_t launch_multi(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st);
cudaError_t launch_raw(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st);
int capacity(int log_n);

// f<LOGQ, LOGCL> for the ring degree
#define AFHE_KS_BY_DEGREE(log_n, f, otherwise) \
    switch (log_n) {                           \
    case 10: return f(10, 0);                  \
    case 11: return f(11, 0);                  \
    case 12: return f(12, 0);                  \
    case 13: return f(12, 1);                  \
    case 14: return f(12, 2);                  \
    case 15: return f(12, 3);                  \
    case 16: return f(13, 3);                  \
    default: return otherwise;                 \
    }

}  // namespace ksf

}  // namespace afhe

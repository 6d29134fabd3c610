// ntt.cuh -- negacyclic NTT / INTT passes for sm_100a.
//
// Computes exactly the transforms of hardware_fpga_model/hls/src/ntt.cpp:
//   forward (ntt.cpp:4-43): Cooley-Tukey, stage with block size t = 2^p uses
//     twiddle tw[N/2^(p+1) + (x >> (p+1))]; natural order in, bit-reversed out;
//   inverse (ntt.cpp:46-80): Gentleman-Sande with itw[...] on the same index,
//     stages in the opposite order, then x N^-1 (fused into the last stage here).
// Every butterfly is an exact operation mod q, so with the same twiddle tables
// the canonical outputs are bit-identical to the reference's.
//
// Layout: a limb is N contiguous uint64 words (limb-major ciphertexts). A
// transform is 1 or 2 passes; a pass covers the butterfly bits
// [lo_bit, lo_bit + P) of the coefficient index:
//   * column pass (lo_bit > 0): a CTA owns 2^logC adjacent low-index columns of
//     the 2^P rows, i.e. 2^P row segments of 2^logC * 8 bytes (coalesced);
//   * chunk pass (lo_bit == 0): a CTA owns 2^logC contiguous chunks of 2^P words.
// The butterflies run in rounds of up to three consecutive stages on eight
// values held in registers (radix-8), exchanged through shared memory between
// rounds.
//
// Arithmetic. The 64-bit Shoup butterfly is bound by the multiply pipe (one
// 64 x 64 high product and two low ones, about ten 32-bit multiplies of which
// six are wide: 2.7 butterflies per clock per SM in registers alone on B200).
// Two cheaper exact forms replace it, picked per prime:
//   * q < 2^50: residues are whole numbers held in doubles (ArFp). B200 has a
//     full-rate FP64 pipe (64 FMA per clock per SM); a product by a constant
//     is a rounded quotient and two exact FMA remainders, 6 operations, and
//     sums need no reduction for several stages: 6.8 butterflies per clock
//     per SM;
//   * larger q (< 2^61): the operand is split into 32-bit halves, each with
//     its own multiple of the constant mod q, so that the quotient is below 2^33
//     and everything but three wide products is a low product (ArSp): 3.3 to 3.7
//     butterflies per clock per SM.
#pragma once
#include <cstdint>
#include "modarith.cuh"

namespace afhe {

// Host-side count of kernels this library has launched (all contexts).
void count_launches(uint64_t k);

// Primes below this take the floating-point arithmetic (ArFp), others the
// split one (ArSp).
constexpr u64 kFpLimit = 1ull << 50;

// A modulus' constants (64 bytes): what sums and products of words need.
struct PrimeBase {
    u64 q;
    u64 r64, r64_sh, one_sh;  // reduce128 constants
    u64 fp;                   // q < kFpLimit
    double qd, qi;            // q and 1/q as doubles (fp)
    u64 over;                 // the bits above q's own
};
// Per-prime constants of the transforms (144 bytes). The arrays are in the form the
// prime's transforms use (see transform_constant).
struct PrimeConst : PrimeBase {
    u64 ninv, w1ninv;         // N^-1 mod q, itw[1] * N^-1 (fused last inverse stage)
    u64 nv[4], w1nv[4];       // the same as transform constants
};

// A constant w mod q as a transform multiplies by it:
//   fp:  o[0] = w centred in (-q/2, q/2], o[1] = that over q (bits of doubles);
//   else o[0] = w, o[1] = w 2^32 mod q, and (o[2], o[3]) = (w, o[1]) / q
//        rounded down to 52 fractional bits, times 2^1000 (bits of doubles).
// (w / q) 2^52 rounded down is the top 52 bits of the Shoup companion. The
// second form alone (any q < 2^61): split_constant.
AFHE_HD u64 bits_of(double x) {
#if defined(__CUDA_ARCH__)
    return (u64)__double_as_longlong(x);
#else
    union { double d; u64 u; } v;
    v.d = x;
    return v.u;
#endif
}
AFHE_HD void split_constant(u64 w, u64 q, u64* o) {
    const u64 sh = shoup_companion(w, q);
    const u64 w1 = (w << 32) - (sh >> 32) * q;          // w 2^32 mod q
    o[0] = w;
    o[1] = w1;
    const double s = 0x1p948;                 // 2^-52 2^1000
    o[2] = bits_of((double)(sh >> 12) * s);
    o[3] = bits_of((double)(shoup_companion(w1, q) >> 12) * s);
}
AFHE_HD void transform_constant(u64 w, u64 q, u64* o) {
    if (q < kFpLimit) {
        const double c = w > (q >> 1) ? -(double)(q - w) : (double)w;
        o[0] = bits_of(c);
        o[1] = bits_of(c / (double)q);
        o[2] = o[3] = 0;
    } else {
        split_constant(w, q, o);
    }
}
AFHE_HD void set_transform_constants(PrimeConst& c) {
    c.fp = c.q < kFpLimit ? 1 : 0;
    c.qd = (double)c.q;
    c.qi = 1.0 / c.qd;
    c.over = ~0ull;
    while (c.q & c.over) c.over <<= 1;
    transform_constant(c.ninv, c.q, c.nv);
    transform_constant(c.w1ninv, c.q, c.w1nv);
}

// One table set: primes [0, count) with twiddles for each, as transform
// constants: the first pair in tw2 / itw2, the second (ArSp primes) in tw2b /
// itw2b. A row holds its N twiddles in the order the rounds read them: the
// stages [R, R + K) of a round (R a multiple of 3, K = min(3, log N - R))
// take, for block b of x >> (R + K), entries nb (1 + slot) + b, nb =
// N >> (R + K), slot = tw_slot(K, s, m) for stage R + s and m of its
// 2^(K - 1 - s) twiddles in the block: neighbouring threads read neighbouring
// entries (the natural order has a stage's twiddles for one block together,
// 16-byte pieces 64 bytes apart across a warp).
struct PrimeTables {
    const PrimeConst* pc;    // [count]
    const ulonglong2* tw2;   // [count][N] forward
    const ulonglong2* itw2;  // [count][N] inverse
    const ulonglong2* tw2b;
    const ulonglong2* itw2b;
};
AFHE_HD constexpr uint32_t tw_slot(int k, int s, uint32_t m) { return ((1u << k) >> (s + 1)) - 1 + m; }
// place of the twiddle of stage p, block c = x >> (p + 1)
AFHE_HD constexpr uint32_t tw_place(int log_n, int p, uint32_t c) {
    const int R = p / 3 * 3, K = log_n - R < 3 ? log_n - R : 3, s = p - R, low = K - 1 - s;
    return (((1u << log_n) >> (R + K)) * (1 + tw_slot(K, s, c & ((1u << low) - 1)))) + (c >> low);
}

AFHE_HD ModConst modconst_of(const PrimeBase& p) {
    ModConst m;
    m.q = p.q; m.r64 = p.r64; m.r64_sh = p.r64_sh; m.one_sh = p.one_sh;
    return m;
}

// A unit of NTT work: one limb. Word offsets: `src` is read by the prologue,
// `dst` holds the limb between passes (relative to the `mid` base), `out` is
// written by the epilogue; `prime` indexes the table set; `aux` is free for
// prologue / epilogue functors (e.g. a digit or output-limb index).
struct LimbJob {
    u64 src;
    u64 dst;
    u64 out;
    uint32_t prime;
    uint32_t aux;
};

struct NttGeom {
    int log_n;
    int lo_bit;   // first butterfly bit of this pass
    int P;        // number of butterfly bits in this pass
    int log_c;    // log2 of tiles per CTA
};

// Word offset of one operand for polynomial z of a batched launch:
//   (arr ? arr[z >> shift] : base + (z >> shift) * stride) + add + (z & low) * hdelta,
// low = 2^shift - 1. A regular batch (operands at a fixed stride) needs no
// memory; an irregular one reads a small device array. shift = 1 describes the
// two polynomials (c0, c1) of ciphertext z >> 1 that differ by hdelta.
struct ZField {
    const u64* arr;
    u64 base, stride, add, hdelta;
    uint32_t shift;
    AFHE_HD u64 at(uint32_t z) const {
        const uint32_t zz = z >> shift;
        const u64 v = arr ? arr[zz] : base + (u64)zz * stride;
        return v + add + (u64)(z & ((1u << shift) - 1u)) * hdelta;
    }
};

inline ZField zf_const(u64 v) { ZField f{}; f.base = v; return f; }
inline ZField zf_stride(u64 base, u64 stride) { ZField f{}; f.base = base; f.stride = stride; return f; }
inline ZField zf_plus(ZField f, u64 add) { f.add += add; return f; }
// entries z0 and on (of a field without zf_pair)
inline ZField zf_skip(ZField f, uint32_t z0) {
    if (f.arr) f.arr += z0;
    else f.base += (u64)z0 * f.stride;
    return f;
}
inline ZField zf_pair(ZField f, u64 hdelta) { f.shift = 1; f.hdelta = hdelta; return f; }

// The operands of one batched launch: meaning of src / out / aux is the
// prologue's and epilogue's; mid is where a limb lives between the passes of
// a two-pass transform (in the `mid` arena).
struct ZBases {
    ZField src, mid, out, aux;
};

// x mod q, any x
__device__ __forceinline__ u64 residue(u64 x, const PrimeBase& pc) {
    return x < pc.q ? x : csub(mul_shoup_lazy(x, 1, pc.one_sh, pc.q), pc.q);
}
// Words from outside as residues: one branch, rarely taken, behind all their
// loads. Unless EXACT, words below the next power of two (so below 2q) stay as
// they are.
template <int M, bool EXACT>
__device__ __forceinline__ void residues(u64* v, const PrimeBase& pc) {
    u64 bits = 0;
    bool words = false;
#pragma unroll
    for (int i = 0; i < M; ++i) {
        if (EXACT) words |= v[i] >= pc.q;
        else bits |= v[i];
    }
    if (EXACT ? words : (bits & pc.over) != 0) {
#pragma unroll
        for (int i = 0; i < M; ++i) v[i] = residue(v[i], pc);
    }
}

// Plain prologues / epilogue. Words of outside (kWords) may be no residues: a
// transform takes them below 4q forward and below 2q inverse, by its bounds alone
// (checking the words before their use keeps loads and arithmetic apart, which
// costs 13% of a forward transform at N = 2^16).
struct LoadPlain {
    static constexpr bool kMany = false;      // one value a call
    static constexpr bool kWords = true;
    const u64* base;
    __device__ __forceinline__ u64 operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x,
                                              const PrimeConst&) const {
        return base[zb.src.at(z) + j.src + x];
    }
};
struct LoadResidue : LoadPlain {
    static constexpr bool kWords = false;
};
struct StorePlain {
    u64* base;
    __device__ __forceinline__ void operator()(const LimbJob& j, const ZBases& zb, uint32_t z, u64 x, u64 v,
                                               const PrimeConst&) const {
        base[zb.out.at(z) + j.out + x] = v;
    }
};

__device__ __forceinline__ double as_double(u64 v) { return __longlong_as_double((long long)v); }
__device__ __forceinline__ u64 as_bits(double v) { return (u64)__double_as_longlong(v); }

// ---- q < 2^50: whole numbers in doubles -------------------------------------
// Bounds are in units of q. A product by a centred constant of a value of
// magnitude A <= 4 is within 1/2 + A/16: the quotient a w / q, |a w / q| <=
// 2^51, is rounded to a whole number with an error of 1/2 plus a (w/q) 2^-53
// for the constant's own rounding; h + l = a w exactly (FMA), and h - c q is a
// whole number below 2^53, so the FMA that forms it is exact too. Sums are
// exact below 8q <= 2^53. A centred value is within 1/2.
constexpr double kFpRound = 0x1.8p52;    // adding and subtracting it rounds to a whole number (|x| <= 2^51)

__device__ __forceinline__ double fp_mul(double a, double w, double wq, double q) {
    const double c = __dadd_rn(__fma_rn(a, wq, kFpRound), -kFpRound);
    const double h = __dmul_rn(a, w);
    const double l = __fma_rn(a, w, -h);
    return __dadd_rn(__fma_rn(-c, q, h), l);
}
__device__ __forceinline__ double fp_center(double x, double q, double qi) {
    const double c = __dadd_rn(__fma_rn(x, qi, kFpRound), -kFpRound);
    return __fma_rn(-c, q, x);
}
// canonical residue <-> double (x < 2^52)
__device__ __forceinline__ double fp_of(u64 x) { return __dadd_rn(as_double(x | 0x4330000000000000ull), -0x1p52); }
__device__ __forceinline__ u64 fp_canon(double x, double q) {     // |x| <= q - 1
    const double y = x < 0 ? __dadd_rn(x, q) : x;
    return as_bits(__dadd_rn(y, 0x1p52)) & 0x000fffffffffffffull;
}

struct ArFp {
    typedef double V;
    struct C { double q, qi; };
    static __device__ __forceinline__ C consts(const PrimeConst& pc) { return C{pc.qd, pc.qi}; }
    static __device__ __forceinline__ V load(u64 bits) { return as_double(bits); }
    static __device__ __forceinline__ u64 store(V v) { return as_bits(v); }
    static __device__ __forceinline__ V of(u64 canonical) { return fp_of(canonical); }
    // a word below 4q, less 2q
    static __device__ __forceinline__ V outside(u64 word, const C& c) {
        return __dadd_rn(as_double(word | 0x4330000000000000ull), -__fma_rn(2, c.q, 0x1p52));
    }
    static __device__ __forceinline__ V mul(V a, const ulonglong2& w, const ulonglong2&, const C& c) {
        return fp_mul(a, as_double(w.x), as_double(w.y), c.q);
    }
    static constexpr bool kSecond = false;      // no second twiddle pair
    // forward output (any lazy value) to its canonical residue
    static __device__ __forceinline__ u64 canon(V v, const C& c) { return fp_canon(fp_center(v, c.q, c.qi), c.q); }
    // inverse output after the last stage's product
    static __device__ __forceinline__ u64 canon_inv(V v, const C& c) { return fp_canon(v, c.q); }
};

// ---- q < 2^61: split products -------------------------------------------------
// a w mod q for any a = a1 2^32 + a0: t = a0 W0 + a1 W1 - c q (W1 = w 2^32 mod
// q), c = floor(a0 W0 / q + a1 W1 / q) < 2^33 or one less where the fraction is
// below 2^-18, so t in [0, q (1 + 2^-18)), computed mod 2^64. The quotient is
// formed in doubles rounded down: the halves enter as denormals (their 32 bits
// in the low word of a zero double: no conversion), times constants scaled by
// 2^1000, so c lands in the low 33 bits of 2^-22 + c 2^-74; the exponent bits
// above it are taken off by the sum's starting value.
constexpr double kSpRound = 0x1p-22;
constexpr uint32_t kSpHigh = 0x3E900000u;       // high word of kSpRound
__device__ __forceinline__ u64 mad_wide_u32(uint32_t a, uint32_t b, u64 c) {
    u64 d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
// nq = 2^64 - q; start = sp_start(nq)
__device__ __forceinline__ u64 sp_start(u64 nq) { return (u64)(0u - kSpHigh * (uint32_t)nq) << 32; }
__device__ __forceinline__ u64 sp_mul(u64 a, u64 w0, u64 w1, double s0, double s1, u64 nq, u64 start) {
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32);
    const double c = __dadd_rd(__fma_rd(__hiloint2double(0, (int)a0), s0, __dmul_rd(__hiloint2double(0, (int)a1), s1)),
                               kSpRound);
    const uint32_t cl = (uint32_t)__double2loint(c), ch = (uint32_t)__double2hiint(c);
    u64 t = mad_wide_u32(a0, (uint32_t)w0, start);
    t = mad_wide_u32(a1, (uint32_t)w1, t);
    t = mad_wide_u32(cl, (uint32_t)nq, t);
    uint32_t th = (uint32_t)(t >> 32) + a0 * (uint32_t)(w0 >> 32);
    th += a1 * (uint32_t)(w1 >> 32);
    th += cl * (uint32_t)(nq >> 32);
    th += ch * (uint32_t)nq;
    return ((u64)th << 32) | (uint32_t)t;
}

// A canonical residue times a constant (transform_constant's form), canonical.
__device__ __forceinline__ u64 mul_tc(u64 a, const u64* __restrict__ k, const PrimeConst& pc) {
    const ulonglong2 w = __ldg((const ulonglong2*)k);
    if (pc.fp) return fp_canon(fp_mul(fp_of(a), as_double(w.x), as_double(w.y), pc.qd), pc.qd);
    const ulonglong2 s = __ldg((const ulonglong2*)k + 1);
    const u64 nq = (u64)0 - pc.q;
    return csub(sp_mul(a, w.x, w.y, as_double(s.x), as_double(s.y), nq, sp_start(nq)), pc.q);
}
// The product of two canonical residues below 2^50, in (-0.76q, 0.76q): the
// quotient from the rounded product is off by less than 0.76, the rest is exact.
__device__ __forceinline__ double fp_mul2(double a, double b, double q, double qi) {
    const double h = __dmul_rn(a, b);
    const double l = __fma_rn(a, b, -h);
    const double c = __dadd_rn(__fma_rn(h, qi, kFpRound), -kFpRound);
    return __dadd_rn(__fma_rn(-c, q, h), l);
}

// The product of any two words, canonical: in doubles where both are residues
// of a prime below 2^50, else 128 bits and their reduction.
__device__ __forceinline__ u64 mul_words(u64 a, u64 b, const PrimeBase& pc) {
    if (pc.fp && a < pc.q && b < pc.q) return fp_canon(fp_mul2(fp_of(a), fp_of(b), pc.qd, pc.qi), pc.qd);
    return mul_mod(a, b, modconst_of(pc));
}

// Base conversions of M values at a time: o[e] = sum over i < size of y(i, e) w_i
// mod q, canonical, w_i = split constants at tab + 4 i row (any q < 2^61). The
// products' low words are summed mod 2^64 and the quotient by q in doubles
// rounded down (sp_mul's form for a sum), so one reduction serves the whole sum
// (a Shoup product for each term costs 2.5 times the multiplier's cycles).
template <int M, class Y>
__device__ __forceinline__ void bconv(u64* o, uint32_t size, const u64* __restrict__ tab, uint32_t row, u64 q, Y&& y) {
    const u64 nq = (u64)0 - q;
    double m[M];
    u64 t[M];
#pragma unroll
    for (uint32_t e = 0; e < M; ++e) {
        t[e] = 0;
        m[e] = 0;
    }
#pragma unroll 1
    for (uint32_t i = 0; i < size; ++i) {
        const ulonglong2 w = __ldg((const ulonglong2*)(tab + 4ull * i * row));
        const ulonglong2 s = __ldg((const ulonglong2*)(tab + 4ull * i * row) + 1);
        const double s0 = as_double(s.x), s1 = as_double(s.y);
        u64 v[M];
#pragma unroll
        for (uint32_t e = 0; e < M; ++e) v[e] = y(i, e);
#pragma unroll
        for (uint32_t e = 0; e < M; ++e) {
            const uint32_t a0 = (uint32_t)v[e], a1 = (uint32_t)(v[e] >> 32);
            m[e] = __fma_rd(__hiloint2double(0, (int)a0), s0, __fma_rd(__hiloint2double(0, (int)a1), s1, m[e]));
            u64 x = mad_wide_u32(a0, (uint32_t)w.x, t[e]);
            x = mad_wide_u32(a1, (uint32_t)w.y, x);
            uint32_t xh = (uint32_t)(x >> 32) + a0 * (uint32_t)(w.x >> 32);
            xh += a1 * (uint32_t)(w.y >> 32);
            t[e] = ((u64)xh << 32) | (uint32_t)x;
        }
    }
#pragma unroll
    for (uint32_t e = 0; e < M; ++e) {
        const double c = __dadd_rd(m[e], kSpRound);
        const uint32_t cl = (uint32_t)__double2loint(c), ch = (uint32_t)__double2hiint(c) - kSpHigh;
        const u64 x = mad_wide_u32(cl, (uint32_t)nq, t[e]);
        uint32_t xh = (uint32_t)(x >> 32) + cl * (uint32_t)(nq >> 32);
        xh += ch * (uint32_t)nq;
        o[e] = csub(((u64)xh << 32) | (uint32_t)x, q);
    }
}

// Values between rounds: forward below 6.5q and at least 0.49q (or canonical,
// entering the first round), inverse canonical or a product (below q (1 + 2^-18)).
// A forward round brings the half that its first stage does not multiply into
// [0.49q, 3.5q) and then only adds: x + t and x - t + q (t < q (1 + 2^-18), so
// the lower bound falls by 2^-18 q a stage), below 6.5q after three stages
// (6.5 2^61 < 2^64).
struct ArSp {
    typedef u64 V;
    struct C { u64 q, nq, start; };
    static __device__ __forceinline__ C consts(const PrimeConst& pc) {
        const u64 nq = (u64)0 - pc.q;
        return C{pc.q, nq, sp_start(nq)};
    }
    static __device__ __forceinline__ V load(u64 bits) { return bits; }
    static __device__ __forceinline__ u64 store(V v) { return v; }
    static __device__ __forceinline__ V of(u64 canonical) { return canonical; }
    static __device__ __forceinline__ V outside(u64 word, const C&) { return word; }
    static __device__ __forceinline__ V mul(V a, const ulonglong2& w, const ulonglong2& s, const C& c) {
        return sp_mul(a, w.x, w.y, as_double(s.x), as_double(s.y), c.nq, c.start);
    }
    static constexpr bool kSecond = true;
    // a forward value below 6.5q into [0.49q, 3.5q) where it was at least 0.49q
    static __device__ __forceinline__ u64 low(u64 v, const C& c) {
        const u64 q3 = 3 * c.q;
        return v >= q3 + (c.q >> 1) ? v - q3 : v;
    }
    static __device__ __forceinline__ u64 canon(V v, const C& c) {
        return csub(csub(low(v, c), c.q << 1), c.q);
    }
    static __device__ __forceinline__ u64 canon_inv(V v, const C& c) { return csub(v, c.q); }
};

// K forward stages (bits high to low) on 2^K values: y = value 2^s apart times
// its twiddle, (x + y, x - y). tw.first(s, m), tw.second(s, m): the constants of
// twiddle m of stage s. from: what the inputs are: residues (below q (1 + 2^-6));
// words below 4q (A::outside); values of an earlier round.
enum Inputs { kResidues, kOutside, kEarlier };
template <class A, int K, int NB = 1, class Tw>
__device__ __forceinline__ void fwd_stages(typename A::V* v, const Tw& tw, const typename A::C& c, Inputs from) {
    constexpr uint32_t NK = 1u << K;
    // the half that the first stage does not multiply
#pragma unroll
    for (uint32_t b = 0; b < NB; ++b) {
#pragma unroll
        for (uint32_t j = 0; j < NK / 2; ++j) {
            typename A::V& x = v[b * NK + j];
            if constexpr (A::kSecond) {
                x = from == kEarlier ? A::low(x, c) : from == kOutside ? A::low(x + c.q, c) : x + c.q;
            } else {
                // the bound grows by less than 0.75 a stage: 1/2 (1, 2) -> at most 2.8 (4) after three
                if (from == kEarlier) x = fp_center(x, c.q, c.qi);
            }
        }
    }
#pragma unroll
    for (int s = K - 1; s >= 0; --s) {
#pragma unroll
        for (uint32_t m = 0; m < (NK >> (s + 1)); ++m) {
            const ulonglong2 ww = tw.first(s, m), w2w = A::kSecond ? tw.second(s, m) : ulonglong2{};
#pragma unroll
            for (uint32_t b = 0; b < NB; ++b) {
#pragma unroll
                for (uint32_t jj = 0; jj < (1u << s); ++jj) {
                    const uint32_t at = b * NK + ((m << (s + 1)) | jj);
                    typename A::V &x = v[at], &y = v[at + (1u << s)];
                    const typename A::V t = A::mul(y, ww, w2w, c);
                    if constexpr (A::kSecond) {
                        y = x - t + c.q;
                        x = x + t;
                    } else {
                        y = __dadd_rn(x, -t);
                        x = __dadd_rn(x, t);
                    }
                }
            }
        }
    }
}

// K inverse stages (bits low to high): (x + y, (x - y) times the twiddle). Inputs
// and outputs within 1 (canonical, products, reduced sums; inputs from outside
// within 2, which is as well within ArFp's exact range): the bounds are
// tracked per value (they fold away when unrolled), and a sum is brought down
// only where it could pass 2 before another stage of the round (ArSp: 4, by
// 2q), or 1 at the end. last: the last stage multiplies its sums and
// differences by the two constants at fin_consts (4 words each) instead: N^-1
// and itw[1] N^-1 (PrimeConst::nv, w1nv), or those times a constant that follows
// the transform.
template <class A, int K, int NB = 1, class Tw>
__device__ __forceinline__ void inv_stages(typename A::V* v, const Tw& tw, const typename A::C& c, bool last,
                                           const u64* fin_consts, Inputs from = kEarlier) {
    constexpr uint32_t NK = 1u << K;
    float bound[NK];
#pragma unroll
    for (uint32_t j = 0; j < NK; ++j) bound[j] = A::kSecond && from == kOutside ? 2.0f : 1.0f;
#pragma unroll
    for (int s = 0; s < K; ++s) {
#pragma unroll
        for (uint32_t m = 0; m < (NK >> (s + 1)); ++m) {
            ulonglong2 ww{}, w2w{};
            const bool fin = last && s == K - 1;
            if (!fin) {
                ww = tw.first(s, m);
                if (A::kSecond) w2w = tw.second(s, m);
            }
#pragma unroll
            for (uint32_t jj = 0; jj < (1u << s); ++jj) {
                const uint32_t ix = (m << (s + 1)) | jj, iy = ix + (1u << s);
                const float bx = bound[ix], by = bound[iy], sum = bx + by;
#pragma unroll
                for (uint32_t b = 0; b < NB; ++b) {
                    typename A::V &x = v[b * NK + ix], &y = v[b * NK + iy];
                    typename A::V u, d;
                    if constexpr (A::kSecond) {
                        // products exceed q by 2^-18 of it, and sums of them
                        // their bound by at most q / 4: the next whole q above
                        u = x + y;
                        d = x - y + (u64)(by + 1.0f) * c.q;
                    } else {
                        u = __dadd_rn(x, y);
                        d = __dadd_rn(x, -y);
                    }
                    if (fin) {
                        const ulonglong2* k = (const ulonglong2*)fin_consts;
                        x = A::mul(u, __ldg(k), A::kSecond ? __ldg(k + 1) : ulonglong2{}, c);
                        y = A::mul(d, __ldg(k + 2), A::kSecond ? __ldg(k + 3) : ulonglong2{}, c);
                    } else {
                        y = A::mul(d, ww, w2w, c);
                        bound[ix] = sum;
                        if constexpr (A::kSecond) {
                            bound[iy] = 1.0f;
                            if (sum > 2.0f) {
                                u = csub(u, 2 * c.q);
                                bound[ix] = 2.0f;
                            }
                            if (s == K - 1) {
                                u = csub(u, c.q);
                                bound[ix] = 1.0f;
                            }
                        } else {
                            bound[iy] = 0.5f + sum / 16;
                            if (sum > (s == K - 1 ? 1.0f : 2.0f)) {
                                u = fp_center(u, c.q, c.qi);
                                bound[ix] = 0.5f;
                            }
                        }
                        x = u;
                    }
                }
            }
        }
    }
}

// Shared-memory layout: one pad word per 16 words, so the strided patterns of
// every round (8-byte elements, strides 1, 2, 8, 16, 64, ...) hit distinct banks.
__device__ __forceinline__ uint32_t padix(uint32_t e) { return e + (e >> 4); }

// One prime's twiddle rows.
struct TwRow {
    const ulonglong2* __restrict__ a;
    const ulonglong2* __restrict__ b;
};
template <bool INV>
__device__ __forceinline__ TwRow tw_row(const PrimeTables& pt, uint32_t prime, int log_n) {
    const u64 at = (u64)prime << log_n;
    return INV ? TwRow{pt.itw2 + at, pt.itw2b + at} : TwRow{pt.tw2 + at, pt.tw2b + at};
}

// A group's twiddles where they lie: entries NB (1 + slot) + blk of the row
// (see PrimeTables), of a table round of KR stages of which K are done. The
// number of blocks NB is known at compile time, so a thread's twiddles are one
// address and constant offsets.
template <int K, int KR, uint32_t NB>
struct TwAt {
    const ulonglong2* __restrict__ a;       // row + blk
    const ulonglong2* __restrict__ b;
    uint32_t blk;                           // (K < KR)
    __device__ __forceinline__ TwAt(const TwRow& row, uint32_t block) {
        a = row.a + (K == KR ? block : 0);
        b = row.b + (K == KR ? block : 0);
        blk = block;
    }
    __device__ __forceinline__ uint32_t at(int s, uint32_t m) const {
        if constexpr (K == KR) {
            return NB * (1 + tw_slot(K, s, m));
        } else {
            const uint32_t c = (blk << (K - 1 - s)) | m;
            const int low = KR - 1 - s;
            return NB * (1 + tw_slot(KR, s, c & ((1u << low) - 1))) + (c >> low);
        }
    }
    __device__ __forceinline__ ulonglong2 first(int s, uint32_t m) const { return __ldg(a + at(s, m)); }
    __device__ __forceinline__ ulonglong2 second(int s, uint32_t m) const { return __ldg(b + at(s, m)); }
};
// The same held in registers (ArFp: 28 of them), loaded before the values
// they multiply. ArSp constants are twice as wide and are loaded stage by
// stage instead.
template <int K>
struct TwHeld {
    ulonglong2 w[(1 << K) - 1];
    template <class At>
    __device__ __forceinline__ TwHeld(const At& t, bool skip_last) {
#pragma unroll
        for (int s = 0; s < K; ++s) {
            if (skip_last && s == K - 1) continue;
#pragma unroll
            for (uint32_t m = 0; m < ((1u << K) >> (s + 1)); ++m) w[tw_slot(K, s, m)] = t.first(s, m);
        }
    }
    __device__ __forceinline__ const ulonglong2& first(int s, uint32_t m) const { return w[tw_slot(K, s, m)]; }
    __device__ __forceinline__ ulonglong2 second(int, uint32_t) const { return ulonglong2{}; }
};

// One round: K consecutive stages on bits [RB, RB + K) of the pass index.
// Each of the TILE / EPT threads holds EPT values per round, as EPT / 2^K
// groups of 2^K; all shapes are compile-time (ring degree 2^LOGN, pass from
// bit LO). The table's round that starts at bit LO + RB has KR stages, K of
// which are done here.
template <class A, bool INV, int LOGN, int LO, int P, int LOGC, bool COL, int RB, int K, int EPT>
struct NttRound {
    typedef typename A::V V;
    static constexpr uint32_t C = 1u << LOGC;
    static constexpr uint32_t T = (1u << (P + LOGC)) / EPT;
    static constexpr uint32_t NK = 1u << K;
    static constexpr uint32_t GROUPS = EPT >> K;
    static constexpr uint32_t STEP_E = COL ? (1u << (RB + LOGC)) : (1u << RB);
    static constexpr u64 STEP_X = 1ull << (LO + RB);     // between a group's values in the limb
    static constexpr int KR = LOGN - LO - RB < 3 ? LOGN - LO - RB : 3;
    typedef TwAt<K, KR, (1u << (LOGN - LO - RB - KR))> Tw;

    struct Group {
        uint32_t base_e;    // the group's first element in the tile
        uint32_t blk;       // x >> (lo_bit + RB + K): the index bits above the round
    };
    __device__ __forceinline__ static Group group(uint32_t gi, uint32_t tile0) {
        const uint32_t r = threadIdx.x + gi * T;
        uint32_t c, brest;
        if (COL) { c = r & (C - 1u); brest = r >> LOGC; }
        else { brest = r & ((1u << (P - K)) - 1u); c = r >> (P - K); }
        const uint32_t base_b = ((brest >> RB) << (RB + K)) | (brest & ((1u << RB) - 1u));
        const uint32_t hb = COL ? 0u : (tile0 + c);     // index bits above the pass
        return Group{COL ? ((base_b << LOGC) | c) : ((c << P) | base_b), (hb << (P - RB - K)) | (brest >> RB)};
    }
    __device__ __forceinline__ static uint32_t element(const Group& g, uint32_t j) { return g.base_e + j * STEP_E; }

    template <int NB, class W>
    __device__ __forceinline__ static void stages(V* v, const W& tw, const typename A::C& c, const u64* fin,
                                                  Inputs from, bool last) {
        if constexpr (INV) inv_stages<A, K, NB>(v, tw, c, last, fin, from);
        else fwd_stages<A, K, NB>(v, tw, c, from);
    }

    // NB sets of values in registers, twiddles from where they lie
    template <int NB = 1>
    __device__ __forceinline__ static void run_regs(V* v, const TwRow& row, uint32_t blk, const typename A::C& c,
                                                    const u64* fin, Inputs from, bool last) {
        const Tw at(row, blk);
        if constexpr (A::kSecond) {
            stages<NB>(v, at, c, fin, from, last);
        } else {
            const TwHeld<K> held(at, INV && last);
            stages<NB>(v, held, c, fin, from, last);
        }
    }

    // The round over NB buffers of the same prime in shared memory: each
    // group's twiddles and addresses serve every buffer. from: where the values
    // come from; last: the round holds the
    // transform's last stage (inverse), and the values are stored as canonical
    // residues.
    template <int NB>
    __device__ __forceinline__ static void run_n(u64* const (&sms)[NB], const TwRow& tw, const typename A::C& c,
                                                 const u64* fin, uint32_t tile0, Inputs from, bool last) {
#pragma unroll(K == 3 ? 1 : GROUPS)      // (whole groups one after another: code size, registers)
        for (uint32_t gi = 0; gi < GROUPS; ++gi) {
            const Group g = group(gi, tile0);
            // base_e has zeros where j * STEP_E has ones, so
            // padix(base_e + j * STEP_E) = padix(base_e) + padix(j * STEP_E):
            // one address per group, compile-time offsets per element
            V v[NB * NK];
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (uint32_t j = 0; j < NK; ++j) v[b * NK + j] = A::load(sms[b][padix(g.base_e) + padix(j * STEP_E)]);
            run_regs<NB>(v, tw, g.blk, c, fin, from, last);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (uint32_t j = 0; j < NK; ++j)
                    sms[b][padix(g.base_e) + padix(j * STEP_E)] =
                        (INV && last) ? A::canon_inv(v[b * NK + j], c) : A::store(v[b * NK + j]);
        }
    }
};

// Rounds of a pass of P bits: at bits 0, 3, 6, ..., the last one with what is
// left. Round i of a direction: forward takes them from the top down.
template <bool INV, int P>
struct Rounds {
    static constexpr int NR = (P + 2) / 3;
    static constexpr int rb(int i) { return 3 * (INV ? i : NR - 1 - i); }
    static constexpr int k(int i) { return P - rb(i) < 3 ? P - rb(i) : 3; }
};

// Rounds [FROM, TO) of a pass over NB tiles in shared memory (same prime),
// each followed by a barrier. from0: what the first of the pass's rounds reads;
// finish: the pass ends the transform
// (inverse).
template <class A, bool INV, int LOGN, int LO, int P, int LOGC, bool COL, int FROM, int TO, int EPT, int NB>
__device__ __forceinline__ void ntt_rounds_n(u64* const (&sms)[NB], const TwRow& tw, const typename A::C& c,
                                             const u64* fin, uint32_t tile0, Inputs from0, bool finish) {
    if constexpr (FROM < TO) {
        typedef Rounds<INV, P> R;
        NttRound<A, INV, LOGN, LO, P, LOGC, COL, R::rb(FROM), R::k(FROM), EPT>::template run_n<NB>(
            sms, tw, c, fin, tile0, FROM > 0 ? kEarlier : from0, finish && FROM == R::NR - 1);
        __syncthreads();
        ntt_rounds_n<A, INV, LOGN, LO, P, LOGC, COL, FROM + 1, TO, EPT, NB>(sms, tw, c, fin, tile0, from0, finish);
    }
}

// One pass over 2^(P + LOGC)-word tiles, EPT values per thread (8 or 16). The
// first round of a pass takes its values straight from memory (through the
// prologue on the first pass) and the last round writes its results straight
// back (through the epilogue on the last pass) wherever neighbouring threads
// hold neighbouring elements in that round; the round at bit 0 of a chunk pass
// (eight adjacent elements per thread) goes through shared memory instead.
// CTAs are sized for 64 registers a thread whatever their thread count.
constexpr uint32_t ntt_threads(int P, int LOGC, int EPT) { return (1u << (P + LOGC)) / EPT; }
constexpr int ntt_min_ctas(int P, int LOGC, int EPT) { return (int)(1024 / ntt_threads(P, LOGC, EPT)); }

template <class A, bool INV, int LOGN, int LO, int P, int LOGC, int EPT, class Pro, class Epi>
__device__ __forceinline__ void ntt_pass(u64* sm, const PrimeTables& pt, const LimbJob& job, u64* __restrict__ mid,
                                         const ZBases& zb, const Pro& pro, const Epi& epi) {
    typedef Rounds<INV, P> R;
    constexpr bool COL = LO > 0;
    constexpr uint32_t C = 1u << LOGC;
    constexpr uint32_t TILE = 1u << (P + LOGC);
    constexpr uint32_t T = TILE / EPT;
    constexpr int NR = R::NR;
    // the pass at the top of the index runs first forward, last inverse
    constexpr bool TOP = LO + P == LOGN, first = INV ? LO == 0 : TOP, last = INV ? TOP : LO == 0;
    static_assert(NR >= 2, "a pass has a first and a last round");
    constexpr bool DIRECT_IN = COL || R::rb(0) > 0, DIRECT_OUT = COL || R::rb(NR - 1) > 0;
    constexpr Inputs FROM = !first ? kEarlier : Pro::kWords ? kOutside : kResidues;
    const uint32_t z = blockIdx.z;
    u64* const mp = mid + zb.mid.at(z) + job.dst;
    PrimeConst pc = pt.pc[job.prime];
    pc.fp = A::kSecond ? 0 : 1;             // (known where prologue and epilogue branch on it)
    const u64* const fin = pt.pc[job.prime].nv;
    const typename A::C c = A::consts(pc);
    const TwRow tw = tw_row<INV>(pt, job.prime, LOGN);
    const uint32_t tile0 = blockIdx.x << LOGC;

    auto gidx = [&](uint32_t e) -> u64 {
        if (!COL) return ((u64)tile0 << P) + e;
        const uint32_t b = e >> LOGC, col = e & (C - 1u);
        return ((u64)b << LO) + tile0 + col;
    };
    auto fetch = [&](u64 x) -> u64 {
        if constexpr (first && !Pro::kMany) {
            const u64 w = pro(job, zb, z, x, pc);
            return A::store(FROM == kOutside && !INV ? A::outside(w, c) : A::of(w));
        }
        else return mp[x];
    };
    auto put = [&](u64 x, u64 v, bool canonical) {
        if constexpr (last) epi(job, zb, z, x, canonical ? v : A::canon(A::load(v), c), pc);
        else mp[x] = v;
    };

    if constexpr (DIRECT_IN) {
        typedef NttRound<A, INV, LOGN, LO, P, LOGC, COL, R::rb(0), R::k(0), EPT> Rd;
#pragma unroll
        for (uint32_t gi = 0; gi < Rd::GROUPS; ++gi) {
            const typename Rd::Group gr = Rd::group(gi, tile0);
            const u64 x = gidx(gr.base_e);
            typename A::V v[Rd::NK];
            if constexpr (first && Pro::kMany) {
                constexpr uint32_t M = Rd::NK < 4 ? Rd::NK : 4;
#pragma unroll
                for (uint32_t j = 0; j < Rd::NK; j += M) {
                    u64 o[M];
                    pro.template many<M>(o, job, zb, z, x + j * Rd::STEP_X, Rd::STEP_X, pc);
#pragma unroll
                    for (uint32_t i = 0; i < M; ++i) v[j + i] = A::of(o[i]);
                }
            } else {
#pragma unroll
                for (uint32_t j = 0; j < Rd::NK; ++j) v[j] = A::load(fetch(x + j * Rd::STEP_X));
            }
            Rd::run_regs(v, tw, gr.blk, c, fin, FROM, false);
            u64* const sp = sm + padix(gr.base_e);
#pragma unroll
            for (uint32_t j = 0; j < Rd::NK; ++j) sp[padix(j * Rd::STEP_E)] = A::store(v[j]);
        }
        __syncthreads();
    } else {
        static_assert(!Pro::kMany, "a prologue of several values needs a first round from memory");
        const u64 x = gidx(threadIdx.x);
#pragma unroll 8
        for (uint32_t k = 0; k < EPT; ++k) sm[padix(threadIdx.x) + padix(k * T)] = fetch(x + (u64)k * T);
        __syncthreads();
    }
    u64* const one[1] = {sm};
    ntt_rounds_n<A, INV, LOGN, LO, P, LOGC, COL, DIRECT_IN ? 1 : 0, DIRECT_OUT ? NR - 1 : NR, EPT, 1>(
        one, tw, c, fin, tile0, FROM, last);
    if constexpr (DIRECT_OUT) {
        typedef NttRound<A, INV, LOGN, LO, P, LOGC, COL, R::rb(NR - 1), R::k(NR - 1), EPT> Rd;
#pragma unroll
        for (uint32_t gi = 0; gi < Rd::GROUPS; ++gi) {
            const typename Rd::Group gr = Rd::group(gi, tile0);
            const u64 x = gidx(gr.base_e);
            typename A::V v[Rd::NK];
            const u64* const sp = sm + padix(gr.base_e);
#pragma unroll
            for (uint32_t j = 0; j < Rd::NK; ++j) v[j] = A::load(sp[padix(j * Rd::STEP_E)]);
            Rd::run_regs(v, tw, gr.blk, c, fin, kEarlier, last);
#pragma unroll
            for (uint32_t j = 0; j < Rd::NK; ++j)
                put(x + j * Rd::STEP_X, (INV && last) ? A::canon_inv(v[j], c) : A::store(v[j]), INV && last);
        }
    } else {
        const u64 x = gidx(threadIdx.x);
#pragma unroll 8
        for (uint32_t k = 0; k < EPT; ++k) put(x + (u64)k * T, sm[padix(threadIdx.x) + padix(k * T)], INV && last);
    }
}

template <bool INV, int LOGN, int LO, int P, int LOGC, int EPT, class Pro, class Epi>
__global__ void __launch_bounds__(ntt_threads(P, LOGC, EPT), ntt_min_ctas(P, LOGC, EPT))
ntt_kernel(const PrimeTables pt, const LimbJob* __restrict__ jobs, u64* __restrict__ mid, const ZBases zb,
           const Pro pro, const Epi epi) {
    extern __shared__ u64 sm[];
    const LimbJob job = jobs[blockIdx.y];
    if (pt.pc[job.prime].fp) ntt_pass<ArFp, INV, LOGN, LO, P, LOGC, EPT>(sm, pt, job, mid, zb, pro, epi);
    else ntt_pass<ArSp, INV, LOGN, LO, P, LOGC, EPT>(sm, pt, job, mid, zb, pro, epi);
}

// Tile shapes of a transform ("plans"), chosen per ring degree at run time
// (afhe_ntt_set_plan; the autotuner times them). Every plan computes the
// same butterflies on the same values, so the residues do not depend on it.
//   N <= 2^13, one pass over the whole limb: plan 0 the default values per
//     thread (16 for 8192-word limbs, else 8), plan 1 the other choice;
//   N >= 2^14, two passes (bits 9 and up in columns, then bits 0-8 in chunks:
//     whole radix-8 rounds): plan = 3 * t + c: columns per CTA 2^{5, 4, 6}[c]
//     in the column pass, chunk-pass tiles of 2^{12, 13}[t] words. Plan 0 is
//     32 columns and 4096-word tiles.
// Values per thread in a two-pass transform: 16 for 8192-word tiles, else 8.
constexpr int kNttPlansOnePass = 2;
constexpr int kNttPlansTwoPass = 6;
inline int ntt_plan_count(int log_n) {
    return log_n < 10 || log_n > 16 ? 0 : (log_n <= 13 ? kNttPlansOnePass : kNttPlansTwoPass);
}
// the plan in force per log_n, process-wide (kernels.cu)
int ntt_plan(int log_n);
void set_ntt_plan(int log_n, int plan);

struct NttPlan {
    int npass;
    int ept[2];
    NttGeom g[2];
};

inline NttPlan make_plan(int log_n, bool inverse, int plan) {
    NttPlan pl;
    if (log_n <= 13) {   // whole limb in shared memory (<= 68 KB)
        pl.npass = 1;
        NttGeom a{};
        a.log_n = log_n; a.lo_bit = 0; a.P = log_n; a.log_c = 0;
        pl.g[0] = a;
        const int def = log_n >= 13 ? 16 : 8;
        pl.ept[0] = plan == 1 ? 24 - def : def;
        return pl;
    }
    static const int col_c[3] = {5, 4, 6};
    const int c = col_c[plan % 3], tl = 12 + plan / 3;
    const int pb = 9;             // low (chunk) pass bits
    const int pa = log_n - pb;    // high (column) pass bits
    NttGeom col{}, chk{};
    col.log_n = log_n; col.lo_bit = pb; col.P = pa; col.log_c = c;
    chk.log_n = log_n; chk.lo_bit = 0; chk.P = pb; chk.log_c = tl - pb;
    const int ept_col = pa + c >= 13 ? 16 : 8, ept_chk = tl >= 13 ? 16 : 8;
    pl.npass = 2;
    if (!inverse) { pl.g[0] = col; pl.g[1] = chk; pl.ept[0] = ept_col; pl.ept[1] = ept_chk; }
    else { pl.g[0] = chk; pl.g[1] = col; pl.ept[0] = ept_chk; pl.ept[1] = ept_col; }
    return pl;
}

template <bool INV, int LOGN, int LO, int P, int LOGC, int EPT, class Pro, class Epi>
inline cudaError_t launch_pass(const PrimeTables& pt, const LimbJob* jobs, uint32_t njobs, uint32_t nz, u64* mid,
                               const ZBases& zb, const Pro& pro, const Epi& epi, cudaStream_t st) {
    constexpr uint32_t TILE = 1u << (P + LOGC);
    const uint32_t ctas = 1u << (LOGN - P - LOGC);
    const size_t smem = (size_t)(TILE + TILE / 16) * sizeof(u64);
    auto kern = ntt_kernel<INV, LOGN, LO, P, LOGC, EPT, Pro, Epi>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<dim3(ctas, njobs, nz), ntt_threads(P, LOGC, EPT), smem, st>>>(pt, jobs, mid, zb, pro, epi);
    count_launches(1);
    return cudaSuccess;
}

// The pass with geometry g and EPT values per thread, dispatched to its
// compile-time instance (every shape some plan uses).
template <bool INV, class Pro, class Epi>
inline cudaError_t launch_shape(const NttGeom& g, int ept, const PrimeTables& pt, const LimbJob* jobs,
                                uint32_t njobs, uint32_t nz, u64* mid, const ZBases& zb, const Pro& pro,
                                const Epi& epi, cudaStream_t st) {
#define AFHE_NTT_SHAPE(N_, LO_, P_, C_, EPT_)                                                        \
    if (g.log_n == N_ && g.lo_bit == LO_ && g.P == P_ && g.log_c == C_ && ept == EPT_)               \
        return launch_pass<INV, N_, LO_, P_, C_, EPT_>(pt, jobs, njobs, nz, mid, zb, pro, epi, st);
    // one pass
    AFHE_NTT_SHAPE(10, 0, 10, 0, 8) AFHE_NTT_SHAPE(10, 0, 10, 0, 16)
    AFHE_NTT_SHAPE(11, 0, 11, 0, 8) AFHE_NTT_SHAPE(11, 0, 11, 0, 16)
    AFHE_NTT_SHAPE(12, 0, 12, 0, 8) AFHE_NTT_SHAPE(12, 0, 12, 0, 16)
    AFHE_NTT_SHAPE(13, 0, 13, 0, 8) AFHE_NTT_SHAPE(13, 0, 13, 0, 16)
    // two passes: columns (bits 9 and up; 16, 32 or 64 per CTA), then 512-word
    // chunks (8 or 16 per CTA)
    AFHE_NTT_SHAPE(14, 9, 5, 4, 8) AFHE_NTT_SHAPE(14, 9, 5, 5, 8) AFHE_NTT_SHAPE(14, 9, 5, 6, 8)
    AFHE_NTT_SHAPE(15, 9, 6, 4, 8) AFHE_NTT_SHAPE(15, 9, 6, 5, 8) AFHE_NTT_SHAPE(15, 9, 6, 6, 8)
    AFHE_NTT_SHAPE(16, 9, 7, 4, 8) AFHE_NTT_SHAPE(16, 9, 7, 5, 8) AFHE_NTT_SHAPE(16, 9, 7, 6, 16)
    AFHE_NTT_SHAPE(14, 0, 9, 3, 8) AFHE_NTT_SHAPE(14, 0, 9, 4, 16)
    AFHE_NTT_SHAPE(15, 0, 9, 3, 8) AFHE_NTT_SHAPE(15, 0, 9, 4, 16)
    AFHE_NTT_SHAPE(16, 0, 9, 3, 8) AFHE_NTT_SHAPE(16, 0, 9, 4, 16)
#undef AFHE_NTT_SHAPE
    return cudaErrorInvalidValue;
}

// Launch a full transform over `njobs` limbs x `nz` polynomials. Between
// passes limb `job` of polynomial z lives at mid + zb.mid[z] + job.dst.
template <bool INV, class Pro, class Epi>
inline cudaError_t launch_ntt(int log_n, const PrimeTables& pt, const LimbJob* jobs, uint32_t njobs, uint32_t nz,
                              u64* mid, const ZBases& zb, Pro pro, Epi epi, cudaStream_t st) {
    if (njobs == 0 || nz == 0) return cudaSuccess;
    NttPlan pl = make_plan(log_n, INV, ntt_plan(log_n));
    for (int i = 0; i < pl.npass; ++i) {
        cudaError_t e = launch_shape<INV>(pl.g[i], pl.ept[i], pt, jobs, njobs, nz, mid, zb, pro, epi, st);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace afhe

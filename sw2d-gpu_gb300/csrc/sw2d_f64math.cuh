// sw2d_f64math.cuh -- double-precision helpers for a GPU whose FP64 pipe is
// the scarce unit (one FP64 warp instruction occupies a scheduler's pipe for
// 64 cycles, an integer or FP32 one for one or two).
//
// Every helper returns the bits of the plain IEEE expression it stands for
// (division, square root, comparison, the deterministic power of the
// friction term); it only takes fewer FP64 instructions for them.  What a
// helper's fast form does not cover (subnormals, infinities, NaN, operands
// near the ends of the exponent range) falls through to the plain expression.
// They compile on the host too, where the tests
// compare them with the plain expressions.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SW2D_HD __host__ __device__ __forceinline__
#else
#define SW2D_HD inline
#endif

namespace sw2d {

constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;

SW2D_HD unsigned long long d_bits(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
SW2D_HD double d_from_bits(unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
SW2D_HD unsigned d_hi(double x) { return (unsigned)(d_bits(x) >> 32); }
SW2D_HD unsigned d_lo(double x) { return (unsigned)d_bits(x); }
SW2D_HD double d_make(unsigned hi, unsigned lo) { return d_from_bits(((unsigned long long)hi << 32) | lo); }
SW2D_HD double d_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
SW2D_HD float f_from_bits(unsigned b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}
SW2D_HD unsigned f_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    unsigned b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
// FP32 seeds: 1/x and 1/sqrt(x) to about 22 bits (any approximation that good
// gives the same final bits; see the users).  On the host SW2D_SEED_ULPS puts
// them off by that many FP32 ulps, so that a test covers the device's.
#ifndef SW2D_SEED_ULPS
#define SW2D_SEED_ULPS 0
#endif
SW2D_HD float f_rcp_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return f_from_bits(f_bits(1.0f / x) + (SW2D_SEED_ULPS));
#endif
}
SW2D_HD float f_rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return f_from_bits(f_bits(1.0f / std::sqrt(x)) + (SW2D_SEED_ULPS));
#endif
}

// ---- comparisons and selections on the bits ---------------------------------

// x >= c for a constant c > 0 (or c == +0 with x not -0), false for NaN
SW2D_HD bool d_ge_pos(double x, unsigned long long cbits) {
    return d_bits(x) - cbits <= kInfBits - cbits;  // in [c, inf] as unsigned
}
SW2D_HD bool d_gt_zero(double x) { return d_bits(x) - 1ull < kInfBits; }
SW2D_HD bool d_lt_zero(double x) { return d_bits(x) - 0x8000000000000001ull < kInfBits; }
SW2D_HD bool d_is_zero(double x) { return (d_bits(x) << 1) == 0ull; }
SW2D_HD bool d_is_nan(double x) { return (d_bits(x) & 0x7fffffffffffffffull) > kInfBits; }
SW2D_HD bool d_is_finite(double x) { return (d_hi(x) & 0x7ff00000u) != 0x7ff00000u; }
// a < b, false when either is NaN; -0 equals +0
SW2D_HD bool d_lt(double a, double b) {
    const long long x = (long long)d_bits(a), y = (long long)d_bits(b);
    const long long m = (long long)0x8000000000000000ull;
    const long long kx = x < 0 ? (long long)((unsigned long long)m - (unsigned long long)x) : x;
    const long long ky = y < 0 ? (long long)((unsigned long long)m - (unsigned long long)y) : y;
    return kx < ky && !d_is_nan(a) && !d_is_nan(b);
}
// fmax(x, 0) with NaN -> 0, as +0 for x <= 0
SW2D_HD double d_clamp0(double x) { return d_bits(x) <= kInfBits ? x : 0.0; }

// 0.5 * x
SW2D_HD double d_half(double x) {
    const unsigned hi = d_hi(x), e = hi & 0x7ff00000u;
    if (e - 0x00200000u < 0x7fd00000u) return d_make(hi - 0x00100000u, d_lo(x));  // exponent field 2 .. 2046
    return d_is_zero(x) ? x : 0.5 * x;
}

// Exponent field in [524, 1524), 2^-499 to 2^500: the quotient of any two such
// values has an exponent of at most 999 either way, far from over- and underflow,
// as has a root.
SW2D_HD bool d_mid(double x) { return (d_hi(x) & 0x7ff00000u) - (524u << 20) < (1000u << 20); }

#ifdef __CUDACC__
static __host__ __device__ __noinline__ double d_div_plain(double a, double b) { return a / b; }
static __host__ __device__ __noinline__ double d_sqrt_plain(double x) { return sqrt(x); }
#else
inline double d_div_plain(double a, double b) { return a / b; }
inline double d_sqrt_plain(double x) { return std::sqrt(x); }
#endif

// ---- division and square root on the integer pipes ---------------------------------
//
// The quotient of two 53-bit mantissas as integers: a 22-bit FP32 seed of the
// reciprocal, one third-order Newton step in 64-bit fixed point (2^-61 relative,
// never above), floor of the quotient to within one by a high product, and the
// exact remainder, which fixes the floor and rounds to nearest.  About 60 integer
// instructions where Newton and Markstein steps on the FP64 pipe take six of 64
// cycles each, and correctly rounded for every operand pair by construction (a quotient of two doubles is never midway between
// two doubles).

SW2D_HD unsigned long long mul_hi(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}

// A seed in (or an ulp or two outside) [1/2, 1) as a 32-bit fraction in [1/2, 1).
SW2D_HD unsigned seed_fraction(float seed) {
    const unsigned s = f_bits(seed);
    return s >= 0x3f800000u ? 0xffffffffu : (s < 0x3f000000u ? 0x80000000u : ((s & 0x7fffffu) | 0x800000u) << 8);
}

// 2^127 / B for B in [2^63, 2^64), as Y <= 2^64 / m with m = B / 2^63, low by
// less than 2^-60 of it.
SW2D_HD unsigned long long recip64(unsigned long long B) {
    typedef unsigned long long u64;
    typedef long long i64;
    const unsigned Bh = (unsigned)(B >> 32), Bl = (unsigned)B;
    const unsigned Y0 = seed_fraction(f_rcp_seed(f_from_bits(0x3f800000u | ((Bh >> 8) & 0x7fffffu))));
    // e = 1 - m y0 in units of 2^-63 (|e| < 2^42)
    const u64 prod = (u64)Bh * Y0 + (((u64)Bl * Y0) >> 32);
    const i64 e = (i64)(0x8000000000000000ull - prod);
    // t = e + e^2; y0 (1 + t)
    const i64 eh = e >> 20;  // |eh| < 2^22
    const i64 t = e + ((eh * eh) >> 23) - 4;
    const u64 tu = t < 0 ? (u64)-t : (u64)t;
    const u64 corr = ((u64)(unsigned)(tu >> 32) * Y0 << 1) + (((u64)(unsigned)tu * Y0) >> 31);
    const u64 base = (u64)Y0 << 32;
    return t < 0 ? base - corr - 2ull : base + corr;
}

// The mantissa quotient: A, B in [2^52, 2^53), Y = recip64(B << 11); the quotient
// rounded to 53 bits in [2^52, 2^53], and *less = 1 where A < B (exponent one less).
SW2D_HD unsigned long long quotient53(unsigned long long A, unsigned long long B, unsigned long long Y, int *less) {
    typedef unsigned long long u64;
    const int l = A < B ? 1 : 0;
    const u64 A2 = A << l;
    u64 Q = mul_hi(A2, Y);
    u64 r = (A2 << 52) - Q * B;  // exact: 0 <= r < 2 B, as Q is the floor or one less
    if (r >= B) Q++, r -= B;
    *less = l;
    return Q + (2 * r > B ? 1ull : 0ull);
}

SW2D_HD unsigned long long d_mant(double x) {
    return (d_bits(x) & 0xfffffffffffffull) | 0x10000000000000ull;
}

// a / b for b in mid range and positive, a in mid range
SW2D_HD double d_div_fast(double a, double b) {
    typedef unsigned long long u64;
    const u64 B = d_mant(b);
    int less;
    const u64 Q = quotient53(d_mant(a), B, recip64(B << 11), &less);
    const int ea = (int)((d_hi(a) >> 20) & 0x7ffu), eb = (int)(d_hi(b) >> 20);
    return d_from_bits((d_bits(a) & 0x8000000000000000ull) + ((u64)(ea - eb + 1022 - less) << 52) + Q);
}

SW2D_HD double d_div(double a, double b) {
    if (d_mid(b) && (int)d_hi(b) > 0) {
        if (d_mid(a)) return d_div_fast(a, b);
        if (d_is_zero(a)) return a;
    }
    return d_div_plain(a, b);
}

// a / d for a divisor known in advance (positive, in mid range): its mantissa, its
// reciprocal (recip64) and its exponent field.
struct KnownDivisor {
    double d;
    unsigned long long B, Y;
    int e, ok;
};
SW2D_HD KnownDivisor known_divisor(double d) {
    KnownDivisor k;
    k.d = d;
    k.ok = d_mid(d) && (int)d_hi(d) > 0;
    k.B = d_mant(d);
    k.Y = recip64(k.B << 11);
    k.e = (int)(d_hi(d) >> 20);
    return k;
}
SW2D_HD double d_div_known(double a, const KnownDivisor &k) {
    typedef unsigned long long u64;
    if (d_is_zero(a)) return a;
    if (!k.ok || !d_mid(a)) return d_div_plain(a, k.d);
    int less;
    const u64 Q = quotient53(d_mant(a), k.B, k.Y, &less);
    const int ea = (int)((d_hi(a) >> 20) & 0x7ffu);
    return d_from_bits((d_bits(a) & 0x8000000000000000ull) + ((u64)(ea - k.e + 1022 - less) << 52) + Q);
}

// sqrt(x), x positive in mid range: the integer root of the mantissa scaled to 106
// or 107 bits, from a 22-bit seed of 1/sqrt and one third-order step, with the
// exact remainder (a root is never midway between two doubles).
SW2D_HD double d_sqrt_fast(double x) {
    typedef unsigned long long u64;
    typedef long long i64;
    const unsigned xh = d_hi(x);
    const int e = (int)(xh >> 20) - 1023;
    const unsigned odd = (unsigned)e & 1u;
    const int k = (e - (int)odd) / 2;
    const u64 M = d_mant(x) << odd;  // m = M / 2^52 in [1, 4)
    const unsigned Y0 = seed_fraction(
        f_rsqrt_seed(f_from_bits((0x3f800000u + (odd << 23)) | ((xh & 0x000fffffu) << 3) | (d_lo(x) >> 29))));
    // e1 = 1 - m y0^2 in units of 2^-62
    const u64 yy = (u64)Y0 * Y0;                      // y0^2 in 2^-64
    const u64 prod = mul_hi(yy, M << 10);             // m y0^2 in units of 2^-62
    const i64 e1 = (i64)(0x4000000000000000ull - prod);  // |e1| < 2^42
    // y = y0 (1 + e1/2 + 3/8 e1^2); S = m y
    const i64 eh = e1 >> 20;
    const i64 t = (e1 >> 1) + ((3 * ((eh * eh) >> 22)) >> 3) - 2;  // in 2^-62
    const u64 tu = t < 0 ? (u64)-t : (u64)t;
    const u64 corr = ((u64)(unsigned)(tu >> 32) * Y0 << 2) + (((u64)(unsigned)tu * Y0) >> 30);  // y0 t in 2^-64
    const u64 base = (u64)Y0 << 32;
    const u64 y = t < 0 ? base - corr - 4ull : base + corr;
    u64 S = mul_hi(M << 10, y) >> 10;                 // the root's floor or one less
    u64 r = (M << 52) - S * S;                        // exact: 0 <= r <= 4 S
    if (r > 2 * S) r -= 2 * S + 1, S++;
    S += r > S ? 1ull : 0ull;                         // nearest: (S + 1/2)^2 = S^2 + S + 1/4
    return d_from_bits(((u64)(1022 + k) << 52) + S);
}

SW2D_HD double d_sqrt(double x) {
    if (d_mid(x) && (int)d_hi(x) > 0) return d_sqrt_fast(x);
    return d_is_zero(x) ? x : d_sqrt_plain(x);
}

// ---- double to float, for estimates only ---------------------------------------

// |x| truncated to FP32 (0 below the normal range, inf from 2^123 on, below the
// divisors that __fdividef gives up on; NaN stays NaN)
SW2D_HD float d_abs_float(double x) {
    const unsigned hi = d_hi(x) & 0x7fffffffu;
    const unsigned v = ((hi - 0x38000000u) << 3) | (d_lo(x) >> 29);
    if (hi - 0x38100000u < 0x47a00000u - 0x38100000u) return f_from_bits(v);
    return hi < 0x38100000u ? 0.f : (hi >= 0x7ff00000u && d_is_nan(x) ? f_from_bits(0x7fc00000u) : f_from_bits(0x7f800000u));
}

// ---- the friction term's power --------------------------------------------------

// Tables of the deterministic log / exp (their plain forms are in
// sw2d_device.cuh, det_log and det_exp): 1/c_k and ln c_k for c_k = 1 + k/128,
// 2^(j/64), and the products with the split ln 2 that the plain forms multiply
// out: e ln2_hi, e ln2_lo for |e| <= 64 and n ln2_hi/64, n ln2_lo/64 for
// |n| <= 2048.
constexpr int kPowE = 64, kPowN = 2048;
struct PowTables {
    double inv[128], logc[128], exp2j[64];
    double ehi[2 * kPowE], elo[2 * kPowE];
    double nhi[2 * kPowN], nlo[2 * kPowN];
};

// v (an unsigned integer below 2^53) times 2^-52, exactly
SW2D_HD double d_from_frac52(unsigned long long v) {
    if (v == 0ull) return 0.0;
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)v);
#else
    const int lz = __builtin_clzll(v);
#endif
    const unsigned long long m = v << (lz - 11);  // leading one at bit 52
    // value = m 2^(11 - lz) 2^-52: exponent 11 - lz of 1.f
    return d_from_bits(((unsigned long long)(1022 + 11 - lz) << 52) + m);
}

// x^1.3333330 = exp(1.3333330 ln x) with the operations of det_exp(1.3333330 *
// det_log(x)) (cu:195, cu:312), for x whose exponent and result lie in the
// tables; sets *ok to false otherwise.  Of the plain form's FP64 operations it
// replaces: m - c (exact, formed from the mantissa's low bits), the products of
// the split ln 2 (tables), the first Horner product (-1/8 r is exact, so one FMA
// rounds as the product and sum do), floor and the integer conversions (on the
// bits) and the final power of two (on the exponent field).
SW2D_HD double d_pow43_fast(double x, const PowTables *__restrict__ T, bool *ok) {
    const unsigned long long b = d_bits(x);
    const int e = (int)(b >> 52) - 1023;  // x > 0
    const int k = (int)((b >> 45) & 127);
    *ok = false;
    if ((unsigned)(e + kPowE) >= 2u * kPowE) return 0.0;
    const double r = d_from_frac52(b & 0x1fffffffffffull) * T->inv[k];
    double p = d_fma(-1.0 / 8.0, r, 1.0 / 7.0);
    p = p * r - 1.0 / 6.0;
    p = p * r + 1.0 / 5.0;
    p = p * r - 1.0 / 4.0;
    p = p * r + 1.0 / 3.0;
    p = p * r - 0.5;
    p = p * r + 1.0;
    const double lr = p * r;
    const double y = 1.3333330 * (T->ehi[e + kPowE] + (T->elo[e + kPowE] + (T->logc[k] + lr)));
    // n = floor(64 y / ln 2 + 0.5), on the bits
    const double v = y * (64.0 * 0x1.71547652b82fep+0) + 0.5;
    const unsigned vh = d_hi(v), vl = d_lo(v);
    const int ev = (int)((vh >> 20) & 0x7ffu) - 1023;
    if (ev > 10) return 0.0;  // |v| >= 2048
    int n;
    if (ev < 0) {
        n = ((int)vh < 0 && !d_is_zero(v)) ? -1 : 0;
    } else {
        const unsigned m = (vh & 0x000fffffu) | 0x00100000u;
        const int mag = (int)(m >> (20 - ev));
        const bool frac = ((m & ((1u << (20 - ev)) - 1u)) | vl) != 0u;
        n = (int)vh < 0 ? -(mag + (frac ? 1 : 0)) : mag;
    }
    const double s = (y - T->nhi[n + kPowN]) - T->nlo[n + kPowN];
    p = 1.0 / 720.0;
    p = p * s + 1.0 / 120.0;
    p = p * s + 1.0 / 24.0;
    p = p * s + 1.0 / 6.0;
    p = p * s + 0.5;
    p = p * s + 1.0;
    p = p * s + 1.0;
    const int j = n & 63, q = (n - j) / 64;
    const double f = p * T->exp2j[j];
    *ok = true;
    return d_make(d_hi(f) + ((unsigned)q << 20), d_lo(f));
}

// ---- the same power on the integer pipes ------------------------------------------
//
// A Horner step p' = c +- p r rounds twice, after the product and after the sum,
// and costs two FP64 instructions of 64 pipe cycles each.  The coefficients, the
// signs and the range of r are known, so the step can be done exactly in 64-bit
// fixed point in about 36 integer instructions: p as an integer PF = p 2^F (F per
// step, 2^60 <= PF < 2^64), r as a mantissa R in [2^63, 2^64) and an exponent.
// The 128-bit product is rounded to 53 bits (to nearest, ties to even, with the
// lower bits jammed into a sticky bit), aligned, added and rounded again at the
// sum's last place.

SW2D_HD int u_clz(unsigned x) {
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}

// High 64 bits of a b, the lower 64 jammed into the last bit.
SW2D_HD unsigned long long mul_jam(unsigned long long a, unsigned long long b) {
    typedef unsigned long long u64;
    const unsigned al = (unsigned)a, ah = (unsigned)(a >> 32), bl = (unsigned)b, bh = (unsigned)(b >> 32);
    const u64 p0 = (u64)al * bl;
    const u64 p1 = (u64)ah * bl + (p0 >> 32);
    const u64 p2 = (u64)al * bh + (unsigned)p1;
    const u64 p3 = (u64)ah * bh + (p1 >> 32) + (p2 >> 32);
    return p3 | (((unsigned)p0 | (unsigned)p2) != 0u ? 1ull : 0ull);
}

// x (>= 2^53, its last bit sticky) rounded to 53 significant bits; *lz: its
// leading zeros before rounding.
SW2D_HD unsigned long long round53(unsigned long long x, int *lz) {
    const int z = u_clz((unsigned)(x >> 32)), d = 11 - z;  // d bits go
    const unsigned lo = (unsigned)x, inc = (1u << (d - 1)) - 1u + ((lo >> d) & 1u);
    *lz = z;
    const unsigned long long t = x + inc;
    return t & ~(unsigned long long)((1u << d) - 1u);
}

// x >> n with the bits lost jammed into the last one, 0 < n < 32
SW2D_HD unsigned long long shift_jam(unsigned long long x, int n) {
    return (x >> n) | (((unsigned)x << (32 - n)) != 0u ? 1ull : 0ull);
}

// v rounded to a multiple of 2^sh, ties to even
SW2D_HD unsigned long long round_at(unsigned long long v, int sh) {
    const unsigned inc = (1u << (sh - 1)) - 1u + (((unsigned)v >> sh) & 1u);
    return (v + inc) & ~(unsigned long long)((1u << sh) - 1u);
}

// c - p r with p, r >= 0: c and p with F = 63, r = R 2^(-sft - 64), result with
// its last place at bit `sh`.
SW2D_HD unsigned long long horner_sub(unsigned long long p, unsigned long long R, int sft, unsigned long long c, int sh) {
    int lz;
    return round_at(c - shift_jam(round53(mul_jam(p, R), &lz), sft), sh);
}

// c + p s for a signed s of mantissa S: `neg` all ones for s < 0.
SW2D_HD unsigned long long horner_add(unsigned long long p, unsigned long long S, int sft, unsigned long long c,
                                      unsigned long long neg, int sh) {
    int lz;
    const unsigned long long x = shift_jam(round53(mul_jam(p, S), &lz), sft);
    return round_at(c + ((x ^ neg) - neg), sh);
}

// c 2^F of a double c, exactly (constants)
SW2D_HD constexpr unsigned long long fixed_of(double c, int F) {
    for (int k = 0; k < F; k++) c *= 2.0;
    return (unsigned long long)c;
}

// d_pow43_fast with both polynomials and the exact products in integers: 8 FP64
// instructions instead of 36.  *ok is false for the operands whose reduced
// argument is 0 or below 2^-28 as well (d_pow43_fast takes those).
SW2D_HD double d_pow43_int(double x, const PowTables *__restrict__ T, bool *ok) {
    typedef unsigned long long u64;
    constexpr u64 c7 = fixed_of(1.0 / 7.0, 63), c6 = fixed_of(1.0 / 6.0, 63), c5 = fixed_of(1.0 / 5.0, 63),
                  c4 = fixed_of(1.0 / 4.0, 63), c3 = fixed_of(1.0 / 3.0, 63), c2 = fixed_of(0.5, 63),
                  c1 = fixed_of(1.0, 63);
    constexpr u64 e720 = fixed_of(1.0 / 720.0, 72), e120 = fixed_of(1.0 / 120.0, 69), e24 = fixed_of(1.0 / 24.0, 67),
                  e6 = fixed_of(1.0 / 6.0, 65);
    const u64 b = d_bits(x);
    const int e = (int)(b >> 52) - 1023;  // x > 0
    const int k = (int)((b >> 45) & 127);
    const u64 frac = b & 0x1fffffffffffull;  // m - c = frac 2^-52
    *ok = false;
    if ((unsigned)(e + kPowE) >= 2u * kPowE || (frac >> 27) == 0ull) return 0.0;
    // r = frac 2^-52 / c rounded: R 2^(er - 63)
    const double inv = T->inv[k];  // in (1/2, 1]: exponent -1 (or 0 for k = 0)
    const int zf = u_clz((unsigned)(frac >> 13));  // frac < 2^45
    const u64 M = ((d_bits(inv) & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
    int lz;
    u64 R = round53(mul_jam(frac << (19 + zf), M), &lz);
    // frac << (19 + zf) = (m - c) 2^(71 + zf), M = inv 2^(63 or 64)
    int er = 63 - (71 + zf + (k ? 64 : 63) - 64);
    if (lz) R <<= 1, er -= 1;  // (rounding up to 2^64 cannot happen: 1/c and m - c do not both end in ones)
    if (R >> 63 == 0ull) return 0.0;
    const int sft = -er - 1;
    if (sft > 27) return 0.0;
    u64 p = round_at(c7 - shift_jam(R, sft + 4), 8);
    p = horner_sub(p, R, sft, c6, 8);
    p = horner_sub(p, R, sft, c5, 8);
    p = horner_sub(p, R, sft, c4, 8);
    p = horner_sub(p, R, sft, c3, 9);
    p = horner_sub(p, R, sft, c2, 9);
    p = horner_sub(p, R, sft, c1, 10);
    const u64 l = round53(mul_jam(p, R), &lz);  // lr = l 2^(er - 62)
    const int zl = u_clz((unsigned)(l >> 32));
    const double lr = d_from_bits(((u64)(1023 + er + 1 - zl) << 52) + (((l << zl) >> 11) & 0xfffffffffffffull));
    const double y = 1.3333330 * (T->ehi[e + kPowE] + (T->elo[e + kPowE] + (T->logc[k] + lr)));
    const double v = y * (64.0 * 0x1.71547652b82fep+0) + 0.5;
    const unsigned vh = d_hi(v), vl = d_lo(v);
    const int ev = (int)((vh >> 20) & 0x7ffu) - 1023;
    if (ev > 10) return 0.0;  // |v| >= 2048
    int n;
    if (ev < 0) {
        n = ((int)vh < 0 && !d_is_zero(v)) ? -1 : 0;
    } else {
        const unsigned m = (vh & 0x000fffffu) | 0x00100000u;
        const int mag = (int)(m >> (20 - ev));
        const bool fr = ((m & ((1u << (20 - ev)) - 1u)) | vl) != 0u;
        n = (int)vh < 0 ? -(mag + (fr ? 1 : 0)) : mag;
    }
    const double s = (y - T->nhi[n + kPowN]) - T->nlo[n + kPowN];
    const u64 sb = d_bits(s);
    const int es = (int)((sb >> 52) & 0x7ffu) - 1023;
    if (es < -29 || es > -8) return 0.0;
    const u64 S = ((sb & 0xfffffffffffffull) | 0x10000000000000ull) << 11, neg = (u64)((long long)sb >> 63);
    const int q0 = -es - 1, lower = (int)(sb >> 63);  // below 1/2 and 1 the last place is one bit finer
    p = horner_add(e720, S, q0 + 3, e120, neg, 10);
    p = horner_add(p, S, q0 + 2, e24, neg, 10);
    p = horner_add(p, S, q0 + 2, e6, neg, 10);
    p = horner_add(p, S, q0 + 2, c2, neg, 10 - lower);
    p = horner_add(p, S, q0, c1, neg, 11 - lower);
    p = horner_add(p, S, q0, c1, neg, 11 - lower);
    // times 2^(j/64), in [1, 2), and 2^q
    const int j = n & 63, q = (n - j) / 64;
    const u64 E = ((d_bits(T->exp2j[j]) & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
    const u64 f = round53(mul_jam(p, E), &lz);  // the product times 2^62
    const int z = u_clz((unsigned)(f >> 32));
    *ok = true;
    return d_from_bits(((u64)(1023 + q + 1 - z) << 52) + (((f << z) >> 11) & 0xfffffffffffffull));
}

}  // namespace sw2d

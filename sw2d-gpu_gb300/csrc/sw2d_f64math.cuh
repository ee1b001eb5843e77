// sw2d_f64math.cuh -- double-precision helpers for a GPU whose FP64 pipe is
// the scarce unit (one FP64 warp instruction occupies a scheduler's pipe for
// 64 cycles, an integer or FP32 one for one or two).
//
// Every helper returns the bits of the plain IEEE expression it stands for
// (division, square root, comparison, the deterministic power of the
// friction term); it only takes fewer FP64 instructions for them.  What a
// helper's fast form does not cover (subnormals, infinities, NaN, operands
// near the ends of the exponent range) falls through to the plain expression.
// The forms with host equivalents compile on the host too, where the tests
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
// gives the same final bits; see the users)
SW2D_HD float f_rcp_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}
SW2D_HD float f_rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / std::sqrt(x);
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

// Exponent field in [200, 1800): far from over- and underflow of anything the
// fast forms below compute.
SW2D_HD bool d_mid(double x) { return (d_hi(x) & 0x7ff00000u) - (200u << 20) < (1600u << 20); }

// ---- division ---------------------------------------------------------------

// a / b, correctly rounded.  The reciprocal comes from an FP32 seed of b's
// mantissa by one third-order Newton step (three FMAs), and the quotient from
// Markstein's correction q + (a - b q) y (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990): six FP64 instructions.  With a seed error of 2^-22 the
// reciprocal is off by half an ulp plus 2^-13 ulp at most, and the rounding of
// the corrected quotient can differ from that of a / b only for a quotient
// within 2^-53 ulp of a midpoint between two doubles that also meets that
// excess, about one in 2^60 operand pairs.
SW2D_HD double d_div_fast(double a, double b) {
    const unsigned bh = d_hi(b), bl = d_lo(b);
    const float m = f_from_bits(0x3f800000u | ((bh & 0x000fffffu) << 3) | (bl >> 29));
    const unsigned s = f_bits(f_rcp_seed(m));
    // the seed as a double times 2^-exponent(b); b's sign is the caller's: +
    const double y0 = d_make((s >> 3) + 0x38000000u - ((bh & 0x7ff00000u) - 0x3ff00000u), s << 29);
    const double e = d_fma(-b, y0, 1.0);
    const double y = d_fma(y0, d_fma(e, e, e), y0);
    const double q = a * y;
    return d_fma(d_fma(-b, q, a), y, q);
}

#ifdef __CUDACC__
static __host__ __device__ __noinline__ double d_div_plain(double a, double b) { return a / b; }
#else
inline double d_div_plain(double a, double b) { return a / b; }
#endif

// a / b for b >= 0 (or any b: what is not in mid range takes the plain form)
SW2D_HD double d_div(double a, double b) {
    if (d_mid(b) && (d_mid(a) || d_is_zero(a)) && (int)d_hi(b) > 0) return d_div_fast(a, b);
    return d_div_plain(a, b);
}

// a / d for a divisor known in advance, rd = 1 / d rounded: the multiplication
// and two FMAs of N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Comput. 53, 2004.
SW2D_HD double d_div_const(double a, double d, double rd) {
    if (d_mid(a) || d_is_zero(a)) {
        const double q = a * rd;
        return d_fma(d_fma(-q, d, a), rd, q);
    }
    return d_div_plain(a, d);
}

// ---- square root --------------------------------------------------------------

// sqrt(x), correctly rounded: FP32 seed of 1/sqrt of the mantissa (scaled to
// [1, 4)), one third-order step on g ~ sqrt(x) and h ~ 1 / (2 sqrt(x)) together
// (Goldschmidt's coupled form), and Markstein's correction g + (x - g g) h:
// eight FP64 instructions.
SW2D_HD double d_sqrt_fast(double x) {
    const unsigned xh = d_hi(x), xl = d_lo(x);
    const int e = (int)(xh >> 20) - 1023;       // x = m 2^e, e = 2 k + odd
    const unsigned odd = (unsigned)e & 1u;
    const int k = (e - (int)odd) / 2;
    const float m = f_from_bits((0x3f800000u + (odd << 23)) | ((xh & 0x000fffffu) << 3) | (xl >> 29));
    const unsigned s = f_bits(f_rsqrt_seed(m));  // in (0.5, 1]
    const unsigned yh = (s >> 3) + 0x38000000u - ((unsigned)k << 20);
    const double y = d_make(yh, s << 29), h = d_make(yh - 0x00100000u, s << 29);
    const double g = x * y;
    const double r = d_fma(-g, h, 0.5);
    const double t = d_fma(1.5 * r, r, r);
    const double g1 = d_fma(g, t, g), h1 = d_fma(h, t, h);
    return d_fma(d_fma(-g1, g1, x), h1, g1);
}

#ifdef __CUDACC__
static __host__ __device__ __noinline__ double d_sqrt_plain(double x) { return sqrt(x); }
#else
inline double d_sqrt_plain(double x) { return std::sqrt(x); }
#endif

// The roots nearest to a midpoint between two doubles are those of the mantissas
// one unit away from 1 (and from 2): those take the plain form.
SW2D_HD double d_sqrt(double x) {
    const unsigned long long m = d_bits(x) & 0x000fffffffffffffull;
    const bool hard = m != 0ull && ((m + 8ull) & 0x000fffffffffffffull) < 17ull;
    if (d_mid(x) && (int)d_hi(x) > 0 && !hard) return d_sqrt_fast(x);
    return d_is_zero(x) ? x : d_sqrt_plain(x);
}

// ---- double to float, for estimates only ---------------------------------------

// |x| truncated to FP32 (0 below the normal range, inf above it, NaN stays NaN)
SW2D_HD float d_abs_float(double x) {
    const unsigned hi = d_hi(x) & 0x7fffffffu;
    const unsigned v = ((hi - 0x38000000u) << 3) | (d_lo(x) >> 29);
    if (hi - 0x38100000u < 0x0fe00000u - 0x00100000u) return f_from_bits(v);
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

}  // namespace sw2d

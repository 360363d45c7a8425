// phd_fp64.cuh -- IEEE FP64 quotients, square roots and comparisons that spare the FP64 pipe.
//
// GB300 issues one FP64 warp instruction per 19 clocks and SM, whatever the number of
// active lanes, against 0.3 clocks for an FP32 or integer one (measured: fused
// multiply-add, addition, product and comparison alike); a division or square root of the
// compiler takes 141-143 clocks, 7.5 FP64 instructions.  Kernels written with the plain
// operations keep that pipe 80-85% busy, so their time is their count of FP64 instructions, and
// 40-odd FP32 and integer instructions run in the shadow of each.  The helpers here therefore
// form everything that need not be an FP64 instruction with FP32 and integer ones (which leaves
// the step's three kernels at 55 to 80% of the pipe on meshes that fill the GPU, the reverse step's
// faces at 75%):
//   * the reciprocal (square root) seeds: FP32 approximation of the operand's leading 24
//     bits, one Newton-Raphson step carried as a float pair with the operand's next 23
//     bits (2^-44 relative), a second one in 64-bit fixed point, rounded to a double:
//     within 0.51 units of the last place;
//   * the quotient from the seed as the nearest 53-bit integer of the significands' quotient:
//     the upper word of a 64-bit product gives it to within one, the remainder, exact in 64
//     bits, says which; the square root likewise.  No FP64 instruction; against the three of a
//     correction by fused multiply-adds: face 359 -> 291 us, gradients 279 -> 232, a whole step
//     of 1024 x 1024 cells 4.13 -> 3.32 ms;
//   * comparisons, halving and sign changes by integer operations on the bits.
// A seed holds for operands in a window of exponents around 1 in which no step can
// overflow, underflow or lose the remainder's low bits; anything else (zero or negative
// radicands, infinities, NaN, subnormals) clears `ok`, and the caller then takes its plain
// IEEE path.  The host versions are the plain operations.
#pragma once
#include <cmath>
#include <cstring>
#include "phd_common.cuh"

namespace phd {

// Exponent windows (biased fields) within which the helpers' steps are exact: denominators
// and radicands 2^-400 .. 2^400, numerators 2^-500 .. 2^500 or zero.
constexpr unsigned F64_DEN_LO = (1023u - 400u) << 20, F64_DEN_SPAN = 800u << 20;
constexpr unsigned F64_NUM_LO = (1023u - 500u) << 20, F64_NUM_SPAN = 1000u << 20;

#ifdef __CUDACC__
// 2^53 y for a float y in [0.5, 1], plus a correction of at most 2^30.
__device__ __forceinline__ long long fix53(float y, float corr) {
    const unsigned m = __float_as_uint(y);
    return ((long long)((m & 0x7fffffu) | 0x800000u) << (m >= 0x3f800000u ? 30 : 29)) +
           (long long)__float2int_rn(corr * 9007199254740992.0f);
}

// y = 1/b rounded to a double; clears ok outside the denominators' window.
__device__ __forceinline__ double rcp_seed(double b, bool &ok) {
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    ok = ok && ((hi & 0x7fffffffu) - F64_DEN_LO < F64_DEN_SPAN);
    // |b| = 2^e (bh + bl), bh in [1, 2) the leading 24 bits, bl the next 23
    const float bh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u);
    const float bl = __uint_as_float(((lo << 3) >> 9) | 0x3f800000u) - 1.0f;      // bl 2^23
    float y0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(bh));                        // in [0.5, 1]
    const float e = __fmaf_rn(-bl * 1.1920928955078125e-7f, y0, __fmaf_rn(-bh, y0, 1.0f));
    const long long Y = fix53(y0, y0 * __fmaf_rn(e, e, e));                        // y0 (1 + e + e^2)
    // the second step: E = 2^105 - B Y (B = 2^52 |b| 2^-e) is below 2^61, so its low 64 bits are it
    const unsigned long long B = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    const long long E = -(long long)(B * (unsigned long long)Y);
    const long long Y10 = (Y << 10) + (((long long)(int)(E >> 32) * (long long)(int)(Y >> 23)) >> 40);
    const unsigned long long y = (unsigned long long)(Y10 + 512) >> 10;
    const unsigned yh = (unsigned)(y >> 32) + (1021u << 20) - ((hi & 0x7ff00000u) - (1023u << 20));
    return __hiloint2double((int)(yh | (hi & 0x80000000u)), (int)(unsigned)y);
}

// a/b from y = rcp_seed(b); clears ok when a is outside the numerators' window.  With 53-bit
// integers A = 2^52 m_a, B = 2^52 m_b: the nearest integer n to X = A 2^t / B, t = 52 (53
// where m_a < m_b), which lies in [2^52, 2^53].  A times the seed gives n to within one, the
// remainder A 2^t - n B, below 2 B and so exact in the low 64 bits, tells which (X is never half
// an integer).
__device__ __forceinline__ double div_seeded(double a, double b, double y, bool &ok) {
    const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
    const unsigned mag = ha & 0x7fffffffu, la = (unsigned)__double2loint(a);
    const bool zero = (mag | la) == 0u;
    ok = ok && (mag - F64_NUM_LO < F64_NUM_SPAN || zero);
    const unsigned long long A = ((unsigned long long)((ha & 0xfffffu) | 0x100000u) << 32) | la;
    const unsigned long long B =
        ((unsigned long long)((hb & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(b);
    // 2^53 / m_b (the seed of a power of two has its exponent one higher)
    unsigned long long Y = ((unsigned long long)(((unsigned)__double2hiint(y) & 0xfffffu) | 0x100000u) << 32) |
                           (unsigned)__double2loint(y);
    Y <<= B == (1ull << 52) ? 2 : 1;
    const bool lt = A < B;
    unsigned long long n = (__umul64hi(A << 11, lt ? Y << 1 : Y) + 1) >> 1;
    const long long r2 = (long long)(((unsigned long long)la << (lt ? 54 : 53)) - 2 * (n * B));      // 2 (A 2^t - n B)
    n += r2 > (long long)B ? 1 : 0;
    n -= r2 < -(long long)B ? 1 : 0;
    const unsigned e = mag - (hb & 0x7ff00000u) - (mag & 0xfffffu) + (lt ? 1021u << 20 : 1022u << 20);
    const unsigned hi = zero ? 0u : e + (unsigned)(n >> 32);
    return __hiloint2double((int)(hi | ((ha ^ hb) & 0x80000000u)), zero ? 0 : (int)(unsigned)n);
}

__device__ __forceinline__ double div_ieee(double a, double b, bool &ok) {
    return div_seeded(a, b, rcp_seed(b, ok), ok);
}

// 1/sqrt(a) to within 0.6 units of the last place; clears ok for zero, negative and
// out-of-window radicands.
__device__ __forceinline__ double rsqrt_seed(double a, bool &ok) {
    const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
    ok = ok && (hi - F64_DEN_LO < F64_DEN_SPAN);
    // a = 4^k (bh + bl), bh in [1, 4)
    const int ex = (int)(hi >> 20) - 1023;
    const unsigned odd = ex & 1;
    const float bh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | (0x3f800000u + (odd << 23)));
    const float bl = (__uint_as_float(((lo << 3) >> 9) | 0x3f800000u) - 1.0f) * (odd ? 2.0f : 1.0f);   // bl 2^23
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(bh));                      // in [0.5, 1]
    const float p = y0 * y0, pl = __fmaf_rn(y0, y0, -p);                           // y0^2 = p + pl
    float e = __fmaf_rn(-bh, p, 1.0f);
    e = __fmaf_rn(-bh, pl, e);
    e = __fmaf_rn(-bl * 1.1920928955078125e-7f, p, e);                             // 1 - (bh + bl) y0^2
    // (bh + bl)^(-1/2) = y0 (1 + e/2 + 3 e^2/8) + O(e^3)
    const long long Y = fix53(y0, y0 * (e * __fmaf_rn(0.375f, e, 0.5f)));
    // the second step: W = 2^53 y^2, A = 2^52 a 4^-k; E = 2^105 (1 - a y^2) is below 2^62, so the
    // low 64 bits of -A W are it; y += y (1 - a y^2) / 2
    const unsigned long long A = (((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << odd;
    const unsigned long long Yu = (unsigned long long)Y << 10;                     // 2^63 y
    const unsigned long long W = (__umul64hi(Yu, Yu) + 256u) >> 9;
    const long long E = -(long long)(A * W);
    const long long Y10 = (Y << 10) + (((long long)(int)(E >> 32) * (long long)(int)(Y >> 23)) >> 41);
    const unsigned long long y = (unsigned long long)(Y10 + 512) >> 10;
    const int k = (ex - (int)odd) >> 1;
    const unsigned yh = (unsigned)(y >> 32) + (unsigned)((1021 - k) << 20);
    return __hiloint2double((int)yh, (int)(unsigned)y);
}

// sqrt(a) from its seed: the nearest integer n to sqrt(A 2^52), A = 2^52 a 4^-k in [2^52, 2^54).
// A times the seed gives n to within a few units, the remainder A 2^52 - n^2 over 2 n how many,
// and the new remainder whether the last one is right: it lies in (-n, n] for the nearest.
__device__ __forceinline__ double sqrt_ieee(double a, bool &ok) {
    const double y = rsqrt_seed(a, ok);
    const unsigned ha = (unsigned)__double2hiint(a), hy = (unsigned)__double2hiint(y);
    const int ex = (int)(ha >> 20) - 1023, odd = ex & 1;
    const unsigned long long A =
        (((unsigned long long)((ha & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(a)) << odd;
    // 2^53 / sqrt(a 4^-k): 2^53 itself for an even power of two
    unsigned long long Y = ((unsigned long long)((hy & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(y);
    if (A == (1ull << 52)) Y <<= 1;
    unsigned long long n = __umul64hi(A << 10, Y << 1);
    long long r = (long long)((A << 52) - n * n);
    n += (unsigned long long)(((r >> 30) * (long long)(Y >> 22) + (1ll << 53)) >> 54);
    r = (long long)((A << 52) - n * n);
    n += r > (long long)n ? 1 : 0;
    n -= r <= -(long long)n ? 1 : 0;
    const unsigned e = (unsigned)(((ex - odd) >> 1) + 1022) << 20;
    return __hiloint2double((int)(e + (unsigned)(n >> 32)), (int)(unsigned)n);
}
#endif

// ---- bits: comparisons, signs and halving off the FP64 pipe (finite operands) ---------
PHD_HD __forceinline__ long long f64_bits(double a) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(a);
#else
    long long b;
    memcpy(&b, &a, sizeof b);
    return b;
#endif
}
PHD_HD __forceinline__ double f64_from(long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double a;
    memcpy(&a, &b, sizeof a);
    return a;
#endif
}
PHD_HD __forceinline__ unsigned f64_hi(double a) { return (unsigned)((unsigned long long)f64_bits(a) >> 32); }

// The same on the host: the plain operations behind the same windows.
PHD_HD __forceinline__ double f64_rcp(double b, bool &ok) {
#ifdef __CUDA_ARCH__
    return rcp_seed(b, ok);
#else
    ok = ok && ((f64_hi(b) & 0x7fffffffu) - F64_DEN_LO < F64_DEN_SPAN);
    return 1.0 / b;
#endif
}
PHD_HD __forceinline__ double f64_div_by(double a, double b, double y, bool &ok) {
#ifdef __CUDA_ARCH__
    return div_seeded(a, b, y, ok);
#else
    ok = ok && ((f64_hi(a) & 0x7fffffffu) - F64_NUM_LO < F64_NUM_SPAN || (f64_bits(a) << 1) == 0);
    return a / b;
#endif
}
PHD_HD __forceinline__ double f64_div(double a, double b, bool &ok) { return f64_div_by(a, b, f64_rcp(b, ok), ok); }
PHD_HD __forceinline__ double f64_sqrt(double a, bool &ok) {
#ifdef __CUDA_ARCH__
    return sqrt_ieee(a, ok);
#else
    ok = ok && f64_hi(a) - F64_DEN_LO < F64_DEN_SPAN;
    return sqrt(a);
#endif
}

// An order-preserving map to signed 64-bit integers; both zeros map to 0.
PHD_HD __forceinline__ long long f64_key(double a) {
    const long long b = f64_bits(a);
    return b < 0 ? (long long)(0x8000000000000000ull - (unsigned long long)b) : b;
}
PHD_HD __forceinline__ bool f64_lt(double a, double b) { return f64_key(a) < f64_key(b); }
PHD_HD __forceinline__ bool f64_le(double a, double b) { return f64_key(a) <= f64_key(b); }
PHD_HD __forceinline__ double f64_min(double a, double b) { return f64_key(b) < f64_key(a) ? b : a; }
PHD_HD __forceinline__ double f64_max(double a, double b) { return f64_key(b) > f64_key(a) ? b : a; }
PHD_HD __forceinline__ bool f64_neg(double a) { return f64_key(a) < 0; }          // a < 0.0
PHD_HD __forceinline__ bool f64_pos(double a) { return f64_bits(a) > 0; }         // a > 0.0
PHD_HD __forceinline__ bool f64_zero(double a) { return (f64_bits(a) << 1) == 0; }
// a / 2; clears ok where that is not one step of the exponent (subnormal results)
PHD_HD __forceinline__ double f64_half(double a, bool &ok) {
    const bool z = f64_zero(a);
    ok = ok && (z || (f64_hi(a) & 0x7fffffffu) >= 0x00200000u);
    return z ? a : f64_from(f64_bits(a) - (1ll << 52));
}
// the larger of m and the magnitude bits of a (a running bound of the operands' exponents)
PHD_HD __forceinline__ unsigned f64_magmax(unsigned m, double a) {
    const unsigned h = f64_hi(a) & 0x7fffffffu;
    return h > m ? h : m;
}

// FP64 -> FP32 by integer operations, truncating: relative error below 2^-23; magnitudes
// outside 2^-126 .. 2^127 go to the nearer end (zero or 2^127).
PHD_HD __forceinline__ float f64_to_f32(double a) {
    const unsigned long long b = (unsigned long long)f64_bits(a);
    const int ex = (int)((b >> 52) & 0x7ffu) - 896;
    const unsigned m = (unsigned)(b >> 29) & 0x7fffffu, s = (unsigned)(b >> 32) & 0x80000000u;
    const unsigned u = ex <= 0 ? s : (ex >= 254 ? (s | (254u << 23)) : (s | ((unsigned)ex << 23) | m));
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
#endif
}

// The same of a 2^-e for magnitudes up to 2^20, a NaN above.
PHD_HD __forceinline__ float f64_to_f32_scaled(double a, int e) {
    const unsigned long long b = (unsigned long long)f64_bits(a);
    const int ex = (int)((b >> 52) & 0x7ffu) - 896 - e;
    const unsigned m = (unsigned)(b >> 29) & 0x7fffffu, s = (unsigned)(b >> 32) & 0x80000000u;
    const unsigned u = ex <= 0 ? s : (ex >= 147 ? 0x7fc00000u : (s | ((unsigned)ex << 23) | m));
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
#endif
}

// ---- powers in 64-bit fixed point -----------------------------------------------------
// x^y = 2^(y log2 x) for positive x by some 400 integer instructions, which run in the shadow
// of the FP64 pipe (CUDA's pow is 84 FP64 instructions: 1600 clocks a warp and SM, measured).
//   log2 x = e + (2/ln 2) artanh s, s = (m - 1)/(m + 1), m in [0.7, 1.42), |s| < 0.172: the odd
//   series to s^25 (the next term is below 2^-66);
//   2^g, |g| <= 1/2: the exponential series to g^16 (the next term is below 2^-72).
// Every product keeps the upper 64 of 128 bits, rounded where it reaches the result directly, so
// that the power, rounded once to a double, is off by less than 0.51 units of its last place
// for exponents up to 15 (and rounded the wrong way in 3 cases of 10,000).  The
// coefficients are 2/(ln 2 (2k + 1)) and (ln 2)^k / k!, rounded to 62 and 64 fractional bits.
PHD_HD __forceinline__ unsigned long long mulhi64(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}

// the same, rounded to the nearest
PHD_HD __forceinline__ unsigned long long mulhi64_rn(unsigned long long a, unsigned long long b) {
    return mulhi64(a, b) + ((a * b) >> 63);
}

struct Log64 {
    int e;                             // log2 x = e + f 2^-64, f taken negative when neg
    bool neg;
    unsigned long long f;
};

// Whether log2_fix takes x: positive, normal, finite.
PHD_HD __forceinline__ bool log2_ok(double x) { return f64_hi(x) - 0x00100000u < 0x7fe00000u; }

PHD_HD __forceinline__ Log64 log2_fix(double x) {
    const unsigned long long b = (unsigned long long)f64_bits(x), mant = (b & 0xfffffffffffffull) | (1ull << 52);
    const bool up = mant >= 0x16a09e667f3bcdull;                   // m >= sqrt 2: m / 2, e + 1
    Log64 r;
    r.e = (int)(b >> 52) - 1023 + (up ? 1 : 0);
    const unsigned long long M = mant << (up ? 10 : 11);           // 2^63 m
    const unsigned long long D = (M >> 1) + (1ull << 62);          // 2^62 (m + 1)
    r.neg = M < (1ull << 63);
    const unsigned long long num = r.neg ? (1ull << 63) - M : M - (1ull << 63);
    // 2^64 / (m + 1): FP32, then two Newton-Raphson steps
    const unsigned dh = (unsigned)(D >> 32);
#ifdef __CUDA_ARCH__
    float y0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__uint2float_rz(dh)));
    const unsigned y32 = __float2uint_rz(y0 * 4611686018427387904.0f);            // 2^62
#else
    const unsigned y32 = (unsigned)((1.0f / (float)dh) * 4611686018427387904.0f);
#endif
    unsigned long long Y = (unsigned long long)y32 << 32;
    long long E = (long long)((1ull << 62) - mulhi64(D, Y));
    Y += (unsigned long long)(((long long)(Y >> 33) * (E >> 8)) >> 21);
    E = (long long)((1ull << 62) - mulhi64(D, Y));
    Y += (unsigned long long)(((long long)(Y >> 33) * E) >> 29);
    const unsigned long long s = mulhi64_rn(num << 2, Y), t = mulhi64(s, s) >> 2;      // 2^65 s, 2^64 s^2
    unsigned long long P = 0x762f8205fd7ff64ull;
    P = 0x80766bf04010a77ull + mulhi64(P, t);
    P = 0x8cb27637e4a486aull + mulhi64(P, t);
    P = 0x9b81e0fa687ff32ull + mulhi64(P, t);
    P = 0xadcd64dba1f86a2ull + mulhi64(P, t);
    P = 0xc4f9d8b4a67fefbull + mulhi64(P, t);
    P = 0xe347ab4698bb00eull + mulhi64(P, t);
    P = 0x10c9a84994022d28ull + mulhi64(P, t);
    P = 0x1484b13d7c02a8f8ull + mulhi64(P, t);
    P = 0x1a61762a7aded93full + mulhi64(P, t);
    P = 0x24eed8a1df37fcf2ull + mulhi64(P, t);
    P = 0x3d8e13b87407fae9ull + mulhi64(P, t);
    P = 0xb8aa3b295c17f0bcull + mulhi64(P, t);
    r.f = mulhi64_rn(s << 1, P);
    return r;
}

// 2^(y log2 x); clears ok where y or the result's exponent is out of the scheme's range.
PHD_HD __forceinline__ double exp2_fix(const Log64 &l, double y, bool &ok) {
    const unsigned long long by = (unsigned long long)f64_bits(y);
    const int ye = (int)((by >> 52) & 0x7ffu) - 1022;              // |y| = Ym 2^(ye - 64)
    ok = ok && ye >= -8 && ye <= 6;
    const bool yneg = (long long)by < 0;
    const unsigned long long Ym = ((by & 0xfffffffffffffull) | (1ull << 52)) << 11;
    const unsigned long long ae = (unsigned long long)(l.e < 0 ? -l.e : l.e);
    unsigned long long lo = ae * Ym, hi = mulhi64(ae, Ym);         // y log2 x, 128 bits signed
    if ((l.e < 0) != yneg) {
        lo = ~lo + 1;
        hi = ~hi + (lo == 0);
    }
    const unsigned long long B = mulhi64(l.f, Ym);
    if (l.neg != yneg) {
        hi -= lo < B;
        lo -= B;
    } else {
        lo += B;
        hi += lo < B;
    }
    if (ye > 0) {
        hi = (hi << (ye & 63)) | (lo >> ((64 - ye) & 63));
        lo <<= (ye & 63);
    } else if (ye < 0) {
        lo = (lo >> (-ye & 63)) | (hi << ((64 + ye) & 63));
        hi = (unsigned long long)((long long)hi >> (-ye & 63));
    }
    // the nearest integer and the rest g, |g| <= 1/2
    const bool down = (long long)lo < 0;
    const long long n = (long long)hi + (down ? 1 : 0);
    const unsigned long long g = down ? ~lo + 1 : lo;
    ok = ok && n >= -900 && n <= 900;
    // |2^g - 1| = |g| (c1 +- |g| (c2 +- ...)): alternating signs below 0
    unsigned long long P = 0x9c7ull;
    P = down ? 0xe1b7ull - mulhi64(P, g) : 0xe1b7ull + mulhi64(P, g);
    P = down ? 0x131496ull - mulhi64(P, g) : 0x131496ull + mulhi64(P, g);
    P = down ? 0x1816193ull - mulhi64(P, g) : 0x1816193ull + mulhi64(P, g);
    P = down ? 0x1c3bd651ull - mulhi64(P, g) : 0x1c3bd651ull + mulhi64(P, g);
    P = down ? 0x1e8cac735ull - mulhi64(P, g) : 0x1e8cac735ull + mulhi64(P, g);
    P = down ? 0x1e4cf5158cull - mulhi64(P, g) : 0x1e4cf5158cull + mulhi64(P, g);
    P = down ? 0x1b5253d395eull - mulhi64(P, g) : 0x1b5253d395eull + mulhi64(P, g);
    P = down ? 0x162c0223a5c8ull - mulhi64(P, g) : 0x162c0223a5c8ull + mulhi64(P, g);
    P = down ? 0xffe5fe2c4586ull - mulhi64(P, g) : 0xffe5fe2c4586ull + mulhi64(P, g);
    P = down ? 0xa184897c363c4ull - mulhi64(P, g) : 0xa184897c363c4ull + mulhi64(P, g);
    P = down ? 0x5761ff9e299cc4ull - mulhi64(P, g) : 0x5761ff9e299cc4ull + mulhi64(P, g);
    P = down ? 0x276556df749cee5ull - mulhi64(P, g) : 0x276556df749cee5ull + mulhi64(P, g);
    P = down ? 0xe35846b82505fc6ull - mulhi64(P, g) : 0xe35846b82505fc6ull + mulhi64(P, g);
    P = down ? 0x3d7f7bff058b1d51ull - mulhi64(P, g) : 0x3d7f7bff058b1d51ull + mulhi64(P, g);
    P = down ? 0xb17217f7d1cf79acull - mulhi64(P, g) : 0xb17217f7d1cf79acull + mulhi64(P, g);
    const unsigned long long u = mulhi64_rn(P, g);
    if (down) {                                                    // 1 - u 2^-64, in [0.7, 1]
        const unsigned long long m = (1ull << 53) - ((u + 1023) >> 11);
        return f64_from((long long)((unsigned long long)(n + 1021) << 52) + (long long)m);
    }
    const unsigned long long m = (1ull << 52) + (u >> 12) + ((u >> 11) & 1ull);
    return f64_from((long long)((unsigned long long)(n + 1022) << 52) + (long long)m);
}

}  // namespace phd

// phd_fp64.cuh -- IEEE FP64 quotients, square roots and comparisons that spare the FP64 pipe.
//
// GB300 issues one FP64 warp instruction per 19 clocks and SM, whatever the number of
// active lanes, against 0.3 clocks for an FP32 or integer one (measured: fused
// multiply-add, addition, product and comparison alike); a division or square root of the
// compiler takes 141-143 clocks, 7.5 FP64 instructions.  The FP64 kernels keep that pipe
// 85% busy, so their time is their count of FP64 instructions, and 40-odd FP32 and integer
// instructions run in the shadow of each.  The helpers here therefore form everything that
// need not be an FP64 instruction with FP32 and integer ones:
//   * the reciprocal (square root) seeds: FP32 approximation of the operand's leading 24
//     bits, one Newton-Raphson step carried as a float pair with the operand's next 23
//     bits (2^-44 relative), a second one in 64-bit fixed point, rounded to a double:
//     within 0.51 units of the last place;
//   * the quotient from the seed y in three FP64 instructions, q0 = a y, q = q0 + (a - b
//     q0) y with the remainder exact by fused multiply-add (Markstein 1990): before its
//     one rounding the correction is off by 2^-106 of q, so q is the IEEE quotient; the
//     square root likewise, s0 = a y, s = s0 + (a - s0^2) y / 2;
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

// a/b from y = rcp_seed(b); clears ok when a is outside the numerators' window.
__device__ __forceinline__ double div_seeded(double a, double b, double y, bool &ok) {
    const unsigned ha = (unsigned)__double2hiint(a);
    const unsigned mag = ha & 0x7fffffffu;
    ok = ok && (mag - F64_NUM_LO < F64_NUM_SPAN || (mag | (unsigned)__double2loint(a)) == 0u);
    const double q0 = __dmul_rn(a, y);
    const double q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
    // a zero numerator's sign (the correction would lose it)
    const unsigned s = (ha ^ (unsigned)__double2hiint(b)) & 0x80000000u;
    return __hiloint2double((int)(((unsigned)__double2hiint(q) & 0x7fffffffu) | s), __double2loint(q));
}

__device__ __forceinline__ double div_ieee(double a, double b, bool &ok) {
    return div_seeded(a, b, rcp_seed(b, ok), ok);
}

// sqrt(a); clears ok for zero, negative and out-of-window radicands.
__device__ __forceinline__ double sqrt_ieee(double a, bool &ok) {
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
    const double ys = __hiloint2double((int)yh, (int)(unsigned)y);
    const double s0 = __dmul_rn(a, ys);
    const double r = __fma_rn(-s0, s0, a);
    return __fma_rn(r, __hiloint2double((int)(yh - (1u << 20)), (int)(unsigned)y), s0);
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

}  // namespace phd

// Device check of the FP64 quotient and square root from FP32 / integer seeds (phd_fp64.cuh:
// div_ieee, sqrt_ieee, rcp_seed) against CUDA's IEEE operations, bit for bit, on seeded
// random operands: mode 0 exponents over the whole range (outside the window the helper must
// decline), 1 around 1, 2 with trailing zeros, 3 with trailing ones, 4 with quotients and
// roots next to the middle of two doubles, 5 within 32 units of powers of two.  Prints per
// mode: pairs, quotients that differ, declined; roots that differ, declined; seeds off by
// more than half a unit (2^-53 of 1).  Test-only: run by tests/test_gpu_fp64_ieee.py.
#include <cstdio>
#include <cstdlib>
#include "phd_fp64.cuh"

using namespace phd;

__device__ unsigned long long next(unsigned long long &s) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }

__global__ void k_check(int mode, int reps, unsigned long long *cnt) {
    unsigned long long s = 1234567ull + mode + 0x9E3779B97F4A7C15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
    for (int k = 0; k < 8; k++) next(s);
    for (int it = 0; it < reps; it++) {
        unsigned long long a = next(s), b = next(s);
        const unsigned long long span = mode == 0 ? 2046 : 60, e0 = mode == 0 ? 1 : 1023 - 30;
        if (mode == 2) { a &= ~((1ull << (next(s) % 53)) - 1); b &= ~((1ull << (next(s) % 53)) - 1); }
        if (mode == 3) { a |= ((1ull << (next(s) % 53)) - 1); b |= ((1ull << (next(s) % 53)) - 1); }
        a = (a & 0x800fffffffffffffull) | ((e0 + next(s) % span) << 52);
        b = (b & 0x800fffffffffffffull) | ((e0 + next(s) % span) << 52);
        if (mode < 4 && next(s) % 50 == 0) a &= 0x8000000000000000ull;
        double x = __longlong_as_double(a), y = __longlong_as_double(b), z = fabs(y);
        if (mode == 4) {
            // x = y times a 54-bit number, z = the square of one, each within 2 units
            const double mhi = x, mlo = __longlong_as_double((a & 0x7ff0000000000000ull) - (53ull << 52)), ah = fabs(mhi);
            double ph = __dmul_rn(y, mhi), pl = fma(y, mlo, fma(y, mhi, -ph));
            x = __longlong_as_double(__double_as_longlong(__dadd_rn(ph, pl)) + (long long)(next(s) % 5) - 2);
            ph = __dmul_rn(ah, ah);
            pl = fma(2 * ah, mlo, fma(ah, ah, -ph));
            z = __longlong_as_double(__double_as_longlong(__dadd_rn(ph, pl)) + (long long)(next(s) % 5) - 2);
        }
        if (mode == 5) {
            x = __longlong_as_double((long long)((1022ull + next(s) % 5) << 52) + (long long)(next(s) % 64) - 32);
            z = y = __longlong_as_double((long long)((1022ull + next(s) % 5) << 52) + (long long)(next(s) % 64) - 32);
        }
        bool ok = true;
        const double q = div_ieee(x, y, ok);
        if (!ok) atomicAdd(cnt + 1, 1ull);
        else if (__double_as_longlong(q) != __double_as_longlong(__ddiv_rn(x, y))) atomicAdd(cnt, 1ull);
        ok = true;
        const double r = sqrt_ieee(z, ok);
        if (!ok) atomicAdd(cnt + 3, 1ull);
        else if (__double_as_longlong(r) != __double_as_longlong(__dsqrt_rn(z))) atomicAdd(cnt + 2, 1ull);
        ok = true;
        const double sd = rcp_seed(y, ok);
        if (ok && fabs(fma(-y, sd, 1.0)) > 1.1103e-16) atomicAdd(cnt + 4, 1ull);
    }
}

// Special operands: every one must be declined (or, a zero numerator, keep its sign).
__global__ void k_special(int *wrong) {
    const double bad[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 4.9e-324, -2.2e-308, 1e-200, 1e200, 1.7e308};
    for (double b : bad) {
        bool ok = true;
        div_ieee(1.0, b, ok);
        if (ok) atomicAdd(wrong, 1);
        ok = true;
        sqrt_ieee(b, ok);
        if (ok) atomicAdd(wrong, 1);
        ok = true;
        div_ieee(b, 3.0, ok);
        if (ok && b != 0.0) atomicAdd(wrong, 1);
    }
    bool ok = true;
    sqrt_ieee(-1.0, ok);
    if (ok) atomicAdd(wrong, 1);
    ok = true;
    if (__double_as_longlong(div_ieee(-0.0, 3.0, ok)) != __double_as_longlong(-0.0) || !ok) atomicAdd(wrong, 1);
}

int main(int argc, char **argv) {
    const int reps = argc > 1 ? atoi(argv[1]) : 100;
    unsigned long long *d = nullptr, h[6];
    int *w = nullptr, hw = 0;
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMalloc(&w, sizeof hw) != cudaSuccess) return 2;
    for (int mode = 0; mode < 6; mode++) {
        cudaMemset(d, 0, sizeof h);
        k_check<<<608, 256>>>(mode, reps, d);
        if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        printf("%lld %llu %llu %llu %llu %llu\n", 608ll * 256 * reps, h[0], h[1], h[2], h[3], h[4]);
    }
    cudaMemset(w, 0, sizeof hw);
    k_special<<<1, 1>>>(w);
    if (cudaMemcpy(&hw, w, sizeof hw, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("%d\n", hw);
    return 0;
}

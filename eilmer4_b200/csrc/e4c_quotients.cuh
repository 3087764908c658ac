// e4c_quotients.cuh -- FP64 quotients of the device code, bit for bit IEEE
// division's, in batches.  (Also compiled for the host, by tests/test_quotients.py.)
#pragma once

namespace e4c {

// ---------------------------------------------------------------------------
// Correctly rounded FP64 quotients without a branch per division.
//
// The compiler's a / b carries its own range test and slow-path call, so
// independent divisions run one after the other, each a chain of dependent
// FP64 operations: the reconstruction's limiter values alone are five to
// twenty such chains.  Here one integer test covers a whole batch; inside the
// tested range every quotient is
//   y0 = rcp.approx (about 2^-20), two Newton steps -> y = 1/b rounded from a
//   value within 2^-80 of it,
//   q = a y, then twice: r = a - q b, q = q + r y,
// and the last step is RN(a/b) by the argument of Markstein's theorem (P. W.
// Markstein, IBM J. Res. Develop. 34(1), 1990): q is then within half an ulp
// (and 2^-50 of it) of a/b and r exact, so the sum before rounding misses a/b
// by at most ulp(q)/2 2^-53 (m/2)(1 + 2^-26), m the mantissa of b, while a/b
// is at least ulp(q)/2 2^-53 (2/m) away from any midpoint of two doubles:
// the result is the division's for m^2 < 4 (1 - 2^-26).  Divisors with the top
// 20 mantissa bits set are left to the compiler's division (div_ieee), as are
// operands outside the range (zero or huge divisors, infinities, NaN).
// A dividend of -0 over a positive divisor would come out as +0 (the residual
// is +0, and the correction turns the -0 of the first product into +0), so -0
// goes to the division too, or is shown not to matter where it is let through.
// tests/test_quotients.py compiles these functions for the host (with a poorer
// reciprocal approximation than the hardware's) and compares their bits with
// IEEE division's, the hardest dividends of each divisor among them.
// ---------------------------------------------------------------------------
static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }

__device__ __forceinline__ unsigned abs_hi(double x) {
    return unsigned(__double2hiint(x)) & 0x7fffffffu;
}
// 2^-200 <= |x| < 2^200 (the high words of the two ends)
__device__ __forceinline__ bool quot_range(double x) {
    return abs_hi(x) - 0x33700000u < 0x19000000u;
}
// the same, or +0 (a dividend)
__device__ __forceinline__ bool quot_range0(double x) {
    return quot_range(x) || (__double2hiint(x) | __double2loint(x)) == 0;
}
// a divisor whose top 20 mantissa bits are all set
__device__ __forceinline__ bool top_mantissa(double x) {
    return (unsigned(__double2hiint(x)) & 0xfffffu) == 0xfffffu;
}
__device__ __forceinline__ bool quot_divisor(double x) { return quot_range(x) && !top_mantissa(x); }

// 1/b for quot, b a quot_divisor
__device__ __forceinline__ double rcp_q(double b) {
    double y;
#ifdef __CUDACC__
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#else
    y = approximate_reciprocal(b);   // the host check's
#endif
    double e = fma(-b, y, 1.0);
    y = fma(y, e, y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}
// 1/b for quot, b in quot_range with any mantissa
__device__ __forceinline__ double rcp_any(double b) {
    return top_mantissa(b) ? div_ieee(1.0, b) : rcp_q(b);
}
// a / b from y = rcp_q(b), or y = RN(1/b)
__device__ __forceinline__ double quot(double a, double b, double y) {
    double q = a * y;
    double r = fma(-q, b, a);
    q = fma(r, y, q);
    r = fma(-q, b, a);
    return fma(r, y, q);
}
// one quotient, any operands
__device__ __forceinline__ double fdiv(double a, double b) {
    if (quot_divisor(b) && quot_range0(a)) return quot(a, b, rcp_q(b));
    return div_ieee(a, b);
}
__device__ __forceinline__ float fdiv(float a, float b) { return a / b; }
// N independent quotients, any operands
template <int N>
__device__ __forceinline__ void fdivs(const double* a, const double* b, double* q) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && quot_divisor(b[i]) && quot_range0(a[i]);
    if (ok) {
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = quot(a[i], b[i], rcp_q(b[i]));
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = div_ieee(a[i], b[i]);
    }
}
template <int N>
__device__ __forceinline__ void fdivs(const float* a, const float* b, float* q) {
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = a[i] / b[i];
}
// N quotients n / d of van Albada values: 1e-12 <= n <= d (1 + 2^-52) wherever
// d is finite, so the divisors' upper end is the only test of range
template <int N>
__device__ __forceinline__ void fdiv_va(const double* n, const double* d, double* q) {
    unsigned top = 0u, man = 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const unsigned h = unsigned(__double2hiint(d[i]));
        const unsigned m = h & 0xfffffu;
        top = top > h ? top : h;
        man = man > m ? man : m;
    }
    // every d below 2^200 (and not negative, infinite or NaN)
    if (top < 0x4c700000u && man < 0xfffffu) {
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = quot(n[i], d[i], rcp_q(d[i]));
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = div_ieee(n[i], d[i]);
    }
}
template <int N>
__device__ __forceinline__ void fdiv_va(const float* n, const float* d, float* q) {
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = n[i] / d[i];
}
// a / b with y from the caller's batch (FAST: y = rcp_or(b)), or the plain
// division
template <bool FAST>
__device__ __forceinline__ double quot_or(double a, double b, double y) {
    if constexpr (FAST) return quot(a, b, y);
    else return a / b;
}
template <bool FAST>
__device__ __forceinline__ float quot_or(float a, float b, float) {
    return a / b;
}
template <bool FAST>
__device__ __forceinline__ double rcp_or(double b) {
    if constexpr (FAST) return rcp_q(b);
    else return 0.0;
}
template <bool FAST>
__device__ __forceinline__ float rcp_or(float) {
    return 0.0f;
}
// (a divisor formed inside the batch: its mantissa is tested here)
template <bool FAST>
__device__ __forceinline__ double rcp_or_any(double b) {
    if constexpr (FAST) return rcp_any(b);
    else return 0.0;
}
template <bool FAST>
__device__ __forceinline__ float rcp_or_any(float) {
    return 0.0f;
}

}  // namespace e4c

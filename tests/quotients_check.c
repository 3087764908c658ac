/* The batched quotients of the device code (eilmer4_b200/csrc/e4c_physics.cuh:
 * rcp_q, quot), restated in C for a CPU check against IEEE division
 * (tests/test_quotients.py compiles and runs this).  The hardware's reciprocal
 * approximation is stood in for by the true reciprocal with a relative error
 * of up to 2^-19 of either sign and its low 32 bits cleared: the steps after
 * it must give the same quotient whatever the approximation was.
 * usage: quotients_check <samples>; prints the mismatch count, exits 1 on any. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t next(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double u01(void) { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }

static double seed_of(double b) {
    double y = (1.0 / b) * (1.0 + (u01() * 2.0 - 1.0) * 0x1p-19);
    uint64_t w;
    memcpy(&w, &y, 8);
    w &= 0xffffffff00000000ull;
    memcpy(&y, &w, 8);
    return y;
}
static double rcp_q(double b) {
    double y = seed_of(b);
    double e = fma(-b, y, 1.0);
    y = fma(y, e, y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}
static double quot(double a, double b, double y) {
    double q = a * y;
    double r = fma(-q, b, a);
    q = fma(r, y, q);
    r = fma(-q, b, a);
    return fma(r, y, q);
}
/* a mantissa in [1, 2): random, next to 1 or 2, or of few bits */
static double mant(void) {
    switch (next() & 7) {
        case 0: return 1.0 + (double)(next() & 4095) * 0x1p-52;
        case 1: return 2.0 - (double)(1 + (next() & 4095)) * 0x1p-52;
        case 2: return 1.0 + (double)(next() & 1023) * 0x1p-10;
        default: return 1.0 + u01();
    }
}

/* divisors the device code leaves to the compiler's division */
static int top_mantissa(double b) {
    uint64_t w;
    memcpy(&w, &b, 8);
    return ((w >> 32) & 0xfffff) == 0xfffff;
}
/* the hardest dividend of an odd-mantissa divisor: a = M b -+ one unit in the
 * last place of the product, M a midpoint of two doubles, so that a / b lies
 * as near to a midpoint as any quotient by b can */
static double hardest(double b) {
    int e;
    const uint64_t B = (uint64_t)ldexp(frexp(b, &e), 53);   /* 53 bits, odd */
    uint64_t inv = B;                                       /* inverse of B modulo 2^64 */
    for (int k = 0; k < 6; ++k) inv *= 2 - B * inv;
    const int up = (int)(next() & 1);
    uint64_t M = up ? (0 - inv) : inv;
    const int low = 53 + (int)(next() & 1);                 /* a = (M B +- 1) / 2^low */
    M &= (1ull << low) - 1;
    M |= 1;
    if (low == 53) M |= (1ull << 53);                       /* 54 bits: a midpoint */
    unsigned __int128 p = (unsigned __int128)M * B;
    p = up ? p + 1 : p - 1;
    const uint64_t a = (uint64_t)(p >> low);
    return ldexp((double)a, -40);                           /* exact if a has 53 bits */
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long bad = 0, bad4 = 0, used = 0;
    for (long i = 0; i < n; ++i) {
        double b = ldexp(mant(), (int)(next() % 399) - 199);
        double a = ldexp(mant(), (int)(next() % 399) - 199);
        if (i % 4 == 1) {
            /* a quotient next to the midpoint of two doubles: a = RN((q + ulp/2) b),
             * one step either way */
            const double q = mant();
            a = fma(q, b, b * 0x1p-53);
            if (next() & 1) a = nextafter(a, (next() & 1) ? INFINITY : 0.0);
        } else if (i % 4 == 2) {
            /* a van Albada value: 1e-12 <= n <= d */
            const double x = ldexp(u01() - 0.5, (int)(next() % 80) - 40);
            const double z = ldexp(u01() - 0.5, (int)(next() % 80) - 40);
            a = x * z + fabs(x * z) + 1.0e-12;
            b = x * x + z * z + 1.0e-12;
        }
        if (i % 4 == 3) {
            if (next() & 1) b = (2.0 - (double)(1 + (next() & 0x3ffffff)) * 0x1p-30) * 0.5;
            b = ldexp(ldexp(frexp(b, &(int){0}), 53), -53);
            if (!((uint64_t)ldexp(b, 53) & 1)) b += 0x1p-53;
            a = hardest(b);
        }
        if (top_mantissa(b)) continue;
        ++used;
        if (next() & 1) a = -a;
        if (i % 4 != 2 && (next() & 1)) b = -b;
        const double y = rcp_q(b);
        if (quot(a, b, y) != a / b) ++bad;
        /* a / (4 b) from y / 4, 1 / (4 b) as a quarter of 1 / b */
        if (quot(a, 4.0 * b, 0.25 * y) != a / (4.0 * b)) ++bad4;
        if (0.25 * quot(1.0, b, y) != 1.0 / (4.0 * b)) ++bad4;
    }
    /* zero dividends */
    if (quot(0.0, 3.0, rcp_q(3.0)) != 0.0 || quot(-0.0, 3.0, rcp_q(3.0)) != 0.0) ++bad;
    printf("samples %ld used %ld mismatches %ld %ld\n", n, used, bad, bad4);
    return (bad || bad4 || used < n / 2) ? 1 : 0;
}

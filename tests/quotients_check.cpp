// The device code's quotients (eilmer4_b200/csrc/e4c_quotients.cuh, the file the
// kernels include) compiled for the host and compared bit for bit with IEEE
// division (tests/test_quotients.py builds and runs this).  The hardware's
// reciprocal approximation is stood in for by the true reciprocal with a
// relative error of up to 2^-19 of either sign and its low 32 bits cleared: the
// steps after it must give the same quotient whatever the approximation was.
// usage: quotients_check <samples>; prints the mismatch counts, exits 1 on any.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

static uint64_t bits(double x) {
    uint64_t w;
    memcpy(&w, &x, 8);
    return w;
}
static double from_bits(uint64_t w) {
    double x;
    memcpy(&x, &w, 8);
    return x;
}

static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double u01() { return double(next() >> 11) * (1.0 / 9007199254740992.0); }

#define __device__
#define __forceinline__ inline
#define __noinline__
static int __double2hiint(double x) { return int(bits(x) >> 32); }
static int __double2loint(double x) { return int(uint32_t(bits(x))); }
static double approximate_reciprocal(double b) {
    return from_bits(bits((1.0 / b) * (1.0 + (u01() * 2.0 - 1.0) * 0x1p-19)) & 0xffffffff00000000ull);
}
using std::fma;
#include "e4c_quotients.cuh"
using namespace e4c;

// the same bits, or both NaN
static bool same(double x, double y) { return bits(x) == bits(y) || (x != x && y != y); }

// a mantissa in [1, 2): random, next to 1 or 2, or of few bits
static double mant() {
    switch (next() & 7) {
        case 0: return 1.0 + double(next() & 4095) * 0x1p-52;
        case 1: return 2.0 - double(1 + (next() & 4095)) * 0x1p-52;
        case 2: return 1.0 + double(next() & 1023) * 0x1p-10;
        default: return 1.0 + u01();
    }
}

// the hardest dividend of an odd-mantissa divisor: a = M b -+ one unit in the
// last place of the product, M a midpoint of two doubles, so that a / b lies
// as near to a midpoint as any quotient by b can
static double hardest(double b) {
    int e;
    const uint64_t B = uint64_t(ldexp(frexp(b, &e), 53));   // 53 bits, odd
    uint64_t inv = B;                                       // inverse of B modulo 2^64
    for (int k = 0; k < 6; ++k) inv *= 2 - B * inv;
    const int up = int(next() & 1);
    uint64_t M = up ? (0 - inv) : inv;
    const int low = 53 + int(next() & 1);                   // a = (M B +- 1) / 2^low
    M &= (1ull << low) - 1;
    M |= 1;
    if (low == 53) M |= (1ull << 53);                       // 54 bits: a midpoint
    unsigned __int128 p = (unsigned __int128)M * B;
    p = up ? p + 1 : p - 1;
    return ldexp(double(uint64_t(p >> low)), -40);          // exact if a has 53 bits
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long bad = 0, bad4 = 0, used = 0, any = 0;
    for (long i = 0; i < n; ++i) {
        double b = ldexp(mant(), int(next() % 399) - 199);
        double a = ldexp(mant(), int(next() % 399) - 199);
        if (i % 4 == 1) {
            // a quotient next to the midpoint of two doubles: a = RN((q + ulp/2) b),
            // one step either way
            const double q = mant();
            a = fma(q, b, b * 0x1p-53);
            if (next() & 1) a = nextafter(a, (next() & 1) ? INFINITY : 0.0);
        } else if (i % 4 == 2) {
            // a van Albada value: 1e-12 <= n <= d
            const double x = ldexp(u01() - 0.5, int(next() % 80) - 40);
            const double z = ldexp(u01() - 0.5, int(next() % 80) - 40);
            a = x * z + fabs(x * z) + 1.0e-12;
            b = x * x + z * z + 1.0e-12;
            // (its batch, whatever the mantissa)
            double q;
            fdiv_va<1>(&a, &b, &q);
            if (!same(q, a / b)) ++any;
        }
        if (i % 4 == 3) {
            int e;
            if (next() & 1) b = (2.0 - double(1 + (next() & 0x3ffffff)) * 0x1p-30) * 0.5;
            b = ldexp(ldexp(frexp(b, &e), 53), -53);
            if (!(uint64_t(ldexp(b, 53)) & 1)) b += 0x1p-53;
            a = hardest(b);
        }
        if (next() & 1) a = -a;
        if (i % 4 != 2 && (next() & 1)) b = -b;
        if (i % 64 == 5) a = std::copysign(0.0, a);
        if (!same(e4c::fdiv(a, b), a / b)) ++any;
        if (!quot_divisor(b) || !quot_range0(a)) continue;
        ++used;
        const double y = rcp_q(b);
        if (!same(quot(a, b, y), a / b)) ++bad;
        // a / (4 b) from y / 4, 1 / (4 b) as a quarter of 1 / b
        if (!same(quot(a, 4.0 * b, 0.25 * y), a / (4.0 * b))) ++bad4;
        if (!same(0.25 * quot(1.0, b, y), 1.0 / (4.0 * b))) ++bad4;
        // a mass fraction over a sum near 1, whose reciprocal is a division
        const double sum = 1.0 + double(int(next() % 17) - 8) * 0x1p-53;
        const double f = (next() & 15) ? u01() : 0.0;
        if (!same(quot(f, sum, 1.0 / sum), f / sum)) ++bad;
    }
    // fdiv and a batch of two over all pairs of special operands
    const double ends[] = {0.0, 0x1p-1074, 0x1p-1022, 0x1p-201, 0x1p-200, 0x1.fffffp-200, 1.0,
                           0x1.ffffe8p0, 0x1.fffffp0, 0x1.fffffffffffffp0, 3.0, 0x1p199,
                           0x1.fffffp199, 0x1p200, 0x1p201, 0x1p1023, 0x1.fffffffffffffp1023,
                           INFINITY, NAN};
    for (double p : ends)
        for (double q : ends)
            for (int sign = 0; sign < 4; ++sign) {
                const double a = sign & 1 ? -p : p, b = sign & 2 ? -q : q;
                if (!same(e4c::fdiv(a, b), a / b)) ++any;
                const double n2[2] = {a, -0.0}, d2[2] = {b, 3.0};
                double q2[2];
                fdivs<2>(n2, d2, q2);
                if (!same(q2[0], a / b) || !same(q2[1], -0.0)) ++any;
                if (!(p >= 0x1p-1000 && p <= 0x1p1000) || !quot_range(b)) continue;
                if (!same(rcp_any(b), 1.0 / b)) ++any;
            }
    printf("samples %ld used %ld mismatches %ld %ld %ld\n", n, used, bad, bad4, any);
    return (bad || bad4 || any || used < n / 2) ? 1 : 0;
}

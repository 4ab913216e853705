// Host check of rn_div.h against the plain division, bit for bit: seeded
// divisors and dividends over the fast range and beyond it, significands of
// all ones and of few bits, zeros, infinities, NaN and subnormals.
#include <cstdio>
#include <random>

#include "rn_div.h"

using namespace zsme;

static uint64_t bits(double x) {
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return u;
}
static double make(uint64_t m, int e, uint64_t s) {
    const uint64_t u = (m & ((1ull << 52) - 1)) | ((uint64_t)(e + 1023) << 52) | (s << 63);
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
}
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }

int main() {
    std::mt19937_64 g(1);
    long odd_n = 0, n = 0;
    for (long i = 0; i < 4000000; ++i) {
        uint64_t mb = g(), ma = g();
        if (i % 6 == 1) mb = ~0ull - (g() & 15);
        if (i % 6 == 2) ma = ~0ull - (g() & 7), mb = g() & 15;
        if (i % 6 == 3) mb = g() & 255;
        if (i % 6 == 4) ma = g() & 255, mb = ~0ull - (g() & 255);
        double b = make(mb, (int)(g() % 190) - 95, 0), a = make(ma, (int)(g() % 1900) - 950, g() & 1);
        if (i % 1000 == 0) a = 0.0;
        if (i % 1001 == 0) a = INFINITY;
        if (i % 1002 == 0) a = NAN;
        if (i % 1003 == 0) a = make(ma, -1023, 0);   // subnormal
        if (i % 1004 == 0) b = make(mb, (int)(g() % 2000) - 1000, 0);
        const RnDivisor d(b);
        const double t = a / b;
        const RnDivisor neg(-b);
        if (!same(d.quotient(a), t) || !same(d.quotient(-a), -t) || !same(neg.quotient(a), -t))
            return printf("quotient %a / %a\n", a, b), 1;
        bool odd = false;
        const double q = d.quotient_or(a, odd);
        if (!odd && !same(q, t)) return printf("quotient_or %a / %a\n", a, b), 1;
        odd_n += odd;
        odd = false;
        const double qs = neg.signed_quotient_or(a, odd);
        if (!odd && !same(qs, -t)) return printf("signed_quotient_or %a / %a\n", a, -b), 1;
        odd = false;
        const double y = rn_reciprocal(b, odd);
        bool odd_neg = false;
        const double yn = rn_reciprocal(-b, odd_neg);
        if (odd_neg != odd || (!odd && (!same(y, 1.0 / b) || !same(yn, -1.0 / b))))
            return printf("rn_reciprocal %a\n", b), 1;
        ++n;
    }
    printf("checked %ld odd %ld\n", n, odd_n);
    return 0;
}

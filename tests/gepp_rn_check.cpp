// Host check of gepp_unswapped against gepp_regs, bit for bit: seeded blocks of
// every size a plugin has, dominant and not, with zeros, tiny and huge entries,
// unless the former reports itself odd (as it does wherever rows are swapped).
#include <cstdio>
#include <random>

#include "gepp_regs.h"

using namespace zsme;

template <int NB>
static long check(long n, long& odd_n) {
    std::mt19937_64 g(NB);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (long t = 0; t < n; ++t) {
        double A[NB][NB], b[NB], x[NB], P[NB][NB], pb[NB], px[NB];
        for (int i = 0; i < NB; ++i) {
            for (int j = 0; j < NB; ++j) {
                A[i][j] = u(g) * (t % 3 == 0 ? std::pow(10.0, 8 * u(g)) : 1.0) + (i == j && t % 2 ? 8.0 : 0.0);
                if (t % 5 == 0 && g() % 4 == 0) A[i][j] = 0.0;
                P[i][j] = A[i][j];
            }
            b[i] = u(g) * std::pow(10.0, t % 7 == 0 ? 300 * u(g) : 0.0);
            if (t % 11 == 0 && g() % 2) b[i] = g() % 2 ? -0.0 : 0.0;
            pb[i] = b[i];
        }
        bool odd = false;
        const bool ok = gepp_unswapped<NB>(A, b, x, odd), pok = gepp_regs<NB>(P, pb, px);
        odd_n += odd;
        if (odd || !pok) continue;
        if (ok != pok || std::memcmp(x, px, sizeof x)) return printf("NB %d trial %ld\n", NB, t), 1;
    }
    return 0;
}

int main() {
    long odd = 0;
    const long n = 100000;
    if (check<1>(n, odd) || check<2>(n, odd) || check<3>(n, odd) || check<5>(n, odd) || check<6>(n, odd)) return 1;
    printf("checked %ld odd %ld\n", 5 * n, odd);
    return 0;
}

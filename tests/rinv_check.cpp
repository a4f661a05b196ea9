// Worst relative error of csrc/rinv.cuh's (d^2 + eps^2)^(-3/2) and ^(-1/2)
// against long double over seeded random separations; prints name value pairs.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../vipp-nbody-bench_gb300/csrc/rinv.cuh"

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    const double scale = std::atof(argv[1]), eps = std::atof(argv[2]);
    const int n = std::atoi(argv[3]);
    const double eps2 = eps * eps;
    const gb::SoftInt e = gb::soft_int(eps2);
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> U(-1, 1);
    long double m3 = 0, m1 = 0;
    int out = 0;
    for (int i = 0; i < n; ++i) {
        double d[3];
        for (double &c : d) c = scale * U(g) * std::pow(2.0, -30 * std::fabs(U(g)));
        if (i % 7 == 0) d[i % 3] = 0;
        if (i % 11 == 0) d[0] = d[1] = 0;
        double f3, f1;
        const bool ok = gb::rinv3(d[0], d[1], d[2], e, f3);
        if (gb::rinv1(d[0], d[1], d[2], e, f1) != ok) return 3;
        if (!ok) {
            if (d[0] != 0 || d[1] != 0 || d[2] != 0) ++out;  // a zero separation without softening has no factor
            continue;
        }
        const long double u = static_cast<long double>(d[0]) * d[0] + static_cast<long double>(d[1]) * d[1] +
                              static_cast<long double>(d[2]) * d[2] + static_cast<long double>(eps2);
        const long double t = 1 / std::sqrt(u), t3 = t * t * t;
        m3 = std::fmax(m3, std::fabs((static_cast<long double>(f3) - t3) / t3));
        m1 = std::fmax(m1, std::fabs((static_cast<long double>(f1) - t) / t));
    }
    std::printf("max3 %.3Le max1 %.3Le out %d\n", m3, m1, out);
    return 0;
}

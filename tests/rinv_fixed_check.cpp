// csrc/rinv.cuh's fixed-point pair (pair_fixed) against long double over seeded
// random positions about an offset; prints name value pairs: worst relative error
// of the factor and of the separation (against its largest component) in the pairs
// it takes, their number, and the number it leaves to the FP64 difference.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../vipp-nbody-bench_gb300/csrc/rinv.cuh"

int main(int argc, char **argv) {
    if (argc < 5) return 2;
    const double scale = std::atof(argv[1]), offset = std::atof(argv[2]), eps = std::atof(argv[3]);
    const int n = std::atoi(argv[4]);
    const gb::SoftInt e = gb::soft_int(eps * eps);
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(-1, 1);
    double x[64][3];
    long double mf = 0, md = 0, sf = 0;
    long taken = 0, left = 0, frames = 0;
    for (int rep = 0; rep < n; ++rep) {
        int top = 0;
        for (int i = 0; i < 64; ++i)
            for (int a = 0; a < 3; ++a) {
                x[i][a] = offset + scale * U(g) * std::pow(2.0, i % 5 == 0 ? -20 * std::fabs(U(g)) : 0);
                // separations a few quanta below a power of two
                if (i % 13 == 1 && a == rep % 3) x[i][a] = offset + scale * 0.25;
                if (i % 13 == 2 && a == rep % 3) x[i][a] = offset + scale * std::ldexp(1.0, -57 - rep % 4);
                if (i % 9 == 0 && a == rep % 3) x[i][a] = x[0][a];  // planes
                const int ex = static_cast<int>((gb::rinv::hi_word(x[i][a] - x[0][a]) >> 20) & 0x7FFu);
                if (ex > top) top = ex;
            }
        const gb::Frame f = gb::make_frame(top, e);
        frames += f.ok;
        if (!f.ok) continue;
        for (int i = 0; i < 64; ++i)
            for (int j = 0; j < 64; ++j) {
                if (i == j) continue;
                long long q[3];
                long double d[3], big = 0, u = static_cast<long double>(eps * eps);
                for (int a = 0; a < 3; ++a) {
                    q[a] = static_cast<long long>(static_cast<unsigned long long>(gb::fixed_point(x[j][a], f.qf)) -
                                                  static_cast<unsigned long long>(gb::fixed_point(x[i][a], f.qf)));
                    d[a] = static_cast<long double>(x[j][a]) - x[i][a];
                    u += d[a] * d[a];
                    big = std::fmax(big, std::fabs(d[a]));
                }
                double fac, s[3];
                if (!gb::pair_fixed(q[0], q[1], q[2], e, f, fac, s[0], s[1], s[2])) {
                    ++left;
                    continue;
                }
                ++taken;
                const long double t = 1 / std::sqrt(u), t3 = t * t * t, r = std::fabs((fac - t3) / t3);
                mf = std::fmax(mf, r), sf += r * r;
                for (int a = 0; a < 3; ++a) md = std::fmax(md, std::fabs(s[a] - d[a]) / big);
            }
    }
    std::printf("factor %.3Le rms %.3Le separation %.3Le taken %ld left %ld frames %ld\n", mf, std::sqrt(sf / (taken ? taken : 1)), md,
                taken, left, frames);
    return 0;
}

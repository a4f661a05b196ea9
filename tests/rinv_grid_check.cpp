// Separations of csrc/rinv.cuh as the two kernels that use them take them, against long
// double, one component at a time, over a sheet normal to `axis` of half-thickness h about
// an offset along it: the worst error in units of 2^-53 of the component itself of
//   near    pairs of two positions on the grid (the near field; the others take the FP64 difference)
//   direct  sources on the grid, and components that are not too_short to the target (the direct sum)
// the worst relative error of their factor in units of 2^-51 (on the grid) and 2^-50 (off it),
// and how many pairs or components of each were taken and left, and how many differences
// have their positions on either side of a multiple of 2^63 quanta.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../vipp-nbody-bench_gb300/csrc/rinv.cuh"

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    const int axis = std::atoi(argv[1]);
    const double h = std::atof(argv[2]), offset = std::atof(argv[3]), extent = argc > 4 ? std::atof(argv[4]) : 1;
    const gb::SoftInt e = gb::soft_int(1e-4);
    std::mt19937_64 g(11);
    std::uniform_real_distribution<double> U(-1, 1);
    constexpr int kN = 96;
    double x[kN][3];
    long double near = 0, direct = 0, factor = 0;
    long wraps = 0, near_taken = 0, near_left = 0, direct_taken = 0, direct_left = 0;
    for (int rep = 0; rep < 60; ++rep) {
        int top = 0;
        for (int i = 0; i < kN; ++i)
            for (int a = 0; a < 3; ++a) {
                x[i][a] = (a == axis ? offset + h * U(g) : extent * U(g)) * 0.91;  // full mantissas
                const int ex = static_cast<int>((gb::rinv::hi_word(x[i][a] - x[0][a]) >> 20) & 0x7FFu);
                if (ex > top) top = ex;
            }
        const gb::Frame f = gb::make_frame(top, e);
        if (!f.ok) return 3;
        for (int i = 0; i < kN; ++i)
            for (int j = 0; j < kN; ++j) {
                if (i == j) continue;
                int64_t q[3];
                bool on[2][3];
                for (int a = 0; a < 3; ++a) {
                    q[a] = gb::separation(gb::fixed_point(x[j][a], f.qf), gb::fixed_point(x[i][a], f.qf));
                    wraps += (gb::fixed_point(x[j][a], f.qf) >> 63) != (gb::fixed_point(x[i][a], f.qf) >> 63);
                    on[0][a] = gb::on_grid(x[i][a], f.qf), on[1][a] = gb::on_grid(x[j][a], f.qf);
                }
                double fac, s[3];
                if (!gb::pair_fixed(q[0], q[1], q[2], e, f, fac, s[0], s[1], s[2])) continue;
                const bool source_on = on[1][0] && on[1][1] && on[1][2];
                const bool both_on = source_on && on[0][0] && on[0][1] && on[0][2];
                both_on ? ++near_taken : ++near_left;
                long double u = static_cast<long double>(1e-4);
                const bool source_xy = on[1][0] && on[1][1];
                for (int a = 0; a < 3; ++a) {
                    const long double d = static_cast<long double>(x[j][a]) - x[i][a];
                    u += d * d;
                    const long double err = d == 0 ? (s[a] == 0 ? 0 : 1e30L) : std::fabs((s[a] - d) / d) * 0x1p53L;
                    if (both_on) near = std::fmax(near, err);
                    if (a == 2) continue;  // the direct sum has z from the FP64 pipe
                    if (source_xy && !gb::too_short(q[a], on[0][a] ? 0 : gb::kOffGrid))
                        direct = std::fmax(direct, err), ++direct_taken;
                    else
                        ++direct_left;
                }
                const long double t = 1 / std::sqrt(u);
                factor = std::fmax(factor, std::fabs((fac - t * t * t) / (t * t * t)) * (both_on ? 0x1p51L : 0x1p50L));
            }
    }
    std::printf("near %.4Lf direct %.4Lf factor %.4Lf near_taken %ld near_left %ld direct_taken %ld direct_left %ld wraps %ld\n", near, direct,
                factor, near_taken, near_left, direct_taken, direct_left, wraps);
    return 0;
}

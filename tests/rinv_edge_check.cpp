// Worst relative error of csrc/rinv.cuh's factors at separations within a few ulp of
// 2^k (whose factors lie within a few ulp of a power of two, on both sides).
#include <cstdio>
#include <cmath>

#include "../vipp-nbody-bench_gb300/csrc/rinv.cuh"

int main() {
    long double worst = 0;
    const gb::SoftInt none = gb::soft_int(0.0);
    for (int k = -40; k <= 40; ++k)
        for (int u = -600; u <= 600; ++u)
            for (int c = 0; c < 3; ++c) {
                double d[3] = {0, 0, 0};
                d[c] = std::ldexp(1.0 + u * (u < 0 ? 0x1p-53 : 0x1p-52), k);
                double f3, f1;
                if (!gb::rinv3(d[0], d[1], d[2], none, f3) || !gb::rinv1(d[0], d[1], d[2], none, f1)) return 3;
                const long double t = 1 / static_cast<long double>(d[c]), t3 = t * t * t;
                worst = std::fmax(worst, std::fmax(std::fabs((f3 - t3) / t3), std::fabs((f1 - t) / t)));
            }
    std::printf("%.3Le\n", worst);
    return 0;
}

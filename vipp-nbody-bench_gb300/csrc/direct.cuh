// FP64 direct softened sum (the accuracy oracle of the GPU path;
// gravity/include/solver_ref_naive.hpp:103-119), split over sources.
//
// Few targets against many sources (the 65,536-particle error sample of a
// 4M-particle system) leave most SMs idle with one thread per target, so the
// sources are cut into `nsplit` slices: block (bx, sy) sums slice sy for 256
// targets into the scratch buffer part[sy][3][nt], and a second kernel adds
// the slices in slice order (deterministic).
//
// Position and output layouts are policies: SoA planes [3][n] (the solver
// context's own buffers) or AoS triples (caller buffers).
#pragma once

#include <climits>

#include <cuda_runtime.h>

#include "rinv.cuh"

namespace gb {

struct SoA {
    const double *p;
    unsigned n;
    __device__ __forceinline__ double x(unsigned i) const { return p[i]; }
    __device__ __forceinline__ double y(unsigned i) const { return p[n + i]; }
    __device__ __forceinline__ double z(unsigned i) const { return p[2 * static_cast<size_t>(n) + i]; }
};

struct AoS {
    const double *p;
    __device__ __forceinline__ double x(unsigned i) const { return p[3 * static_cast<size_t>(i)]; }
    __device__ __forceinline__ double y(unsigned i) const { return p[3 * static_cast<size_t>(i) + 1]; }
    __device__ __forceinline__ double z(unsigned i) const { return p[3 * static_cast<size_t>(i) + 2]; }
};

constexpr int kDirectTB = 256;

// Sources in tiles, each with its frame (rinv.cuh). Bound by the issue of integer
// instructions (about 230 a pair, 4.2 FP64): 4,096 targets over 262,144 Plummer sources
// 35.2 ms with the FP64 factor, 11.7 with the integer factor, 9.0 with x's and y's
// separations from the frame (z's stays on the FP64 pipe, which has room for it).
// The frame of a tile is as wide as the system, so a few percent of the coordinates
// are off its grid (rinv.cuh): x and y of a source off it, and those below 2^54 quanta to
// a target off it (too_short), come from the FP64 pipe like z, one at a time. What is taken
// is within 5/4 2^-53 of each component. The factor follows the pair's norm: off the grid
// it is within 2^-50, as the FP64 form's.
//
// high word of the largest |component|: orders like the component; above 0x7FEFFFFF for infinities and NaN
__device__ __forceinline__ unsigned top_word(double x, double y, double z) {
    return max(static_cast<unsigned>(__double2hiint(x)) & 0x7FFFFFFFu,
               max(static_cast<unsigned>(__double2hiint(y)) & 0x7FFFFFFFu, static_cast<unsigned>(__double2hiint(z)) & 0x7FFFFFFFu));
}

// dx = dy = dz = 0, off the FP64 pipe (three comparisons hold it as long as the three sums of a pair)
__device__ __forceinline__ bool all_zero(double dx, double dy, double dz) {
    return (top_word(dx, dy, dz) | static_cast<unsigned>(__double2loint(dx) | __double2loint(dy) | __double2loint(dz))) == 0;
}

// kCheckTargets: target indices come from device memory the host never saw;
// an index outside [0, n) is not dereferenced and its result is NaN.
template <class Pos, bool kCheckTargets = false>
__global__ void __launch_bounds__(kDirectTB) k_direct_part(Pos pos, unsigned n, const long long *__restrict__ targets,
                                                           unsigned nt, unsigned nsplit, double Gm, double eps2, SoftInt soft,
                                                           double *__restrict__ part) {
    __shared__ double sx[kDirectTB], sy[kDirectTB], sz[kDirectTB], ref[3];
    __shared__ uint64_t fx[kDirectTB], fy[kDirectTB], fz[kDirectTB];
    __shared__ unsigned wtop[kDirectTB / 32], sgrid[kDirectTB / 32];
    const unsigned k = blockIdx.x * kDirectTB + threadIdx.x;
    bool act = k < nt;
    bool bad = false;
    long long ti = act ? (targets ? targets[k] : static_cast<long long>(k)) : 0;
    if (kCheckTargets && act && (ti < 0 || ti >= static_cast<long long>(n))) {
        bad = true;
        act = false;
        ti = 0;
    }
    const unsigned i = static_cast<unsigned>(ti);
    const double tx = act ? pos.x(i) : 0.0, ty = act ? pos.y(i) : 0.0, tz = act ? pos.z(i) : 0.0;
    const unsigned per = (n + nsplit - 1) / nsplit;
    const unsigned lo = blockIdx.y * per;
    const unsigned hi = min(n, lo + per);
    double ax = 0, ay = 0, az = 0;
    // frames: extents of the block's targets and of a tile's sources about the first target
    if (threadIdx.x == 0) ref[0] = tx, ref[1] = ty, ref[2] = tz;
    __syncthreads();
    const unsigned ttop = act ? top_word(tx - ref[0], ty - ref[1], tz - ref[2]) : 0u;
    int qf = INT_MIN, kx = 0, ky = 0;
    uint64_t gx = 0, gy = 0, gz = 0;
    for (unsigned b = lo; b < hi; b += kDirectTB) {
        const unsigned j = b + threadIdx.x;
        double px = 0, py = 0, pz = 0;
        unsigned top = ttop;
        if (j < hi) {
            px = pos.x(j), py = pos.y(j), pz = pos.z(j);
            sx[threadIdx.x] = px;
            sy[threadIdx.x] = py;
            sz[threadIdx.x] = pz;
            top = max(top, top_word(px - ref[0], py - ref[1], pz - ref[2]));
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if ((threadIdx.x & 31) == 0) wtop[threadIdx.x >> 5] = top;
        __syncthreads();
        for (int w = 0; w < kDirectTB / 32; ++w) top = max(top, wtop[w]);
        const Frame fr = make_frame(static_cast<int>(top >> 20), soft);
        if (fr.ok) {
            fx[threadIdx.x] = fixed_point(px, fr.qf), fy[threadIdx.x] = fixed_point(py, fr.qf), fz[threadIdx.x] = fixed_point(pz, fr.qf);
            if (fr.qf != qf) {
                qf = fr.qf, gx = fixed_point(tx, qf), gy = fixed_point(ty, qf), gz = fixed_point(tz, qf);
                kx = on_grid(tx, qf) ? 0 : kOffGrid, ky = on_grid(ty, qf) ? 0 : kOffGrid;
            }
            const unsigned g = __ballot_sync(0xffffffffu, on_grid(px, qf) && on_grid(py, qf));
            if ((threadIdx.x & 31) == 0) sgrid[threadIdx.x >> 5] = g;
        }
        __syncthreads();
        const unsigned cnt = min(static_cast<unsigned>(kDirectTB), hi - b);
        for (unsigned q0 = 0; q0 < cnt; q0 += 32) {
            unsigned grid = sgrid[q0 >> 5];
            const unsigned q1 = min(q0 + 32, cnt);
#pragma unroll 1
            for (unsigned q = q0; q < q1; ++q, grid >>= 1) {
                if (b + q == i) continue;  // i == j is skipped (solver_ref_naive.hpp:109-111)
                double f, dx, dy, unused, dz = sz[q] - tz;
                const int64_t hx = separation(fx[q], gx), hy = separation(fy[q], gy);
                if (fr.ok && pair_fixed(hx, hy, separation(fz[q], gz), soft, fr, f, dx, dy, unused)) {
                    if (!(grid & 1u) || too_short(hx, kx)) dx = sx[q] - tx;
                    if (!(grid & 1u) || too_short(hy, ky)) dy = sy[q] - ty;
                } else {
                    dx = sx[q] - tx, dy = sy[q] - ty;
                    if (!rinv3(dx, dy, dz, soft, f)) {
                        // r^-3 leaves FP64's range at 1e103 and 1e-103, r^-2 (d / r) only with the result
                        const double ri = rsqrt(dx * dx + dy * dy + dz * dz + eps2);
                        f = ri * ri;
                        dx *= ri, dy *= ri, dz *= ri;
                    }
                }
                ax += f * dx;
                ay += f * dy;
                az += f * dz;
            }
        }
        __syncthreads();
    }
    if (act || bad) {
        if (bad) ax = ay = az = __longlong_as_double(0x7ff8000000000000LL);
        double *o = part + static_cast<size_t>(blockIdx.y) * 3 * nt;
        o[k] = Gm * ax;
        o[nt + k] = Gm * ay;
        o[2 * static_cast<size_t>(nt) + k] = Gm * az;
    }
}

// out_soa: planes [3][nt]; out_aos: triples. Exactly one of them is non-null.
static __global__ void k_direct_reduce(const double *__restrict__ part, unsigned nt, unsigned nsplit, double *__restrict__ out_soa,
                                double *__restrict__ out_aos) {
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt) return;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double s = 0;
        for (unsigned q = 0; q < nsplit; ++q) s += part[(static_cast<size_t>(q) * 3 + a) * nt + k];
        if (out_soa)
            out_soa[static_cast<size_t>(a) * nt + k] = s;
        else
            out_aos[3 * static_cast<size_t>(k) + a] = s;
    }
}

// Source slices that fill about four waves of blocks, at least 256 sources each.
inline unsigned direct_nsplit(unsigned n, unsigned nt, int num_sms) {
    const unsigned bx = (nt + kDirectTB - 1) / kDirectTB;
    unsigned s = (4u * static_cast<unsigned>(num_sms) + bx - 1) / (bx ? bx : 1);
    const unsigned smax = n / kDirectTB > 0 ? n / kDirectTB : 1;
    if (s > smax) s = smax;
    if (s > 256) s = 256;
    return s ? s : 1;
}

}  // namespace gb

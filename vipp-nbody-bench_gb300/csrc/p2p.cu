// Near field (P2P, gravity/include/fmm.hpp:377-385, 513-540) and the FP64
// direct-sum oracle (solver_ref_naive.hpp:103-119) on the GPU.
//
// Work decomposition: every leaf is cut into chunks (common.cuh chunk_at):
// full chunks of 32 targets, and remainders of t < 32 targets that run
// floor(32/t) lane groups over disjoint subsets of the same sources (combined
// at the end through shared memory), so small leaves keep most lanes busy. A
// persistent grid of warps pulls chunks from a device counter (work queue).
// A warp streams the leaf's near-field source ranges through shared memory
// 32 sources at a time, prefetching the next batch into registers while it
// works on the current one; lanes read the staged sources with broadcast
// shared-memory loads, two sources per step on paired FP32 instructions in
// chunks of every size (a slice's last batch is filled up with sources that add
// nothing).
//
// Mixed precision (FP32): positions are kept as hi + lo float pairs relative
// to the root-box centre; targets and staged sources are re-expressed relative
// to the target leaf's centre ((hi - c_hi) + (lo - c_lo)), so FP32 differences
// carry ~1e-7 of the neighbourhood size rather than of the coordinate.
// Pair term: rsqrt.approx.ftz (a Newton step on request: it leaves the RMS
// error unchanged to 1e-10 at 20% of the cost), r^-3 d (equal masses: m
// and the reference's G, fmm.hpp:539, multiply the sum once); per-batch FP32
// partial sums folded into a compensated (Kahan) per-target accumulator.
#include "direct.cuh"
#include "rinv.cuh"
#include "workspace.cuh"

namespace gb {

namespace {

constexpr int kP2PWarps = 4;

__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Source batches of a slice [v0, v0 + len) of the concatenation of a leaf's
// source ranges: up to 32 sources taken across range boundaries, lane l getting
// the l-th (a batch is cut only at the slice's end). The state is uniform over
// the warp; the ranges are read 32 at a time, one per lane, and handed around by
// shuffles, so that neither finding the slice's start nor crossing into the next
// range waits for a chain of dependent loads (a range holds ~155 sources at 4M).
struct BatchCursor {
    const uint2 *rng;
    uint2 mine;  // range r0 + lane
    unsigned nr, r0, r, b, end, rem;
    __device__ __forceinline__ void window(unsigned lane) {
        mine = r0 + lane < nr ? rng[r0 + lane] : make_uint2(0, 0);
    }
    __device__ __forceinline__ void start(const uint2 *ranges, unsigned n, unsigned v0, unsigned len, unsigned lane) {
        rng = ranges, nr = n, r0 = 0, rem = len, b = 0, end = 0;
        window(lane);
        while (true) {
            unsigned cum = mine.y - mine.x;  // sources of this window's ranges up to and with this lane's
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, cum, o);
                if (lane >= o) cum += y;
            }
            const unsigned past = __ballot_sync(0xffffffffu, cum > v0);
            if (past) {
                const int q = __ffs(past) - 1;
                const unsigned at = __shfl_sync(0xffffffffu, mine.y - (cum - v0), q);
                r = r0 + q, b = at, end = __shfl_sync(0xffffffffu, mine.y, q);
                return;
            }
            v0 -= __shfl_sync(0xffffffffu, cum, 31);
            r0 += 32;
            if (r0 >= nr) {  // an empty slice
                r = nr, rem = 0;
                return;
            }
            window(lane);
        }
    }
    // the next batch: its size, and this lane's source index (lane < size)
    __device__ __forceinline__ unsigned next(unsigned lane, unsigned &idx) {
        unsigned filled = 0;
        idx = 0;
        while (filled < 32u && rem > 0 && r < nr) {
            const unsigned take = min(min(32u - filled, end - b), rem);
            if (lane >= filled && lane < filled + take) idx = b + (lane - filled);
            filled += take, rem -= take, b += take;
            if (b >= end && ++r < nr) {
                if (r - r0 == 32) r0 = r, window(lane);
                b = __shfl_sync(0xffffffffu, mine.x, r - r0), end = __shfl_sync(0xffffffffu, mine.y, r - r0);
            }
        }
        return filled;
    }
};

// Work item -> (leaf, first target, targets, slices [sl, se) of ns, slot of the
// first slice's partial sums). An item with all of its leaf's slices adds their
// sums in slice order itself; else k_p2p_combine does.
struct Item {
    int li, t0, nt, sl, se, ns, pslot;
    __device__ __forceinline__ explicit Item(const int4 w)
        : li(w.x), t0(w.y), nt(item_nt(w.z)), sl(item_slice(w.z)), ns(item_nslices(w.z)), pslot(w.w) {}
    __device__ __forceinline__ void of_leaf(int spi) { se = min(ns, sl + spi); }
    __device__ __forceinline__ bool whole() const { return sl == 0 && se == ns; }
};
// A source pair (j, j') against a target on paired FP32 instructions (.f32x2);
// each component rounds exactly like the scalar operation.
template <bool kNewton, bool kSoft>
__device__ __forceinline__ void pair2_f32(float2 x, float2 y, float2 z, float2 ntx, float2 nty, float2 ntz, float2 e2,
                                          float2 &ax, float2 &ay, float2 &az) {
    const float2 dx = __fadd2_rn(x, ntx), dy = __fadd2_rn(y, nty), dz = __fadd2_rn(z, ntz);
    float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
    if (kNewton) r2.x = fminf(r2.x, 3e38f), r2.y = fminf(r2.y, 3e38f);  // the step makes a NaN of infinity
    float2 ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    if (kNewton) {
        ri.x = ri.x * fmaf(-0.5f * r2.x * ri.x, ri.x, 1.5f);
        ri.y = ri.y * fmaf(-0.5f * r2.y * ri.y, ri.y, 1.5f);
    }
    if (!kSoft) ri.x = r2.x > 0.f ? ri.x : 0.f, ri.y = r2.y > 0.f ? ri.y : 0.f;
    const float2 f = __fmul2_rn(ri, __fmul2_rn(ri, ri));
    ax = __ffma2_rn(dx, f, ax);
    ay = __ffma2_rn(dy, f, ay);
    az = __ffma2_rn(dz, f, az);
}

// Coordinate of the sources that fill up a slice's last batch. r^2 overflows and its
// reciprocal root is 0, so they add exactly nothing, whatever the system's size (1e18, where
// r^-3 underflows, lay inside systems of that size).
constexpr float kNowhere = 1e30f;

// Compiled for 6 resident blocks per SM (80 registers). Bound by the FMA pipe
// and what a batch costs beside its pairs: the pair loop alone reaches 8.9 pairs
// per clock and SM (11 FP32 operations a pair: 84% of the measured FMA rate), with
// the staging of a batch and the compensated sums 8.0, with the 94% of lanes that
// a leaf's chunks fill 7.5; the kernel runs at 7.0 (4M Plummer, 1.03e10 pairs: 4.83
// ms, 4.92 before; 1M unit cube 0.475 -> 0.465; 1M at p = 10 2.06 -> 1.96). A
// 64-register build (8 blocks) spills 24 bytes and measured 1-5% slower on every
// workload; a 96-register build kept the cluster M2M from starting beside P2P. The
// softened kMulti build spills 8 bytes.
// kMulti: items of several consecutive slices (a forest's); a single tree's items are
// one slice each, and the bookkeeping between slices costs the kernel 1.7%.
template <bool kNewton, bool kSoft, bool kMulti>
__global__ void __launch_bounds__(kP2PWarps * 32, 6) k_p2p_f32(const int4 *__restrict__ chunks, const unsigned *counts,
                                                            unsigned *queue, const LeafRec *__restrict__ recs,
                                                            const uint2 *__restrict__ ranges, const float4 *__restrict__ ph,
                                                            const float4 *__restrict__ pl, float *__restrict__ part, float Gm,
                                                            float eps2, float *__restrict__ nearv, unsigned n) {
    __shared__ __align__(16) float src[kP2PWarps][3][32];  // the staged batch, leaf-relative
    __shared__ float red[kP2PWarps][3][32], sum[kMulti ? kP2PWarps : 1][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned nch = counts[5];
    unsigned ci = 0;
    if (lane == 0) ci = atomicAdd(queue, 1u);
    while (true) {
        ci = __shfl_sync(0xffffffffu, ci, 0);
        if (ci >= nch) break;
        Item it(chunks[ci]);
        const LeafRec rec = recs[it.li];
        it.of_leaf(rec.spi);
        const int nt = it.nt;
        const int g = 32 / nt;
        const int grp = lane / nt;
        const int t = lane - grp * nt;
        const bool tact = grp < g;
        const int i = it.t0 + t;
        // minus the leaf centre: a position is (hi - centre hi) + (lo - centre lo)
        const float2 chxy = make_float2(-rec.hx, -rec.hy), clxy = make_float2(-rec.lx, -rec.ly);
        const float chz = -rec.hz, clz = -rec.lz;
        float2 txy = make_float2(0.f, 0.f);
        float tz = 0;
        if (tact) {
            const float4 h = ph[i], l = pl[i];
            txy = __fadd2_rn(__fadd2_rn(make_float2(h.x, h.y), chxy), __fadd2_rn(make_float2(l.x, l.y), clxy));
            tz = (h.z + chz) + (l.z + clz);
        }
        const float2 ntx = make_float2(-txy.x, -txy.x), nty = make_float2(-txy.y, -txy.y), ntz = make_float2(-tz, -tz);
        const float2 e2 = make_float2(eps2, eps2);
        // Consecutive slices share one stream of batches (a batch ends with its slice);
        // a slice's sum goes to the item's sums in shared memory, or to its slot.
        if (kMulti) sum[w][0][lane] = 0.f, sum[w][1][lane] = 0.f, sum[w][2][lane] = 0.f;
        float sx = 0, sy = 0, sz = 0, kx = 0, ky = 0, kz = 0;  // Kahan sums and compensations
        auto slice_sum = [&]() {  // of the lane groups, in group 0
            sx -= kx, sy -= ky, sz -= kz;
            if (g > 1) {
                red[w][0][lane] = sx, red[w][1][lane] = sy, red[w][2][lane] = sz;
                __syncwarp();
                if (grp == 0)
                    for (int q = 1; q < g; ++q)
                        sx += red[w][0][t + q * nt], sy += red[w][1][t + q * nt], sz += red[w][2][t + q * nt];
                __syncwarp();
            }
        };
        int sl = it.sl;
        const unsigned v0 = min(rec.src_total, static_cast<unsigned>(sl) * rec.slice);
        unsigned left = rec.src_total - v0;  // sources from this slice on
        BatchCursor cur;
        cur.start(ranges + rec.rng_off, rec.rng_len, v0, min(rec.slice, left), static_cast<unsigned>(lane));
        float4 h = make_float4(0, 0, 0, 0), l = h;
        unsigned sidx;
        unsigned cnt = cur.next(static_cast<unsigned>(lane), sidx);
        if (static_cast<unsigned>(lane) < cnt) h = ph[sidx], l = pl[sidx];
        bool taken = false;
        while (cnt) {
            const bool on = static_cast<unsigned>(lane) < cnt;
            const float2 xy = __fadd2_rn(__fadd2_rn(make_float2(h.x, h.y), chxy), __fadd2_rn(make_float2(l.x, l.y), clxy));
            src[w][0][lane] = on ? xy.x : kNowhere;
            src[w][1][lane] = xy.y;
            src[w][2][lane] = (h.z + chz) + (l.z + clz);
            __syncwarp();
            const bool ends = cur.rem == 0;  // the staged batch is its slice's last
            if (kMulti && ends && ++sl < it.se) {
                left -= rec.slice;
                cur.rem = min(rec.slice, left);
            } else if (ends && !taken) {  // nothing more to fetch: take the next item
                taken = true;
                if (lane == 0) ci = atomicAdd(queue, 1u);
            }
            cnt = cur.next(static_cast<unsigned>(lane), sidx);  // prefetch the next batch while this one is computed
            if (static_cast<unsigned>(lane) < cnt) h = ph[sidx], l = pl[sidx];
            float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
            if (g == 1) {
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const float4 x = reinterpret_cast<const float4 *>(src[w][0])[m];
                    const float4 y = reinterpret_cast<const float4 *>(src[w][1])[m];
                    const float4 z = reinterpret_cast<const float4 *>(src[w][2])[m];
                    pair2_f32<kNewton, kSoft>(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), ntx, nty, ntz,
                                              e2, ax, ay, az);
                    pair2_f32<kNewton, kSoft>(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), ntx, nty, ntz,
                                              e2, ax, ay, az);
                }
            } else {
#pragma unroll 2
                for (int m = tact ? grp : 16; m < 16; m += g)
                    pair2_f32<kNewton, kSoft>(reinterpret_cast<const float2 *>(src[w][0])[m],
                                              reinterpret_cast<const float2 *>(src[w][1])[m],
                                              reinterpret_cast<const float2 *>(src[w][2])[m], ntx, nty, ntz, e2, ax, ay, az);
            }
            __syncwarp();
            float y = (ax.x + ax.y) - kx, tt = sx + y;
            kx = (tt - sx) - y, sx = tt;
            y = (ay.x + ay.y) - ky, tt = sy + y;
            ky = (tt - sy) - y, sy = tt;
            y = (az.x + az.y) - kz, tt = sz + y;
            kz = (tt - sz) - y, sz = tt;
            if (kMulti && ends) {
                slice_sum();
                if (it.whole()) {
                    sum[w][0][lane] += sx, sum[w][1][lane] += sy, sum[w][2][lane] += sz;
                } else if (grp == 0) {  // sl is already the next slice
                    float *o = part + static_cast<size_t>(it.pslot + sl - 1 - it.sl) * 96;
                    o[t] = sx, o[32 + t] = sy, o[64 + t] = sz;
                }
                sx = sy = sz = kx = ky = kz = 0;
            }
        }
        if (!taken && lane == 0) ci = atomicAdd(queue, 1u);  // no sources
        if (kMulti)
            sx = sum[w][0][lane], sy = sum[w][1][lane], sz = sum[w][2][lane];
        else
            slice_sum();
        if (grp == 0) {
            if (it.whole()) {
                nearv[i] = Gm * sx;
                nearv[n + i] = Gm * sy;
                nearv[2 * static_cast<size_t>(n) + i] = Gm * sz;
            } else if (!kMulti) {
                float *o = part + static_cast<size_t>(it.pslot) * 96;
                o[t] = sx, o[32 + t] = sy, o[64 + t] = sz;
            }
        }
    }
}

// FP64: separations and factors from fixed-point positions (rinv.cuh pair_fixed), in a
// frame per batch of 32 sources about the item's first target. A pair takes them when
// both positions are on the frame's grid, so that its separation is as exact in every
// component as the FP64 difference, which the others take: a source off the grid alone,
// and the whole batch where a target is off it (together a quarter of the pairs of
// 131,071 Plummer particles, about the coordinate planes; none inside a unit cube). Bound by the issue of
// integer instructions (about 220 a pair) and the FP64 pipe (3 operations a pair, 6 off
// the grid, of 64 cycles each). Per launch, with FP64 separations throughout and as
// built: 131,071 Plummer 13.2 and 10.5 ms, 262,144 unit cube 5.1 and 4.4 ms; and the
// FP64 pipe it leaves takes the M2L beside it: RK4 step of the cube 28.3 and 21.1 ms.
// 64 registers, 12 bytes spilled: builds of 72 to 96 are 1 to 8% faster alone, but leave
// the M2L fewer registers beside four blocks (cube 24.6 to 25.9 ms). z's separation on
// the FP64 pipe, as the direct sum has it: 4% faster alone, cube 22.4 ms.
__global__ void __launch_bounds__(kP2PWarps * 32, 8) k_p2p_f64(const int4 *__restrict__ chunks, const unsigned *counts,
                                                            unsigned *queue, const LeafRec *__restrict__ recs,
                                                            const uint2 *__restrict__ ranges, const double *__restrict__ xs,
                                                            double *__restrict__ part, double Gm, double eps2, SoftInt soft,
                                                            double *__restrict__ nearv, unsigned n) {
    __shared__ double src[kP2PWarps][3][32];
    __shared__ uint64_t fix[kP2PWarps][3][32];
    __shared__ double red[kP2PWarps][3][32], sum[kP2PWarps][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned nch = counts[5];
    while (true) {
        unsigned ci = 0;
        if (lane == 0) ci = atomicAdd(queue, 1u);
        ci = __shfl_sync(0xffffffffu, ci, 0);
        if (ci >= nch) break;
        Item it(chunks[ci]);
        const uint4 rec = reinterpret_cast<const uint4 *>(recs + it.li)[0];  // rng_off, rng_len, src_total, spi
        const unsigned slice = recs[it.li].slice;
        it.of_leaf(static_cast<int>(rec.w));
        const int nt = it.nt;
        const int g = 32 / nt;
        const int grp = lane / nt;
        const int t = lane - grp * nt;
        const bool tact = grp < g;
        const int i = it.t0 + t;
        const double *ys = xs + n, *zs = ys + n;
        // frames: extents of the item's targets and of a batch's sources about the first target
        // (positions of targets are read again where they are needed: registers for them cost more)
        const int r0 = it.t0;
        const unsigned ttop = tact ? top_word(xs[i] - xs[r0], ys[i] - ys[r0], zs[i] - zs[r0]) : 0u;
        int qf = INT_MIN;
        bool tgrid = false;  // every target of the item is on the grid of qf
        uint64_t gx = 0, gy = 0, gz = 0;
        sum[w][0][lane] = 0, sum[w][1][lane] = 0, sum[w][2][lane] = 0;  // the finished slices' sums
        for (int sl = it.sl; sl < it.se; ++sl) {
            unsigned v0, len;
            v0 = min(rec.z, static_cast<unsigned>(sl) * slice), len = min(slice, rec.z - v0);
            double ax = 0, ay = 0, az = 0;
            BatchCursor cur;
            cur.start(ranges + rec.x, rec.y, v0, len, static_cast<unsigned>(lane));
            unsigned j;
            for (unsigned cnt; (cnt = cur.next(static_cast<unsigned>(lane), j)) != 0;) {
                double px = 0, py = 0, pz = 0;
                unsigned top = ttop;
                if (static_cast<unsigned>(lane) < cnt) {
                    px = xs[j], py = ys[j], pz = zs[j];
                    src[w][0][lane] = px, src[w][1][lane] = py, src[w][2][lane] = pz;
                    top = max(top, top_word(px - xs[r0], py - ys[r0], pz - zs[r0]));
                }
                const Frame fr = make_frame(static_cast<int>(__reduce_max_sync(0xffffffffu, top) >> 20), soft);
                unsigned grid = 0;  // sources whose separations the frame holds exactly
                if (fr.ok) {
                    fix[w][0][lane] = fixed_point(px, fr.qf), fix[w][1][lane] = fixed_point(py, fr.qf), fix[w][2][lane] = fixed_point(pz, fr.qf);
                    if (fr.qf != qf) {
                        qf = fr.qf;
                        if (tact) gx = fixed_point(xs[i], qf), gy = fixed_point(ys[i], qf), gz = fixed_point(zs[i], qf);
                        tgrid = __all_sync(0xffffffffu, !tact || (on_grid(xs[i], qf) && on_grid(ys[i], qf) && on_grid(zs[i], qf)));
                    }
                    grid = __ballot_sync(0xffffffffu, tgrid && on_grid(px, qf) && on_grid(py, qf) && on_grid(pz, qf));
                }
                __syncwarp();
                if (tact)
#pragma unroll 2
                    for (unsigned k = grp; k < cnt; k += g) {
                        double f, dx, dy, dz;
                        if (!(grid >> k & 1u) || !pair_fixed(separation(fix[w][0][k], gx), separation(fix[w][1][k], gy),
                                                             separation(fix[w][2][k], gz), soft, fr, f, dx, dy, dz)) {
                            dx = src[w][0][k] - xs[i], dy = src[w][1][k] - ys[i], dz = src[w][2][k] - zs[i];
                            if (all_zero(dx, dy, dz)) continue;  // the target itself, or one at its place
                            if (!rinv3(dx, dy, dz, soft, f)) {
                                const double r2 = dx * dx + dy * dy + dz * dz + eps2, ri = r2 > 0.0 ? rsqrt(r2) : 0.0;
                                f = ri * ri * ri;
                            }
                        }
                        ax += f * dx;
                        ay += f * dy;
                        az += f * dz;
                    }
                __syncwarp();
            }
            if (g > 1) {
                red[w][0][lane] = ax, red[w][1][lane] = ay, red[w][2][lane] = az;
                __syncwarp();
                if (grp == 0)
                    for (int q = 1; q < g; ++q) ax += red[w][0][t + q * nt], ay += red[w][1][t + q * nt], az += red[w][2][t + q * nt];
                __syncwarp();
            }
            if (it.whole()) {
                sum[w][0][lane] += ax, sum[w][1][lane] += ay, sum[w][2][lane] += az;
            } else if (grp == 0) {
                double *o = part + static_cast<size_t>(it.pslot + sl - it.sl) * 96;
                o[t] = ax, o[32 + t] = ay, o[64 + t] = az;
            }
        }
        if (grp == 0 && it.whole()) {
            nearv[i] = Gm * sum[w][0][lane];
            nearv[n + i] = Gm * sum[w][1][lane];
            nearv[2 * static_cast<size_t>(n) + i] = Gm * sum[w][2][lane];
        }
    }
}

// Sum the slices of every split chunk in slice order (deterministic).
template <typename T>
__global__ void k_p2p_combine(const int4 *__restrict__ chunks, const unsigned *counts, const LeafRec *__restrict__ recs,
                              const T *__restrict__ part, T scale, T *__restrict__ nearv, unsigned n) {
    const unsigned nit = counts[5];
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < nit * 32u; q += gridDim.x * blockDim.x) {
        const int4 w = chunks[q >> 5];
        const int t = static_cast<int>(q & 31u);
        const int ns = item_nslices(w.z);
        if (item_slice(w.z) != 0 || t >= item_nt(w.z) || ns <= recs[w.x].spi) continue;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            T s = 0;
            for (int k = 0; k < ns; ++k) s += part[static_cast<size_t>(w.w + k) * 96 + 32 * a + t];
            nearv[static_cast<size_t>(a) * n + w.y + t] = scale * s;
        }
    }
}

// Near-field potential (diagnostic, FP64, after an evaluation): for every
// target i of a work item, sum over its near-field sources j != i (tree
// indices) of (|x_j - x_i|^2 + eps^2)^(-1/2). Split items leave per-slice
// partial sums in part[slot][0..31]; k_p2p_phi_combine adds them in slice order.
__global__ void __launch_bounds__(kP2PWarps * 32) k_p2p_phi(const int4 *__restrict__ chunks, const unsigned *counts,
                                                            unsigned *queue, const LeafRec *__restrict__ recs,
                                                            const uint2 *__restrict__ ranges, const double *__restrict__ xs,
                                                            double *__restrict__ part, double Gm, double eps2, SoftInt soft,
                                                            double *__restrict__ phiv, unsigned n) {
    __shared__ double src[kP2PWarps][3][32];
    __shared__ double red[kP2PWarps][32];
    __shared__ unsigned sidx[kP2PWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned nch = counts[5];
    while (true) {
        unsigned ci = 0;
        if (lane == 0) ci = atomicAdd(queue, 1u);
        ci = __shfl_sync(0xffffffffu, ci, 0);
        if (ci >= nch) break;
        Item it(chunks[ci]);
        const uint4 rec = reinterpret_cast<const uint4 *>(recs + it.li)[0];  // rng_off, rng_len, src_total, spi
        const unsigned slice = recs[it.li].slice;
        it.of_leaf(static_cast<int>(rec.w));
        const int nt = it.nt;
        const int g = 32 / nt;
        const int grp = lane / nt;
        const int t = lane - grp * nt;
        const bool tact = grp < g;
        const unsigned i = static_cast<unsigned>(it.t0 + t);
        const double tx = tact ? xs[i] : 0.0, ty = tact ? xs[n + i] : 0.0, tz = tact ? xs[2 * static_cast<size_t>(n) + i] : 0.0;
        double opot = 0;  // the finished slices' sums
        for (int sl = it.sl; sl < it.se; ++sl) {
            unsigned v0, len;
            v0 = min(rec.z, static_cast<unsigned>(sl) * slice), len = min(slice, rec.z - v0);
            double pot = 0;
            BatchCursor cur;
            cur.start(ranges + rec.x, rec.y, v0, len, static_cast<unsigned>(lane));
            unsigned j;
            for (unsigned cnt; (cnt = cur.next(static_cast<unsigned>(lane), j)) != 0;) {
                if (static_cast<unsigned>(lane) < cnt) {
                    src[w][0][lane] = xs[j];
                    src[w][1][lane] = xs[n + j];
                    src[w][2][lane] = xs[2 * static_cast<size_t>(n) + j];
                    sidx[w][lane] = j;
                }
                __syncwarp();
                if (tact)
                    for (unsigned k = grp; k < cnt; k += g) {
                        if (sidx[w][k] == i) continue;
                        const double dx = src[w][0][k] - tx, dy = src[w][1][k] - ty, dz = src[w][2][k] - tz;
                        double f;
                        if (!rinv1(dx, dy, dz, soft, f)) f = 1.0 / sqrt(dx * dx + dy * dy + dz * dz + eps2);
                        pot += f;
                    }
                __syncwarp();
            }
            if (g > 1) {
                red[w][lane] = pot;
                __syncwarp();
                if (grp == 0)
                    for (int q = 1; q < g; ++q) pot += red[w][t + q * nt];
                __syncwarp();
            }
            if (it.whole())
                opot += pot;
            else if (grp == 0)
                part[static_cast<size_t>(it.pslot + sl - it.sl) * 96 + t] = pot;
        }
        if (grp == 0 && it.whole()) phiv[i] = Gm * opot;
    }
}

// Forest: the near field (or potential) of each particle position times its
// system's G m (the P2P kernels ran with G m = 1; one rounding either way).
template <typename T>
__global__ void k_scale_by_system(T *__restrict__ v, unsigned n, int comps, const int *__restrict__ psys,
                                  const TreeInfo *__restrict__ info) {
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const T g = static_cast<T>(info[psys[j]].gm);
        for (int a = 0; a < comps; ++a) v[static_cast<size_t>(a) * n + j] = g * v[static_cast<size_t>(a) * n + j];
    }
}

__global__ void k_p2p_phi_combine(const int4 *__restrict__ chunks, const unsigned *counts,
                                  const LeafRec *__restrict__ recs, const double *__restrict__ part, double Gm, double *__restrict__ phiv) {
    const unsigned nit = counts[5];
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < nit * 32u; q += gridDim.x * blockDim.x) {
        const int4 w = chunks[q >> 5];
        const int t = static_cast<int>(q & 31u);
        const int ns = item_nslices(w.z);
        if (item_slice(w.z) != 0 || t >= item_nt(w.z) || ns <= recs[w.x].spi) continue;
        double s = 0;
        for (int k = 0; k < ns; ++k) s += part[static_cast<size_t>(w.w + k) * 96 + t];
        phiv[w.y + t] = Gm * s;
    }
}

}  // namespace

void near_potential(Workspace &ws, double *phiv) {
    cudaMemsetAsync(ws.queue, 0, sizeof(unsigned), ws.st);
    const unsigned gs = static_cast<unsigned>(ws.num_sms) * 8;
    const double Gm = ws.forest() ? 1.0 : ws.G * ws.m;
    k_p2p_phi<<<gs, kP2PWarps * 32, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.queue, ws.leaf_rec, ws.ranges, ws.xs,
                                                static_cast<double *>(ws.part), Gm, ws.eps * ws.eps,
                                                soft_int(ws.eps * ws.eps), phiv, ws.n);
    k_p2p_phi_combine<<<gs, 256, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.leaf_rec, static_cast<const double *>(ws.part), Gm, phiv);
    ws.launches += 2;
    if (ws.forest()) {
        k_scale_by_system<double><<<gs, 256, 0, ws.st>>>(phiv, ws.n, 1, ws.psys, ws.info);
        ws.launches += 1;
    }
}

// Near-field kernel over the work queue, `per_sm` blocks per SM. The queue
// counter is zeroed at the start of every evaluation (build_tree); several
// launches (on any streams) may drain the same queue, each item is taken once.
// p2p_finish adds the slices of split items after all of them.

void p2p_pass(Workspace &ws, unsigned per_sm) {
    if (per_sm == 0) return;
    timer_begin(ws, kTP2P);
    const unsigned gs = capped_grid(static_cast<unsigned>(ws.num_sms) * per_sm, ceil_div(ws.ch_cap, kP2PWarps));
    const bool soft = ws.eps > 0;
    if (ws.mixed) {
        const float eps2 = static_cast<float>(ws.eps * ws.eps);
        const float Gm = ws.forest() ? 1.0f : static_cast<float>(ws.G * ws.m);  // a forest scales in p2p_finish
        auto *o = static_cast<float *>(ws.nearf);
        auto *pf = static_cast<float *>(ws.part);
#define GB_P2P32_(NW, SF, MU)                                                                                           \
    full_shared(k_p2p_f32<NW, SF, MU>);                                                                                  \
    k_p2p_f32<NW, SF, MU><<<gs, kP2PWarps * 32, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.queue, ws.leaf_rec, ws.ranges, ws.ph, \
                                                        ws.pl, pf, Gm, eps2, o, ws.n)
#define GB_P2P32(NW, SF)             \
    if (forest) {                    \
        GB_P2P32_(NW, SF, true);     \
    } else {                         \
        GB_P2P32_(NW, SF, false);    \
    }
        const bool forest = ws.forest();
        if (ws.p2p_newton && soft) {
            GB_P2P32(true, true);
        } else if (ws.p2p_newton) {
            GB_P2P32(true, false);
        } else if (soft) {
            GB_P2P32(false, true);
        } else {
            GB_P2P32(false, false);
        }
#undef GB_P2P32
#undef GB_P2P32_
    } else {
        const double Gm = ws.forest() ? 1.0 : ws.G * ws.m, eps2 = ws.eps * ws.eps;
        auto *o = static_cast<double *>(ws.nearf);
        auto *pd = static_cast<double *>(ws.part);
        const SoftInt si = soft_int(eps2);
        full_shared(k_p2p_f64);
        k_p2p_f64<<<gs, kP2PWarps * 32, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.queue, ws.leaf_rec, ws.ranges, ws.xs, pd, Gm, eps2,
                                                    si, o, ws.n);
    }
    ws.launches += 1;
    timer_end(ws, kTP2P);
}

void p2p_finish(Workspace &ws) {
    const unsigned gs = capped_grid(static_cast<unsigned>(ws.num_sms) * 8, ceil_div(ws.ch_cap, 8));
    const bool forest = ws.forest();
    const double Gm = forest ? 1.0 : ws.G * ws.m;
    if (ws.mixed)
        k_p2p_combine<float><<<gs, 256, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.leaf_rec, static_cast<const float *>(ws.part),
                                                    static_cast<float>(Gm), static_cast<float *>(ws.nearf), ws.n);
    else
        k_p2p_combine<double><<<gs, 256, 0, ws.st>>>(ws.chunks, ws.d_counts, ws.leaf_rec, static_cast<const double *>(ws.part), Gm,
                                                     static_cast<double *>(ws.nearf), ws.n);
    ws.launches += 1;
    if (forest) {
        if (ws.mixed)
            k_scale_by_system<float><<<gs, 256, 0, ws.st>>>(static_cast<float *>(ws.nearf), ws.n, 3, ws.psys, ws.info);
        else
            k_scale_by_system<double><<<gs, 256, 0, ws.st>>>(static_cast<double *>(ws.nearf), ws.n, 3, ws.psys, ws.info);
        ws.launches += 1;
    }
}

void direct_sum(Workspace &ws, const double *x_orig, const long long *targets, unsigned nt, double *out_soa,
                double *part, unsigned nsplit) {
    const dim3 grid((nt + kDirectTB - 1) / kDirectTB, nsplit);
    k_direct_part<SoA><<<grid, kDirectTB, 0, ws.st>>>(SoA{x_orig, ws.n}, ws.n, targets, nt, nsplit, ws.G * ws.m,
                                                     ws.eps * ws.eps, soft_int(ws.eps * ws.eps), part);
    k_direct_reduce<<<(nt + 255) / 256, 256, 0, ws.st>>>(part, nt, nsplit, out_soa, nullptr);
    ws.launches += 2;
}

}  // namespace gb

// M2L in FP64 (gravity/include/fmm.hpp:277-304), restated on scaled real-basis
// expansions, with the interaction list's mirror symmetry used to cut the FP64
// operations.
//
// GB300's FP64 pipe (2 lanes per clock and SM) bounds this stage: a dense K x K
// operator per source is 189 K^2 multiply-adds per target. The real basis is
// even or odd in x, y and z: with pi(r) the three parity bits of coefficient r,
// the operator of a mirrored offset is T_s[j,k] = (-1)^|s & (pi(j) ^ pi(k))| T[j,k]
// (s: the mirrored axes). The sources of a target whose offsets differ in signs
// only therefore share one K x K product: with the signed sums
//     H_r[k] = sum_s (-1)^|s & r| M_s[k]      (a Walsh-Hadamard transform)
// L[j] += sum_k T[j,k] H_{pi(j) ^ pi(k)}[k]. The 189 offsets are 56 classes of
// (|x|, |y|, |z|), and where a component is 0, T[j,k] vanishes unless j and k
// agree in that parity: 39.5 K^2 multiply-adds and 378 K additions per target
// instead of 189 K^2 (4.3x fewer operations at p = 8, 3.5x at p = 4).
//
// A block takes 32 targets of one octant (a lane each; their slots map to the
// same offsets) and keeps the H of a run of input parities in shared memory; a
// warp owns K / 8 outputs. An FP64 operation holds the pipe 64 cycles per warp,
// so one broadcast operator load and one shared load per multiply-add are free
// and no register tiling is needed.
//
// Small trees leave SMs idle with one block per 32 targets and octant, so
// up to m2l_split_tiles of them the 28 class groups of a tile run as blocks of their
// own and the last one to finish adds the groups. Every form adds the groups in
// the same order, so the results do not depend on it (a forest's systems keep
// the bits of their own contexts).
//
// Measured, ms per evaluation, a dense operator per source on tiles of 64 targets
// -> this kernel: 217 cells, p = 4 2.04 -> 0.064; 745 cells, p = 4 3.57 -> 0.125;
// 2,817 cells, p = 8 24.7 -> 2.38; 4,681 cells (unit cube), p = 6 10.3 -> 1.59.
// Bound by the FP64 pipe (the operations above take 1.3 ms in the third case; the pipe
// is 87% active). 120 registers at p = 8; p = 10 spills 100 bytes at its 128.
#include "workspace.cuh"

namespace gb {

namespace {

constexpr int kThreadsF64 = 256, kWarpsF64 = 8, kLanesF64 = 32;
constexpr int kGroupsF64 = 28, kClassesF64 = 56;  // two classes per group
constexpr int kHRows = 192;                       // H rows of 32 doubles in shared memory (48 KB)

// (|x|, |y|, |z|) classes as 2-bit fields, those without zeros first: dealt out
// in turn, group g takes entries g and g + 28 (one dense class, one with zeros).
struct ClassTab {
    unsigned char c[kClassesF64];
};
constexpr ClassTab class_table() {
    ClassTab t{};
    int n = 0;
    for (int zeros = 0; zeros <= 2; ++zeros)
        for (int q = 0; q < 64; ++q) {
            const int a = q & 3, b = (q >> 2) & 3, c = q >> 4;
            if (a < 2 && b < 2 && c < 2) continue;
            if ((a == 0) + (b == 0) + (c == 0) == zeros) t.c[n++] = static_cast<unsigned char>(q);
        }
    return t;
}
__constant__ ClassTab c_class = class_table();

template <int NB>
__device__ __forceinline__ void gather_transform(const int (*src)[kLanesF64], const unsigned char *kord, int kb, int nk,
                                                 int K, const double *__restrict__ M, double *H, int warp, int lane) {
    constexpr int V = 1 << NB;
    size_t row[V];
    bool on[V];
#pragma unroll
    for (int s = 0; s < V; ++s) {
        const int c = src[s][lane];
        on[s] = c >= 0;
        row[s] = static_cast<size_t>(on[s] ? c : 0) * K;
    }
    for (int i = warp; i < nk; i += kWarpsF64) {
        const int k = kord[kb + i];
        double v[V];
#pragma unroll
        for (int s = 0; s < V; ++s) v[s] = on[s] ? M[row[s] + k] : 0.0;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int s = 0; s < V; ++s)
                if (!(s & (1 << b))) {
                    const double u = v[s], w = v[s | (1 << b)];
                    v[s] = u + w, v[s | (1 << b)] = u - w;
                }
#pragma unroll
        for (int s = 0; s < V; ++s) H[(s * nk + i) * kLanesF64 + lane] = v[s];
    }
}

template <int P>
__global__ void __launch_bounds__(kThreadsF64, 2)
    k_m2l_f64(const TreeInfo *__restrict__ info, const int *__restrict__ m2l_src, const double *__restrict__ ops_all,
              const int4 *__restrict__ otile, const int *__restrict__ oct_list, const double *__restrict__ M,
              double *__restrict__ Lx, double *__restrict__ part, unsigned *pcnt, int split_tiles) {
    constexpr int K = (P + 1) * (P + 1);
    constexpr int NJ = (K + kWarpsF64 - 1) / kWarpsF64;
    extern __shared__ __align__(16) unsigned char smraw[];
    double *H = reinterpret_cast<double *>(smraw);  // [parity combination][input][target]
    __shared__ int src[8][kLanesF64], trow[kLanesF64];
    __shared__ unsigned char kord[K], kpar[K], kbeg[9];  // coefficients sorted by parity
    __shared__ int last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int base = info->level_start[2];
    const int ntgt = info->n_targets_m2l;
    if (ntgt <= 0) return;
    auto par = [](int r) {
        int n, m, im;
        rdecode(r, n, m, im);
        return ((m + im) & 1) | (im << 1) | (((n + m) & 1) << 2);
    };
    if (tid < K) {
        const int mine = par(tid);
        int at = 0;
        for (int r = 0; r < K; ++r) {
            const int q = par(r);
            at += q < mine || (q == mine && r < tid);
        }
        kord[at] = static_cast<unsigned char>(tid), kpar[at] = static_cast<unsigned char>(mine);
    }
    if (tid < 9) {
        int b = 0;
        for (int r = 0; r < K; ++r) b += par(r) < tid;
        kbeg[tid] = static_cast<unsigned char>(b);
    }
    const int per_class = ntgt / 8;
    const int tiles = 8 * (otile ? info->n_otiles : (per_class + kLanesF64 - 1) / kLanesF64);
    const bool split = tiles <= split_tiles;
    const int units = split ? kGroupsF64 * tiles : tiles;
    for (int w = blockIdx.x; w < units; w += gridDim.x) {
        const int tile = w % tiles, cls = tile & 7;
        const int g0 = split ? w / tiles : 0, g1 = split ? g0 + 1 : kGroupsF64;
        const double *ops = ops_all;
        __syncthreads();  // the previous unit is done with trow and src
        if (tid < kLanesF64) {
            if (otile) {
                const int4 ot = otile[tile >> 3];
                trow[tid] = tid < ot.z ? base + cls + 8 * oct_list[ot.y + tid] : -1;
            } else {
                const int t = (tile >> 3) * kLanesF64 + tid;
                trow[tid] = t < per_class ? base + cls + 8 * t : -1;
            }
        }
        if (otile) ops = ops_all + static_cast<size_t>(otile[tile >> 3].x) * kNumOps * K * K;
        const int u[3] = {1 - (cls & 1), 1 - ((cls >> 1) & 1), 1 - ((cls >> 2) & 1)};
        double tot[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) tot[j] = 0;
        for (int g = g0; g < g1; ++g) {
            double acc[NJ];
#pragma unroll
            for (int j = 0; j < NJ; ++j) acc[j] = 0;
            for (int q = g; q < kClassesF64; q += kGroupsF64) {
                const int code = c_class.c[q];
                // offset of the class: 0, +-1 and +-2 with both signs, 3 towards the target's outer side only
                int off[3], bit[3], nb = 0, zmask = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int v = (code >> (2 * a)) & 3;
                    bit[a] = -1, off[a] = v;
                    if (v == 0) zmask |= 1 << a;
                    if (v == 3) off[a] = u[a] ? -3 : 3;
                    if (v == 1 || v == 2) bit[a] = nb++;
                }
                const int V = 1 << nb;
                __syncthreads();  // trow is set; the previous class is done with src and H
                int any = 0;
                if (warp < V) {
                    int dd = 0, o = 0;
                    constexpr int st[3] = {1, 3, 9};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const int x = u[a] + (bit[a] >= 0 && (warp >> bit[a] & 1) ? -off[a] : off[a]);  // child coordinate
                        dd += ((x + 4) / 2 - 1) * st[a];  // floor(x / 2) + 1
                        o |= (1 - (x & 1)) << a;
                    }
                    const int c = trow[lane] >= 0 ? m2l_src[static_cast<size_t>(trow[lane]) * kM2LSlots + 8 * dd + o] : -1;
                    src[warp][lane] = c;
                    any = c >= 0;
                }
                if (!__syncthreads_or(any)) continue;
                const double *op = ops + static_cast<size_t>((off[0] + 3) + 7 * (off[1] + 3) + 49 * (off[2] + 3)) * K * K;
                for (int c0 = 0; c0 < 8;) {
                    int c1 = c0 + 1;
                    while (c1 < 8 && (kbeg[c1 + 1] - kbeg[c0]) * V <= kHRows) ++c1;
                    const int kb = kbeg[c0], nk = kbeg[c1] - kb;
                    if (c0 > 0) __syncthreads();  // H is free
                    switch (nb) {
                        case 0: gather_transform<0>(src, kord, kb, nk, K, M, H, warp, lane); break;
                        case 1: gather_transform<1>(src, kord, kb, nk, K, M, H, warp, lane); break;
                        case 2: gather_transform<2>(src, kord, kb, nk, K, M, H, warp, lane); break;
                        default: gather_transform<3>(src, kord, kb, nk, K, M, H, warp, lane); break;
                    }
                    __syncthreads();
                    for (int pc = c0; pc < c1; ++pc) {
                        const int b = kbeg[pc], e = kbeg[pc + 1];
                        int hp[NJ], tp[NJ];  // offsets of the outputs' H rows (-1: T vanishes) and operator rows
#pragma unroll
                        for (int j = 0; j < NJ; ++j) {
                            const int jp = warp + kWarpsF64 * j;
                            const int d = jp < K ? kpar[jp] ^ pc : 0;
                            int r = 0;
#pragma unroll
                            for (int a = 0; a < 3; ++a)
                                if (bit[a] >= 0) r |= (d >> a & 1) << bit[a];
                            hp[j] = jp < K && !(d & zmask) ? (r * nk + b - kb) * kLanesF64 + lane : -1;
                            tp[j] = (jp < K ? kord[jp] : 0) * K;
                        }
                        for (int i = b; i < e; ++i) {
                            const int k = kord[i];
#pragma unroll
                            for (int j = 0; j < NJ; ++j)
                                if (hp[j] >= 0) acc[j] += __ldg(op + tp[j] + k) * H[hp[j] + (i - b) * kLanesF64];
                        }
                    }
                    c0 = c1;
                }
            }
            if (split) {
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int jp = warp + kWarpsF64 * j;
                    if (jp < K) part[((static_cast<size_t>(tile) * kGroupsF64 + g) * K + jp) * kLanesF64 + lane] = acc[j];
                }
            } else {
#pragma unroll
                for (int j = 0; j < NJ; ++j) tot[j] += acc[j];
            }
        }
        if (split) {
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                last = atomicAdd(pcnt + tile, 1u) == kGroupsF64 - 1;
                if (last) pcnt[tile] = 0;  // ready for the next evaluation
            }
            __syncthreads();
            if (!last) continue;
            __threadfence();
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int jp = warp + kWarpsF64 * j;
                if (jp >= K) continue;
                const double *q = part + (static_cast<size_t>(tile) * kGroupsF64 * K + jp) * kLanesF64 + lane;
#pragma unroll 7
                for (int g = 0; g < kGroupsF64; ++g) tot[j] += __ldcg(q + static_cast<size_t>(g) * K * kLanesF64);
            }
        }
        if (trow[lane] >= 0) {
            double *o = Lx + static_cast<size_t>(trow[lane]) * K;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int jp = warp + kWarpsF64 * j;
                if (jp < K) o[kord[jp]] = tot[j];
            }
        }
    }
}

template <int P>
void launch_m2l_f64(Workspace &ws) {
    constexpr size_t smem = static_cast<size_t>(kHRows) * kLanesF64 * sizeof(double);
    cudaFuncSetAttribute(k_m2l_f64<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    full_shared(k_m2l_f64<P>);
    const unsigned gs = capped_grid(static_cast<unsigned>(ws.num_sms) * 2, static_cast<size_t>(m2l_f64_tiles(ws)) * kGroupsF64);
    k_m2l_f64<P><<<gs, kThreadsF64, smem, ws.st>>>(ws.info, ws.m2l_src, ws.ops_d, ws.forest() ? ws.otile : nullptr, ws.oct_list,
                                                   static_cast<const double *>(ws.Mexp), static_cast<double *>(ws.Lexp),
                                                   ws.f64_sums.part, ws.f64_sums.cnt, static_cast<int>(ws.f64_sums.tiles));
    ws.launches += 1;
}

}  // namespace

unsigned m2l_f64_tiles(const Workspace &ws) {
    return 8 * static_cast<unsigned>(ceil_div(ceil_div(ws.c_cap, 8), kLanesF64) + (ws.forest() ? ws.nsys : 0));
}
size_t m2l_f64_part_doubles(int p) { return static_cast<size_t>(kGroupsF64) * (p + 1) * (p + 1) * kLanesF64; }

void m2l_pass_f64(Workspace &ws) {
    switch (ws.p) {
#define GB_CASE(PP)              \
    case PP:                     \
        launch_m2l_f64<PP>(ws);  \
        break;
        GB_CASE(1)
        GB_CASE(2)
        GB_CASE(3)
        GB_CASE(4)
        GB_CASE(5)
        GB_CASE(6)
        GB_CASE(7)
        GB_CASE(8)
        GB_CASE(9)
        GB_CASE(10)
#undef GB_CASE
        default:
            break;
    }
}

}  // namespace gb

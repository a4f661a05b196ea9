// (d^2 + eps^2)^(-3/2) and (d^2 + eps^2)^(-1/2) of an FP64 separation, to
// FP64 accuracy, on the integer pipe.
//
// GB300's FP64 pipe takes 2 lanes per clock and SM, so an FP64 operation holds
// it for 64 cycles per warp and scheduler, while integer and FP32 operations
// take 1-2. The sum of squares, the reciprocal root and its cube cost 12 of the
// 18 FP64 operations of a softened pair; here they run on integers beside the
// FP64 pipe, and a pair keeps 6 FP64 operations: the separation and the
// accumulation; with the separation from fixed-point positions (Frame), 3 between
// positions on its grid.
//
// Arithmetic (fixed point, u = d^2 + eps^2):
//   a_c   |d_c| as a 62-bit integer on a common exponent e (the largest of the
//         components' and eps'): |d_c| = a_c 2^(e-61), a_c truncated below 2^-61
//   U     sum a_c^2 + eps^2 in units of 2^(2e-58): 58 to 62 bits, error < 4 units
//   y     MUFU rsqrt of U's top 32 bits with one FP32 Newton step (~2^-24), held
//         as the integer Y = y 2^44
//   delta 1 - u y^2 from the 128-bit product U Y^2, |delta| < 2^-22, to 2^-54
//   u^-1/2 = y (1 + delta/2 + 3/8 delta^2), u^-3/2 = y^3 (1 + 3/2 delta + 15/8 delta^2)
// and the result is rounded to 53 bits: relative error 0.8e-16 rms, below 2^-51
// (4.4e-16) at most, over random separations, where the FP64 form (sum of
// squares rounded three times, rsqrt, two products) has 2.4e-16 rms, 9e-16 max.
// Exponents outside [-300, 300] (overflow, underflow, zero separation without
// softening, infinities and NaN) are left to the FP64 form.
//
// Measured, FP64 operations per pair 18 (36 with 1/sqrt) -> 6 (4) -> 3 or 4 with
// Frame: direct sum of 4,096 targets over 262,144 sources 35.2 -> 11.7 -> 9.0 ms; near
// field of 131,071 Plummer particles (1.07e9 pairs) 39.6 -> 12.7 -> 10.5 ms, its
// potential 63 -> 8 ms; unit cube of 262,144 (4.0e8 pairs) 14.0 -> 5.0 -> 4.4 ms.
#pragma once

#include <cstdint>
#include <cstring>

#include "common.cuh"

#ifndef __CUDACC__
#include <cmath>
#endif

namespace gb {

// eps^2 for the integer form: mantissa of eps^2 in units of 2^(2 e_eps - 58) and
// the exponent field of eps.
struct SoftInt {
    uint64_t e2;   // eps^2 2^(58 - 2 e): in [2^58, 2^60), 0 without softening
    int ef;        // exponent field of eps << 20 (0 without softening)
};

namespace rinv {

GB_HD uint32_t hi_word(double x) {
#ifdef __CUDA_ARCH__
    return static_cast<uint32_t>(__double2hiint(x));
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return static_cast<uint32_t>(b >> 32);
#endif
}
GB_HD uint32_t lo_word(double x) {
#ifdef __CUDA_ARCH__
    return static_cast<uint32_t>(__double2loint(x));
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return static_cast<uint32_t>(b);
#endif
}
GB_HD double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(b));
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
GB_HD uint64_t wide(uint32_t a, uint32_t b) { return static_cast<uint64_t>(a) * b; }
GB_HD uint64_t shr(uint64_t v, uint32_t s) {  // 0 from 64 on
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63 ? 0 : v >> s;
#endif
}
GB_HD int clz32(uint32_t v) {
#ifdef __CUDA_ARCH__
    return __clz(static_cast<int>(v));
#else
    return v ? __builtin_clz(v) : 32;
#endif
}
GB_HD float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return static_cast<float>(1.0 / std::sqrt(static_cast<double>(x)));
#endif
}
GB_HD int max_field(int a, int b) { return a > b ? a : b; }

constexpr int kFieldLo = (1023 - 300) << 20, kFieldHi = (1023 + 300) << 20;

// |d| on the common exponent field ef
GB_HD uint64_t mantissa(uint32_t h, uint32_t l, int ef) {
    const uint64_t m = (static_cast<uint64_t>((h & 0xFFFFFu) | 0x100000u) << 32) | l;  // 53 bits
    return shr(m << 9, static_cast<uint32_t>(ef - static_cast<int>(h & 0x7FF00000u)) >> 20);
}

struct Root {
    uint32_t Y;     // y 2^44, in (2^29, 2^31]
    uint64_t Q;     // Y^2
    int delta;      // (1 - u y^2) 2^53
    int ef;         // common exponent field
};

GB_HD void root_of(uint64_t ax, uint64_t ay, uint64_t az, int ef, const SoftInt &e, Root &r) {
    const uint32_t x1 = static_cast<uint32_t>(ax >> 32), y1 = static_cast<uint32_t>(ay >> 32), z1 = static_cast<uint32_t>(az >> 32);
    const uint64_t s2 = wide(x1, static_cast<uint32_t>(ax)) + wide(y1, static_cast<uint32_t>(ay)) + wide(z1, static_cast<uint32_t>(az));
    const uint64_t U = wide(x1, x1) + wide(y1, y1) + wide(z1, z1) + (s2 >> 31) +
                       shr(e.e2, static_cast<uint32_t>(ef - e.ef) >> 19);
    const float uf = static_cast<float>(static_cast<uint32_t>(U >> 32));
    const float y = rsqrt_seed(uf);
#ifdef __CUDA_ARCH__
    const float q = __fmaf_rn(-__fmul_rn(uf, y), y, 1.0f);
    const uint32_t Y = __float2uint_rn(__fmul_rn(y, 0x1p44f)) + static_cast<uint32_t>(__float2int_rn(__fmul_rn(__fmul_rn(y, 0x1p43f), q)));
    const uint64_t Q = wide(Y, Y);
    const uint64_t prod = __umul64hi(U, Q);
#else
    const float q = fmaf(-(uf * y), y, 1.0f);
    const uint32_t Y = static_cast<uint32_t>(y * 0x1p44f) + static_cast<uint32_t>(static_cast<int>(std::lrint((y * 0x1p43f) * q)));
    const uint64_t Q = wide(Y, Y);
    const uint64_t prod = static_cast<uint64_t>((static_cast<unsigned __int128>(U) * Q) >> 64);
#endif
    r.Y = Y, r.Q = Q, r.ef = ef;
    r.delta = static_cast<int>((static_cast<int64_t>(1ull << 56) - static_cast<int64_t>(prod) + 4) >> 3);
}

GB_HD bool root(double dx, double dy, double dz, const SoftInt &e, Root &r) {
    const uint32_t hx = hi_word(dx), hy = hi_word(dy), hz = hi_word(dz);
    const int ef = max_field(max_field(static_cast<int>(hx & 0x7FF00000u), static_cast<int>(hy & 0x7FF00000u)),
                             max_field(static_cast<int>(hz & 0x7FF00000u), e.ef));
    root_of(mantissa(hx, lo_word(dx), ef), mantissa(hy, lo_word(dy), ef), mantissa(hz, lo_word(dz), ef), ef, e, r);
    return ef >= kFieldLo && ef <= kFieldHi;
}

// 8 delta^2 in units of 2^-53
GB_HD int square8(int delta) { return static_cast<int>((static_cast<int64_t>(delta) * delta) >> 50); }

// m (1 + c 2^-53) 2^ex as a double, m in [2^32, 2^62), |c| < 2^31
GB_HD double pack(uint64_t m, int c, int ex) {
    const int lz = clz32(static_cast<uint32_t>(m >> 32)) - 1;  // top bit to bit 62
    m <<= lz;
    const int64_t corr = static_cast<int64_t>(static_cast<int32_t>(m >> 32)) * c;
    // 2^9: half a unit of the result where the correction does not carry m past a power of
    // two (else up to a whole one); added before the last shift, after which it could pass 2^64
    uint64_t f = m + static_cast<uint64_t>(corr >> 21) + 0x200;
    const int l2 = clz32(static_cast<uint32_t>(f >> 32));  // 0, 1 or 2
    f <<= l2;
    return from_bits((static_cast<uint64_t>(1022 + 63 + ex - lz - l2) << 52) + (f >> 11));
}

}  // namespace rinv

GB_HD SoftInt soft_int(double eps2) {
    SoftInt s{0, 0};
    if (!(eps2 > 0)) return s;
    const int f = static_cast<int>(rinv::hi_word(eps2) >> 20) - 1023;  // floor(log2 eps^2)
    const int e = f >= 0 ? f / 2 : -((1 - f) / 2);                     // floor(f / 2)
    const uint64_t m = (static_cast<uint64_t>((rinv::hi_word(eps2) & 0xFFFFFu) | 0x100000u) << 32) | rinv::lo_word(eps2);
    s.e2 = m << (6 + f - 2 * e);  // m 2^(f-52) = e2 2^(2e-58)
    s.ef = (1023 + e) << 20;
    return s;
}

// false: outside the integer form's exponent range, the caller takes the FP64 form
namespace rinv {
GB_HD double cube(const Root &r) {
    const uint64_t g = wide(static_cast<uint32_t>(r.Q >> 32), r.Y) + (wide(static_cast<uint32_t>(r.Q), r.Y) >> 32);
    const int c = r.delta + (r.delta >> 1) + ((15 * square8(r.delta) + 32) >> 6);
    return pack(g, c, -61 - 3 * ((r.ef >> 20) - 1023));
}
}  // namespace rinv

GB_HD bool rinv3(double dx, double dy, double dz, const SoftInt &e, double &f) {
    rinv::Root r;
    const bool ok = rinv::root(dx, dy, dz, e, r);
    f = rinv::cube(r);
    return ok;
}
GB_HD bool rinv1(double dx, double dy, double dz, const SoftInt &e, double &f) {
    rinv::Root r;
    const bool ok = rinv::root(dx, dy, dz, e, r);
    const int c = (r.delta >> 1) + ((3 * rinv::square8(r.delta) + 32) >> 6);
    f = rinv::pack(static_cast<uint64_t>(r.Y) << 30, c, -61 - ((r.ef >> 20) - 1023));
    return ok;
}

// Separations as differences of fixed-point positions. A frame is a quantum 2^q for
// a set of sources and targets whose separations stay below 2^(q+62): positions
// as multiples of it modulo 2^64 (fixed_point), whose difference is the separation
// whatever the positions' own size. A coordinate with no bits below the quantum (on_grid:
// all but those within 2^-8 of the set's extent of the coordinate planes) is held
// exactly, so that between two of them every component, however small beside the
// others, is rounded once, to 53 bits of its own, as the FP64 difference is (within
// 2^-53 of itself). A coordinate off the grid is held to half a quantum: what that is
// of a component depends on the component, and the kernels say which they take.
// Pairs with no component of 53 bits of quanta are left to the FP64 difference.
struct Frame {
    int ok;    // 0: no such frame (no extent, overflow, infinities, NaN, softening far above the extent)
    int qf;    // exponent field of the quantum
    int nmax;  // largest left shift of a separation that keeps eps below 2^62 quanta
};
// top: exponent field of the largest |component| of position - reference
GB_HD Frame make_frame(int top, const SoftInt &e) {
    const int ee = e.ef >> 20;
    Frame f;
    const int t = rinv::max_field(top, ee - 1);
    f.qf = t - 60;
    f.nmax = e.ef ? 61 - (ee - f.qf) : 62;
    f.ok = top >= 1023 - 280 && t <= 1023 + 280 && t - top <= 2;
    return f;
}
GB_HD uint64_t shl(uint64_t v, uint32_t s) {  // 0 from 64 on
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63 ? 0 : v << s;
#endif
}
GB_HD uint64_t fixed_point(double x, int qf) {  // x / 2^(qf - 1023) to the nearest, modulo 2^64
    const uint32_t h = rinv::hi_word(x);
    const int ex = static_cast<int>((h >> 20) & 0x7FFu);
    const uint64_t m = ex ? (static_cast<uint64_t>((h & 0xFFFFFu) | 0x100000u) << 32) | rinv::lo_word(x) : 0;
    const int s = ex - 52 - qf;  // m 2^s quanta
    const uint64_t a = s >= 0 ? shl(m, static_cast<uint32_t>(s)) : (rinv::shr(m, static_cast<uint32_t>(-s - 1)) + 1) >> 1;
    return (h >> 31) ? 0 - a : a;
}
// Source minus target in quanta. The positions are residues: their difference wraps in
// ordinary runs (a leaf across x = 2^(q+63) has some on either side), so it is taken in
// unsigned arithmetic and only the result, below 2^62 in size, is read with its sign.
GB_HD int64_t separation(uint64_t source, uint64_t target) { return static_cast<int64_t>(source - target); }
// fixed_point(x, qf) is x: the mantissa's last bit is no smaller than the quantum
GB_HD bool on_grid(double x, int qf) {
    const uint32_t h = rinv::hi_word(x);
    return static_cast<int>((h >> 20) & 0x7FFu) >= qf + 52 || ((h << 1) | rinv::lo_word(x)) == 0;
}
// Below 2^54 quanta to a position off the grid (`off`: kOffGrid, or 0 for one on it): half a
// quantum is then more than a quarter of the rounding to 53 bits.
constexpr int kOffGrid = 1 << 22;  // high word of 2^54 quanta
GB_HD bool too_short(int64_t f, int off) {  // in [-off, off) 2^32 quanta
    return static_cast<uint32_t>(static_cast<int>(f >> 32) + off) < 2u * static_cast<uint32_t>(off);
}
namespace rinv {
// a 2^(ef - 1023 - 61), a < 2^62, with the sign of s (0 or -1)
GB_HD double to_double(uint64_t a, uint32_t s, int ef) {
    const uint32_t h = static_cast<uint32_t>(a >> 32), l = static_cast<uint32_t>(a);
    const uint64_t v = h ? a : static_cast<uint64_t>(l) << 31;
    const uint32_t t = static_cast<uint32_t>(v >> 32);
    const int lz = clz32(t) - 1;  // top bit to bit 62: the rounding cannot pass 2^64
    const uint64_t m = v << (lz & 31);
    const int field = (ef >> 20) - lz - (h ? 0 : 31);
    const uint64_t b = (static_cast<uint64_t>(static_cast<uint32_t>(field)) << 52) + ((m + 0x200) >> 10);
    return from_bits(a ? b | (static_cast<uint64_t>(s & 0x80000000u) << 32) : 0);
}
}  // namespace rinv

// Separation (fx, fy, fz quanta of a frame that is ok) as doubles and its factor
// f = (d^2 + eps^2)^(-3/2). false: too close for the frame, the caller takes the
// FP64 difference of the positions.
GB_HD bool pair_fixed(int64_t fx, int64_t fy, int64_t fz, const SoftInt &e, const Frame &fr, double &f, double &dx, double &dy,
                      double &dz) {
    const uint32_t sx = static_cast<uint32_t>(fx >> 63), sy = static_cast<uint32_t>(fy >> 63), sz = static_cast<uint32_t>(fz >> 63);
    const uint64_t ux = static_cast<uint64_t>(fx), uy = static_cast<uint64_t>(fy), uz = static_cast<uint64_t>(fz);
    uint64_t ax = fx < 0 ? 0 - ux : ux, ay = fy < 0 ? 0 - uy : uy, az = fz < 0 ? 0 - uz : uz;
    const uint32_t m = static_cast<uint32_t>(rinv::max_field(static_cast<int>(ax >> 32),
                                                             rinv::max_field(static_cast<int>(ay >> 32), static_cast<int>(az >> 32))));
    const int lead = rinv::clz32(m) - 2;  // 0 to 8 for the separations taken here
    const int n = lead < fr.nmax ? lead : fr.nmax;
    ax <<= n, ay <<= n, az <<= n;
    const int ef = (fr.qf + 61 - n) << 20;
    rinv::Root r;
    rinv::root_of(ax, ay, az, ef, e, r);
    f = rinv::cube(r);
    dx = rinv::to_double(ax, sx, ef), dy = rinv::to_double(ay, sy, ef), dz = rinv::to_double(az, sz, ef);
    return m >= (1u << 21);
}

}  // namespace gb

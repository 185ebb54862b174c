// idg_tc.cuh -- shared pieces of the tensor-core gridder and degridder.
//
// The phase of pixel (x, y) and visibility v is, in turns,
//   phi = a_v hx + b_v hy + g_v n(x, y),  hx = x + 1/2 - S/2, hy likewise,
// with a_v = (X + S/2 - G/2)/S - k u d2pi (b_v likewise) and
// g_v = w_step (Z + 1/2) - k w / 2 pi.  n depends on l^2 + m^2 only and splits as
//   n(l, m) = f(l) + f(m) + c(l, m),  f(l) = n(l, 0),
// where c is tiny (l^2 m^2 / 4 and smaller) and, to a relative 0.6 l^2 m^2, a
// product cx(l) cx(m).  With g_v = g0 + d_v (g0: the middle of the subgrid's
// range of g) the phasor becomes
//   e^{i phi} = e^{i g0 n(x, y)} P_v(x) Q_v(y) (1 + i d_v cx(x) cx(y) + ...),
//   P_v(x) = e^{i (a_v hx + d_v f(x))},  Q_v(y) = e^{i (b_v hy + d_v f(y))}:
// an exact per-pixel factor outside the sum, and a sum over visibilities that
// is a matrix product of the S x-factors with the S y-factors.  That takes the
// work per pixel-visibility from a sincos and 17 FMA to 16 multiply-adds of a
// matrix product, which run on the tensor cores: fp16 pairs hi + lo carry each
// fp32 operand to 2^-22 (three products hi hi, hi lo, lo hi, fp32 accumulators).
// The first-order term i d cx cx is one more product (its size, at most
// kTcEps, leaves its fp16 rounding below 1e-6); it is left out where
// it is below kTcEpsSkip.  Subgrids whose range of g is too wide for the
// expansion, or whose arguments are not finite, are counted in a.fallback and
// done by the general kernel.
#pragma once

#include <cmath>
#include <cuda_fp16.h>

#include "idg_device.cuh"
#include "idg_umma.cuh"

namespace idg {

// Bounds of the expansion, in radians of phase at the subgrid's corner pixel:
// the neglected second-order term is eps^2 / 2 there and 0.05 times that RMS
// over pixels and a uniform range (2e-3: 1e-7); a neglected first-order term is
// 0.12 eps RMS (5e-7: 6e-8).
constexpr float kTcEps = 2e-3f;
constexpr float kTcEpsSkip = 5e-7f;
constexpr float kTcMaxSlope = 0.75f;     // turns of d f(x): the sincos argument stays within 1.25 turns
constexpr float kTcMaxStep = 65536.f;    // turns per pixel before reduction
constexpr double kTcMaxHalfImage = 0.12; // radians: bounds the error of c = cx cx
constexpr uint64_t kTcWaitNs = 2000000000ull;
// Visibilities of one item: the scout waits for as long as the item before takes,
// at most 0.2 s in the gridder and, uncut and in four blocks, 0.6 s in the
// degridder.  Longer subgrids go to the general kernel, whose waits are for a tile.
constexpr int64_t kTcMaxVis = 1 << 23;

// n(r2) = 1 - sqrt(1 - r2) by its series, for r2 <= 2 * 0.12^2 (next term < 1e-13).
inline double tc_n(double r2) {
    const double c[9] = {1.0 / 2,     1.0 / 8,      1.0 / 16,      5.0 / 128,     7.0 / 256,
                         21.0 / 1024, 33.0 / 2048, 429.0 / 32768, 715.0 / 65536};
    double s = c[8];
    for (int i = 7; i >= 0; --i) s = s * r2 + c[i];
    return s * r2;
}

// Constants of one launch, from the host (the GPU's FP64 rate is too low to
// make them in every CTA).
inline TcConst tc_const(int S, double image_size) {
    TcConst t{};
    const auto split = [](double v, float &hi, float &lo) {
        hi = (float)v;
        lo = (float)(v - hi);
    };
    const double step = image_size / S, edge = 0.5 * (S - 1) * step;
    const double e2 = edge * edge, cmm = tc_n(2 * e2) - 2 * tc_n(e2);
    for (int i = 0; i < S / 2; ++i) {
        const double l = (i + 0.5) * step, l2 = l * l;
        t.f[i] = (float)tc_n(l2);
        t.cx[i] = (float)((tc_n(l2 + e2) - tc_n(l2) - tc_n(e2)) / std::sqrt(cmm));
    }
    t.f_max = (float)tc_n(e2);
    t.eps_per_g = (float)(kTwoPi * cmm);
    t.turns_per_step = (float)(step / kTwoPi);
    split(0.25 * step * step, t.s2h, t.s2l);
    split(image_size / (S * kTwoPi), t.d2h, t.d2l);
    split(1.0 / kTwoPi, t.i2h, t.i2l);
    return t;
}
inline bool tc_image_fits(double image_size) { return 0.5 * image_size <= kTcMaxHalfImage; }

// Pixel geometry along one axis, by pairs of pixels 2i, 2i + 1: eight floats
// (hx0, hx1, f0, f1) (cx0, cx1, -, -).
__device__ __forceinline__ void tc_axis_table(const KernelArgs &a, float4 *tab, int npairs, int tid, int nt) {
    const int Sh = a.S / 2;
    for (int i = tid; i < npairs; i += nt) {
        float h[2], f[2], c[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int x = 2 * i + e, k = x < Sh ? Sh - 1 - x : x - Sh;
            h[e] = (float)(2 * x + 1 - a.S) * 0.5f;
            f[e] = k < Sh ? a.tc.f[k] : 0.f;
            c[e] = k < Sh ? a.tc.cx[k] : 0.f;
        }
        tab[2 * i] = make_float4(h[0], h[1], f[0], f[1]);
        tab[2 * i + 1] = make_float4(c[0], c[1], 0.f, 0.f);
    }
}
// n of one quadrant as float pairs hi + lo: tab[y * Sh + x], y, x < Sh = S / 2.
// With r2 = q step^2 / 4 and q a small integer, r2 / 2 and r2^2 / 8 are kept to
// twice the precision; the rest of the series is below 1e-4 of the sum.
__device__ __forceinline__ void tc_n_table(const KernelArgs &a, float2 *tab, int tid, int nt) {
    const int Sh = a.S / 2;
    for (int i = tid; i < Sh * Sh; i += nt) {
        const int y = i / Sh, x = i - y * Sh, hx = 2 * x + 1 - a.S, hy = 2 * y + 1 - a.S;
        const float q = (float)(hx * hx + hy * hy);
        const float r = __fmul_rn(q, a.tc.s2h), re = fmaf(q, a.tc.s2l, fmaf(q, a.tc.s2h, -r));
        const float b = __fmul_rn(r, r), be = fmaf(2.f * r, re, fmaf(r, r, -b));
        const float c = b * r * fmaf(r, fmaf(r, fmaf(r, fmaf(r, 33.f / 2048, 21.f / 1024), 7.f / 256), 5.f / 128), 1.f / 16);
        const float s = __fadd_rn(0.5f * r, 0.125f * b), e = __fsub_rn(0.125f * b, __fsub_rn(s, 0.5f * r));
        const float lo = e + 0.5f * re + 0.125f * be + c, hi = __fadd_rn(s, lo);
        tab[i] = make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s)));
    }
}
// Per channel: k * d2pi and k / 2 pi as float pairs hi + lo.
__device__ __forceinline__ void tc_channel_table(const KernelArgs &a, float4 *tab, int tid, int nt) {
    for (int c = tid; c < a.C; c += nt) {
        const float k = a.wavenumbers[c], p = __fmul_rn(k, a.tc.d2h), q = __fmul_rn(k, a.tc.i2h);
        tab[c] = make_float4(p, fmaf(k, a.tc.d2l, fmaf(k, a.tc.d2h, -p)), q, fmaf(k, a.tc.i2l, fmaf(k, a.tc.i2h, -q)));
    }
}

// What a subgrid's phases need beside its rows.
struct TcSubgrid {
    float xh, xl, yh, yl; // (X + S/2 - G/2)/S modulo 2 turns, hi + lo; Y likewise
    float mid;            // middle of the range of k w / 2 pi
    float g0h, g0l;       // g0 = w_step (Z + 1/2) - mid, hi + lo
    int cross;            // whether the first-order term is needed
};

__device__ __forceinline__ unsigned tc_ord(float v) { // order-preserving map to unsigned
    const unsigned b = __float_as_uint(v);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float tc_unord(unsigned u) {
    return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

// (X + S/2 - G/2)/S modulo 2 as hi + lo: reduced as an integer over 2 S, the
// remainder of the fp32 division recovered exactly.
__device__ __forceinline__ void tc_offset(int X, int S, int G, float &hi, float &lo) {
    const int r = (2 * (X % (2 * S)) + (S - G) % (4 * S)) % (4 * S);
    const float n = (float)r, q = (float)(2 * S);
    hi = __fdiv_rn(n, q);
    lo = fmaf(-hi, q, n) / q;
}

constexpr int kTcScratch = 6;
// Whether the expansion holds for a (valid) subgrid; NT threads (whole warps,
// of consecutive numbers) call it and get the same answer, `sync` being their barrier.
// `scratch`: kTcScratch words of shared memory, not used by a single warp.  Only the
// ranges of u, v, w and of the wavenumbers enter.
template <int NT, typename Sync>
__device__ inline bool tc_fits(const KernelArgs &a, const SubgridInfo &si, unsigned *scratch, TcSubgrid *out,
                               Sync sync) {
    if ((int64_t)si.T * (si.c1 - si.c0) > kTcMaxVis) return false;
    const TcConst &tc = a.tc;
    const int tid = threadIdx.x % NT, nt = NT;
    if constexpr (NT > 32) {
        sync();
        if (tid < kTcScratch) scratch[tid] = 0u;
        sync();
    }
    // max of ord(w), ord(-w), ord(k), ord(-k); |u| |v| |w| and |k| as bits, which a NaN
    // leads (its ord may be anything)
    unsigned m[kTcScratch] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (int t = tid; t < si.T; t += nt) {
        const float *p = a.uvw + 3 * ((int64_t)si.row0 + t);
        const float u = p[0], v = p[1], w = p[2];
        m[0] = max(m[0], tc_ord(w));
        m[1] = max(m[1], tc_ord(-w));
        m[4] = max(m[4], max(__float_as_uint(fabsf(u)), max(__float_as_uint(fabsf(v)), __float_as_uint(fabsf(w)))));
    }
    for (int c = si.c0 + tid; c < si.c1; c += nt) {
        const float k = a.wavenumbers[c];
        m[2] = max(m[2], tc_ord(k));
        m[3] = max(m[3], tc_ord(-k));
        m[5] = max(m[5], __float_as_uint(fabsf(k)));
    }
#pragma unroll
    for (int i = 0; i < kTcScratch; ++i) {
        m[i] = __reduce_max_sync(0xffffffffu, m[i]);
        if (NT > 32 && (tid & 31) == 0 && m[i]) atomicMax(&scratch[i], m[i]);
    }
    if constexpr (NT > 32) {
        sync();
#pragma unroll
        for (int i = 0; i < kTcScratch; ++i) m[i] = scratch[i];
    }
    const float wmax = tc_unord(m[0]), wmin = -tc_unord(m[1]);
    const float kmax = tc_unord(m[2]), kmin = -tc_unord(m[3]);
    const float reach = __uint_as_float(m[4]), kabs = __uint_as_float(m[5]);
    // Every operation that decides is rounded on its own: the tensor-core kernels
    // and the general ones behind them ask this question separately, in kernels
    // compiled separately, and a subgrid on the edge must get one answer.
    const float g[4] = {__fmul_rn(kmin, wmin), __fmul_rn(kmin, wmax), __fmul_rn(kmax, wmin), __fmul_rn(kmax, wmax)};
    const float gmin = __fmul_rn(fminf(fminf(g[0], g[1]), fminf(g[2], g[3])), 1.f / kTwoPiF);
    const float gmax = __fmul_rn(fmaxf(fmaxf(g[0], g[1]), fmaxf(g[2], g[3])), 1.f / kTwoPiF);
    const float half = __fmul_rn(0.5f * __fsub_rn(gmax, gmin), 1.0001f), mid = 0.5f * __fadd_rn(gmax, gmin);
    const float step = __fmul_rn(__fmul_rn(kabs, reach), tc.turns_per_step);
    out->mid = mid;
    const float eps = __fmul_rn(half, tc.eps_per_g);
    out->cross = eps > kTcEpsSkip;
    tc_offset(si.X, a.S, a.G, out->xh, out->xl);
    tc_offset(si.Y, a.S, a.G, out->yh, out->yl);
    // g0 = w_step (Z + 1/2) - mid: exact product (fma), two-sum
    const float z = __fadd_rn((float)si.Z, 0.5f), p = __fmul_rn(a.w_step, z), pe = fmaf(a.w_step, z, -p);
    const float d = __fsub_rn(p, mid), bb = __fsub_rn(d, p);
    out->g0h = d;
    out->g0l = __fadd_rn(__fadd_rn(__fsub_rn(p, __fsub_rn(d, bb)), __fsub_rn(-mid, bb)), pe);
    // written so that a NaN anywhere fails; one in u, v, w or k is in `step`
    return eps <= kTcEps && __fmul_rn(half, tc.f_max) <= kTcMaxSlope && step <= kTcMaxStep &&
           fabsf(out->g0h) <= 1e7f;
}

// An axis slope of one visibility in turns per pixel, off - (kh + kl) u modulo
// 2 turns, as hi + lo: hi is a multiple of 2^-16, so that hi * hx (hx a
// half-integer below 32) is exact in fp32.
__device__ __forceinline__ void tc_slope(float kh, float kl, float u, float offh, float offl, float &hi, float &lo) {
    const float M = 12582912.f; // 1.5 * 2^23
    const float p = __fmul_rn(kh, u);
    const float e = fmaf(kl, u, fmaf(kh, u, -p));
    const float q = __fsub_rn(__fadd_rn(0.5f * p, M), M);
    const float r = fmaf(-2.f, q, p);
    const float d = __fsub_rn(offh, r), bb = __fsub_rn(d, offh); // two-sum of offh and -r
    const float err = __fadd_rn(__fsub_rn(offh, __fsub_rn(d, bb)), __fsub_rn(-r, bb));
    const float R = 192.f; // ulp 2^-16 between 128 and 256
    hi = __fsub_rn(__fadd_rn(d, R), R);
    lo = __fsub_rn(d, hi) + ((err + offl) - e);
}
// d_v = mid - (kh + kl) w, in turns per unit n.
__device__ __forceinline__ float tc_delta(float kh, float kl, float w, float mid) {
    const float p = __fmul_rn(kh, w);
    const float e = fmaf(kl, w, fmaf(kh, w, -p));
    return __fsub_rn(__fsub_rn(mid, p), e);
}

// cos and sin of 2 pi (hi h + lo h + d f) for a pair of pixels; lo and d come
// multiplied by 2 pi.  hi h is exact and so is its reduction to half a turn;
// the radians are then rounded once at their full size.
__device__ __forceinline__ void tc_sincos(f2 hi, f2 lo2pi, f2 d2pi, f2 h, f2 f, f2 &c, f2 &s) {
    const f2 M = 0x4b4000004b400000ull; // 1.5 * 2^23, twice
    const f2 r = ffma2(hi, h, fsub2(M, ffma2(hi, h, M))); // hi h - rint(hi h): every step is exact
    const f2 x = ffma2(r, pack2(kTwoPiF, kTwoPiF), ffma2(lo2pi, h, fmul2(d2pi, f)));
    float x0, x1;
    unpack2(x, x0, x1);
    c = pack2(cos_ftz(x0), cos_ftz(x1));
    s = pack2(sin_ftz(x0), sin_ftz(x1));
}

// fp32 pair -> fp16 pairs hi and lo, v = hi + lo to 2^-22 of v.
__device__ __forceinline__ uint32_t tc_half2(f2 v) {
    float a, b;
    unpack2(v, a, b);
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ void tc_split(f2 v, uint32_t &hi, uint32_t &lo) {
    hi = tc_half2(v);
    const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    lo = tc_half2(fsub2(v, pack2(h.x, h.y)));
}

// Power of two that brings a largest magnitude (as float bits) to [2^12, 2^13),
// and its reciprocal; 1 for zero and for values that are not finite.
__device__ __forceinline__ float tc_scale(unsigned max_bits, float &inv) {
    int e = (int)(max_bits >> 23);
    if (max_bits == 0u || e == 255) {
        inv = 1.f;
        return 1.f;
    }
    e = max(e, 14); // both factors stay normal
    inv = __uint_as_float((unsigned)(e - 12) << 23);
    return __uint_as_float((unsigned)(254 + 12 - e) << 23);
}

// The tensor core truncates its fp32 accumulator towards zero after every
// product.  Over the few full-size products of one sum that shrinks the result
// by 1.6e-7 to 2.1e-7 (measured against 64 bits, whatever the lengths); this
// factor puts the mean of it back.
constexpr float kTcTruncation = 1.f + 2.384185791015625e-7f; // 1 + 2^-22
// The gridder's accumulators take four full-size products per stage.
constexpr float kTcTruncationPerStage = 1.0e-7f;

// Bounded wait; on expiry raises the CTA's abort flag and the status bit, after
// which every wait returns at once: the roles run to their next common check
// on stale data (all addresses stay valid) and the CTA ends.  While the scout
// looks at claims that it has to leave out, nothing else moves: the limit counts
// from its last look.
struct TcWatch {
    uint64_t looked; // when the scout last took a claim up, ns
    int abort;
};
__device__ __forceinline__ void tc_wait(uint64_t *bar, uint32_t phase, volatile TcWatch *watch, unsigned *status) {
    if (mbar_try_wait(bar, phase)) return;
    const uint64_t t0 = global_timer_ns();
    while (!mbar_try_wait(bar, phase)) {
        if (watch->abort) return;
        const uint64_t now = global_timer_ns();
        if (now - t0 > kTcWaitNs && now > watch->looked + kTcWaitNs) {
            watch->abort = 1;
            flag_status(status, kStatusTimeout);
            return;
        }
    }
}
template <int ID, int NT>
__device__ __forceinline__ void named_sync() {
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(NT) : "memory");
}

// e^{2 pi i g0 n}, n = nh + nl.
__device__ __forceinline__ cf tc_pixel_factor(float g0h, float g0l, float2 n) {
    const float p = __fmul_rn(g0h, n.x);
    const float e = fmaf(g0l, n.x, fmaf(g0h, n.y, fmaf(g0h, n.x, -p)));
    float s, c;
    sincospif(2.f * (__fsub_rn(p, rintf(p)) + e), &s, &c);
    return {c, s};
}

} // namespace idg

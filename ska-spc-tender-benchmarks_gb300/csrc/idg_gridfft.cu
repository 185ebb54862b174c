// idg_gridfft.cu -- 2-D FFT of the uv-grid (the imaging step after the adder).
//
// For every plane (w-plane, polarisation) of grid[W][4][G][G], G = 2^k:
//   direction -1 (uv -> image):
//     out[y][x] = c[y] c[x] sum_{v,u} grid[v][u] exp(-2 pi i ((u-G/2)(x-G/2) + (v-G/2)(y-G/2)) / G)
//   direction +1 (image -> uv): the adjoint,
//     out[v][u] = sum_{y,x} c[y] c[x] grid[y][x] exp(+2 pi i ((u-G/2)(x-G/2) + (v-G/2)(y-G/2)) / G)
// with c the optional separable grid correction (length G; 1 when NULL).  The
// centre cell G/2 is the origin of both domains.  For G divisible by 4 the
// shifts factorise into (-1)^(u+v) before and (-1)^(x+y) after an unshifted
// DFT, so each 1-D pass is: multiply by (-1)^index (and c), unshifted FFT,
// multiply by (-1)^index (and c).
//
// FFT(shifted input) and the sign (-1)^k of an output are each a rotation by
// half the length on the other side, so both centre shifts are index changes:
// element i is read from, and written to, position i ^ G/2.
//
// Two passes over the grid: rows, then columns in place.  A CTA transforms a
// strip of 2 H lines at a time (H = 2 at G = 4096: four rows, or four
// neighbouring columns = one 32-byte sector of every row; the sectors of a
// 128-byte line are asked for by neighbouring CTAs at about the same time and
// meet in L2).  A thread holds 16 points of two lines in registers; a radix-16
// Stockham pass is a 4 x 4 butterfly in registers and an exchange through
// shared memory, one line of each pair after the other, so that the exchange
// needs half the strip's size and the next strip can be on its way into the
// rest: rows by one bulk copy, columns by each thread's own 16-byte
// asynchronous copies.  Twiddles e^{-2 pi i m / G} come from a table computed
// in FP64 on the host: of the 15 powers a butterfly needs six are read and
// nine are products of two of them.
// Measured on GB300, four planes of 4096^2: 557 us (rows 210, columns 345), where
// rows, transpose, rows, transpose took 897 (269 + 172 each way).  DRAM traffic is
// the algorithmic 2 x 537 MB per pass, 158 us at the copy rate.  Rows are bound by
// the wavefronts of the exchange and the stores; columns wait for the load-store
// unit, whose instructions touch 16 lines each.  256^2: 28 us (40), 2048^2: 132 (240).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "idg_device.cuh"
#include "idg_host.h"
#include "idg_internal.h"
#include "idg_ptx.cuh"

namespace idg {

namespace {

constexpr uint64_t kWaitNs = 2000000000ull; // a staged strip not complete after 2 s is declared lost

// The complex numbers of a butterfly: additions of (re, im) in one instruction.
__device__ __forceinline__ float2 ca(float2 a, float2 b) {
    float2 r;
    unpack2(fadd2(pack2(a.x, a.y), pack2(b.x, b.y)), r.x, r.y);
    return r;
}
__device__ __forceinline__ float2 cs(float2 a, float2 b) {
    float2 r;
    unpack2(fsub2(pack2(a.x, a.y), pack2(b.x, b.y)), r.x, r.y);
    return r;
}
__device__ __forceinline__ float2 cm(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a + SIGN i b
template <int SIGN>
__device__ __forceinline__ float2 cai(float2 a, float2 b) {
    return SIGN > 0 ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}
// Twiddle entries are e^{-i t}; the image -> uv direction takes the conjugate.
template <int DIR>
__device__ __forceinline__ float2 ct(float2 a, float2 w) {
    return cm(a, make_float2(w.x, DIR < 0 ? w.y : -w.y));
}

// One float2 of padding after every 16 elements of a line in the exchange: a
// thread's stride-16 outputs of the first pass fall in distinct banks.
__host__ __device__ constexpr int pad16(int i) { return i + (i >> 4); }

// cos / sin of 2 pi m / 16 (compile-time constants once m is).
__host__ __device__ constexpr float kcos16(int m) {
    constexpr float t[16] = {1.f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f,
                             0.f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f,
                             -1.f, -0.92387953251128674f, -0.70710678118654752f, -0.38268343236508977f,
                             0.f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f};
    return t[m & 15];
}
__host__ __device__ constexpr float ksin16(int m) { return kcos16(m - 4); }

// DFTs in registers, natural order in and out: element r of a butterfly is x[r * ST].
template <int DIR, int ST>
__device__ __forceinline__ void dft4(float2 *x) {
    const float2 s = ca(x[0], x[2 * ST]), d = cs(x[0], x[2 * ST]), t = ca(x[ST], x[3 * ST]), u = cs(x[ST], x[3 * ST]);
    x[0] = ca(s, t);
    x[ST] = cai<DIR>(d, u);
    x[2 * ST] = cs(s, t);
    x[3 * ST] = cai<-DIR>(d, u);
}
template <int DIR, int R, int ST>
__device__ __forceinline__ void dft(float2 *x) {
    if constexpr (R == 2) {
        const float2 a = x[0], b = x[ST];
        x[0] = ca(a, b);
        x[ST] = cs(a, b);
    } else if constexpr (R == 4) {
        dft4<DIR, ST>(x);
    } else { // R = 4 B: four-point DFTs of every B-th element, twiddles, B-point DFTs
        constexpr int B = R / 4;
        float2 y[4][B]; // [c][b]
#pragma unroll
        for (int b = 0; b < B; ++b) {
            float2 z[4] = {x[b * ST], x[(B + b) * ST], x[(2 * B + b) * ST], x[(3 * B + b) * ST]};
            dft4<DIR, 1>(z);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int m = b * c * (16 / R); // of 16
                if (m == 0)
                    y[c][b] = z[c];
                else if (m == 4)
                    y[c][b] = DIR > 0 ? make_float2(-z[c].y, z[c].x) : make_float2(z[c].y, -z[c].x);
                else
                    y[c][b] = cm(z[c], make_float2(kcos16(m), DIR * ksin16(m)));
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            dft<DIR, B, 1>(y[c]);
#pragma unroll
            for (int d = 0; d < B; ++d) x[(c + 4 * d) * ST] = y[c][d];
        }
    }
}

// Pass P of a length-G transform: radix 16 while at least 16 points of the
// length are left, then one pass of radix 2, 4 or 8.
template <int G, int P>
struct Pass {
    static constexpr int L = 1 << (4 * P); // product of the radices before it
    static constexpr int R = G / L >= 16 ? 16 : G / L;
};

// The twiddles of thread b's butterflies of pass P.
template <int G, int P>
__device__ __forceinline__ void load_twiddles(float2 (&w)[16], const float2 *tw, int b) {
    using Q = Pass<G, P>;
    if constexpr (G == 256) {
#pragma unroll
        for (int r = 1; r < 16; ++r) w[r] = __ldg(tw + r * b);
    } else if constexpr (Q::R == 16) {
        const int k = (b & (Q::L - 1)) * (G / (Q::L * 16));
        w[0] = __ldg(tw + k);
        w[1] = __ldg(tw + 2 * k);
        w[2] = __ldg(tw + 3 * k);
        w[3] = __ldg(tw + 4 * k);
        w[4] = __ldg(tw + 8 * k);
        w[5] = __ldg(tw + 12 * k);
    } else {
#pragma unroll
        for (int j = 0; j < 16 / Q::R; ++j)
#pragma unroll
            for (int r = 1; r < Q::R; ++r) w[j * (Q::R - 1) + r - 1] = __ldg(tw + r * (b + j * (G / 16)));
    }
}

// Pass P on a line's elements b + m G/16 (m < 16), which thread b holds: 16 / R
// butterflies, element r of butterfly j at m = j + r 16/R.
template <int DIR, int G, int P>
__device__ __forceinline__ void do_pass(float2 (&x)[16], const float2 (&w)[16]) {
    using Q = Pass<G, P>;
    if constexpr (P > 0 && G == 256) {
#pragma unroll
        for (int r = 1; r < 16; ++r) x[r] = ct<DIR>(x[r], w[r]);
    } else if constexpr (P > 0 && Q::R == 16) {
        float2 v[4] = {w[0], w[0], w[1], w[2]}; // powers 0 (unused), 1, 2, 3
#pragma unroll
        for (int r = 1; r < 16; ++r) {
            const int lo = r & 3, hi = r >> 2;
            const float2 f = hi == 0 ? v[lo] : lo == 0 ? w[2 + hi] : cm(v[lo], w[2 + hi]);
            x[r] = ct<DIR>(x[r], f);
        }
    } else if constexpr (P > 0) {
#pragma unroll
        for (int j = 0; j < 16 / Q::R; ++j)
#pragma unroll
            for (int r = 1; r < Q::R; ++r)
                x[j + r * (16 / Q::R)] = ct<DIR>(x[j + r * (16 / Q::R)], w[j * (Q::R - 1) + r - 1]);
    }
#pragma unroll
    for (int j = 0; j < 16 / Q::R; ++j) dft<DIR, Q::R, 16 / Q::R>(x + j);
}

// Pairs of lines per strip, G H points of one line of each pair: 8192 columns'
// points keep 512 threads busy with whole sectors, rows go in half of that so
// that two CTAs of an SM overlap; short lines stop at 32 (16) per strip.
__host__ __device__ constexpr int fft_pairs(int G, bool col) {
    const int points = col ? 8192 : 4096, h = points / G, most = col ? 16 : 8;
    return h < 1 ? 1 : h > most ? most : h;
}
template <int LOGG, bool COL>
struct Strip {
    static constexpr int G = 1 << LOGG, H = fft_pairs(G, COL), TG = G / 16, threads = TG * H;
    static constexpr uint32_t bytes = (uint32_t)G * H * 16u;
    static constexpr size_t smem = 16 + bytes + (size_t)pad16(G) * H * 8;
};

// Transforms every line of planes of G x G: COL: columns, else rows.  DIR = -1
// uses e^{-2 pi i ...}, DIR = +1 its conjugate; position p of a line is
// multiplied by corr[p] (when given) after the transform for DIR = -1 and
// before it for DIR = +1.  Persistent CTAs take strips blockIdx.x,
// + gridDim.x, ...; the next strip's copy is issued as soon as this one's is
// in registers.  A strip of rows arrives by one bulk copy, its completion
// counted on an mbarrier, the wait bounded by kWaitNs: a copy that does not
// arrive in time sets the timeout bit of `status` and the CTA stops (`lost`
// extra expected bytes on the first copy make that happen in tests).
template <int DIR, int LOGG, bool COL>
__global__ void __launch_bounds__(Strip<LOGG, COL>::threads, 512 / Strip<LOGG, COL>::threads)
    grid_fft_kernel(float2 *__restrict__ data, int strips, const float2 *__restrict__ tw,
                    const float *__restrict__ corr, unsigned *status, uint32_t lost) {
    using T = Strip<LOGG, COL>;
    constexpr int G = T::G, H = T::H, TG = T::TG, kPasses = (LOGG + 3) / 4, kHalf = 8; // kHalf: G/2 in units of TG
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    unsigned char *C = smem + 16;                            // the strip as it arrives
    float2 *X = reinterpret_cast<float2 *>(C + T::bytes);    // exchange: one line of each pair
    __shared__ int abort_flag;
    const int tid = threadIdx.x;
    const int b = COL ? tid / H : tid % TG, pair = COL ? tid % H : tid / TG;
    float2 *xp = X + (COL ? pair : pair * pad16(G));
    constexpr int kStep = COL ? H : 1; // between elements of a line in the exchange
    const uint32_t c_addr = smem_addr(C);

    auto strip_base = [&](int s) -> float2 * {
        if (!COL) return data + (int64_t)s * 2 * H * G;
        constexpr int per = G / (2 * H);
        return data + (int64_t)(s / per) * G * G + (s % per) * (2 * H);
    };
    auto fetch = [&](int s, uint32_t extra) {
        const float2 *src = strip_base(s);
        if constexpr (COL) { // every thread its own 16 elements of two columns
            const float2 *p = src + (int64_t)b * G + 2 * pair;
#pragma unroll
            for (int m = 0; m < 16; ++m)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(c_addr + (uint32_t)(m * T::threads + tid) * 16u),
                             "l"(p + (int64_t)m * TG * G));
            asm volatile("cp.async.commit_group;");
        } else if (tid == 0) {
            fence_proxy_async();
            mbar_arrive_expect_tx(bar, T::bytes + extra);
            bulk_g2s(C, src, T::bytes, bar);
        }
    };
    if (!COL) {
        if (tid == 0) {
            mbar_init(bar, 1);
            mbar_init_fence();
            abort_flag = 0;
        }
        __syncthreads();
    }
    uint32_t phase = 0;
    int s = blockIdx.x;
    if (s < strips) fetch(s, lost); // lost > 0 only under IDG_FLAG_TEST_LOST_COPY
    for (; s < strips; s += gridDim.x) {
        float2 x[2][16], w[16];
        if constexpr (COL) {
            asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                const float4 e = reinterpret_cast<const float4 *>(C)[(m ^ kHalf) * T::threads + tid];
                x[0][m] = make_float2(e.x, e.y);
                x[1][m] = make_float2(e.z, e.w);
            }
        } else {
            if (!mbar_wait_bounded(bar, phase, kWaitNs)) abort_flag = 1;
            __syncthreads();
            if (abort_flag) {
                if (tid == 0) {
                    flag_status(status, kStatusTimeout);
                    mbar_wait_bounded(bar, phase, kWaitNs); // the copy in flight, once more
                }
                break;
            }
            phase ^= 1u;
            const float2 *c = reinterpret_cast<const float2 *>(C) + 2 * pair * G + b;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                x[0][m] = c[(m ^ kHalf) * TG];
                x[1][m] = c[(m ^ kHalf) * TG + G];
            }
        }
        if (DIR > 0 && corr) {
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                const float f = __ldg(corr + b + (m ^ kHalf) * TG);
                x[0][m] = make_float2(x[0][m].x * f, x[0][m].y * f);
                x[1][m] = make_float2(x[1][m].x * f, x[1][m].y * f);
            }
        }
        // everyone is done with the previous strip's exchange and (rows) with C
        __syncthreads();
        if (s + (int)gridDim.x < strips) fetch(s + gridDim.x, 0u);

        auto put = [&](const float2(&v)[16], auto p) {
            constexpr int L = 1 << (4 * decltype(p)::value);
            float2 *o = xp + kStep * pad16((b / L) * L * 16 + (b & (L - 1)));
            if constexpr (L == 1) {
#pragma unroll
                for (int r = 0; r < 16; ++r) o[kStep * r] = v[r];
            } else {
#pragma unroll
                for (int r = 0; r < 16; ++r) o[kStep * r * (L + L / 16)] = v[r];
            }
        };
        auto get = [&](float2(&v)[16]) {
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = xp[kStep * pad16(b + m * TG)];
        };
        do_pass<DIR, G, 0>(x[0], w);
        // the two lines take turns: one is exchanged while the other is transformed
        auto exchange = [&](auto p) {
            constexpr int P = decltype(p)::value;
            put(x[0], p);
            do_pass<DIR, G, P>(x[1], w);
            load_twiddles<G, P + 1>(w, tw, b);
            __syncthreads();
            get(x[0]);
            __syncthreads();
            put(x[1], p);
            do_pass<DIR, G, P + 1>(x[0], w);
            __syncthreads();
            get(x[1]);
            if constexpr (P + 2 < kPasses) __syncthreads();
        };
        exchange(std::integral_constant<int, 0>{});
        if constexpr (kPasses > 2) exchange(std::integral_constant<int, 1>{});
        if constexpr (kPasses > 3) exchange(std::integral_constant<int, 2>{});
        do_pass<DIR, G, kPasses - 1>(x[1], w);

        float2 *out = strip_base(s);
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int p = b + (m ^ kHalf) * TG;
            const float f = DIR < 0 && corr ? __ldg(corr + p) : 1.f;
            const float4 v = make_float4(x[0][m].x * f, x[0][m].y * f, x[1][m].x * f, x[1][m].y * f);
            if constexpr (COL) {
                *reinterpret_cast<float4 *>(out + (int64_t)p * G + 2 * pair) = v;
            } else {
                out[2 * pair * G + p] = make_float2(v.x, v.y);
                out[(2 * pair + 1) * G + p] = make_float2(v.z, v.w);
            }
        }
    }
}

template <int DIR, int LOGG, bool COL>
cudaError_t fft_pass(float2 *grid, int planes, const float2 *tw, const float *corr, unsigned *status, uint32_t lost,
                     cudaStream_t st) {
    using T = Strip<LOGG, COL>;
    auto kern = grid_fft_kernel<DIR, LOGG, COL>;
    const LaunchDevice d = launch_device();
    if (d.error != cudaSuccess) return d.error;
    static std::atomic<uint64_t> allowed{0};
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kern), &allowed);
    if (e != cudaSuccess) return e;
    const int64_t strips = (int64_t)planes * (T::G / (2 * T::H));
    if (strips > INT32_MAX) return cudaErrorInvalidValue;
    const int64_t per_sm = std::max<int64_t>(1, std::min<int64_t>(512 / T::threads, (int64_t)(227 * 1024 / (T::smem + 1040))));
    const int64_t blocks = std::min<int64_t>(strips, d.sms * per_sm);
    kern<<<(unsigned)blocks, T::threads, T::smem, st>>>(grid, (int)strips, tw, corr, status, lost);
    return cudaGetLastError();
}

template <int DIR, int LOGG>
cudaError_t both_passes(float2 *grid, int planes, const float2 *tw, const float *corr, unsigned *status, uint32_t lost,
                        cudaStream_t st) {
    cudaError_t e = fft_pass<DIR, LOGG, false>(grid, planes, tw, corr, status, lost, st);
    if (e != cudaSuccess) return e;
    return fft_pass<DIR, LOGG, true>(grid, planes, tw, corr, status, 0u, st);
}

template <int DIR>
cudaError_t grid_fft_g(int logG, float2 *grid, int planes, const float2 *tw, const float *corr, unsigned *status,
                       uint32_t lost, cudaStream_t st) {
    switch (logG) {
    case 6: return both_passes<DIR, 6>(grid, planes, tw, corr, status, lost, st);
    case 7: return both_passes<DIR, 7>(grid, planes, tw, corr, status, lost, st);
    case 8: return both_passes<DIR, 8>(grid, planes, tw, corr, status, lost, st);
    case 9: return both_passes<DIR, 9>(grid, planes, tw, corr, status, lost, st);
    case 10: return both_passes<DIR, 10>(grid, planes, tw, corr, status, lost, st);
    case 11: return both_passes<DIR, 11>(grid, planes, tw, corr, status, lost, st);
    case 12: return both_passes<DIR, 12>(grid, planes, tw, corr, status, lost, st);
    case 13: return both_passes<DIR, 13>(grid, planes, tw, corr, status, lost, st);
    default: return cudaErrorInvalidValue;
    }
}

std::mutex g_tw_mutex;
std::map<std::pair<int, int>, float2 *> g_tw; // (device, G) -> e^{-2 pi i m / G}, m < G

cudaError_t twiddles(int G, const float2 **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_tw_mutex);
    auto it = g_tw.find({dev, G});
    if (it != g_tw.end()) {
        *out = it->second;
        return cudaSuccess;
    }
    std::vector<float2> h(G);
    for (int m = 0; m < G; ++m) {
        const double a = -2.0 * M_PI * (double)m / (double)G;
        h[m] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    float2 *d = nullptr;
    e = cudaMalloc(&d, sizeof(float2) * G);
    if (e != cudaSuccess) return e;
    e = cudaMemcpy(d, h.data(), sizeof(float2) * G, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return e;
    }
    g_tw[{dev, G}] = d;
    *out = d;
    return cudaSuccess;
}

} // namespace

bool grid_fft_size_supported(int G) { return G >= 64 && G <= 8192 && (G & (G - 1)) == 0; }

cudaError_t launch_grid_fft(float2 *grid, int G, int planes, int direction, const float *corr, unsigned *status,
                            bool test_lost_copy, cudaStream_t st) {
    const uint32_t lost = test_lost_copy ? 16u : 0u;
    if (!grid_fft_size_supported(G)) return cudaErrorInvalidValue;
    const float2 *tw = nullptr;
    cudaError_t e = twiddles(G, &tw);
    if (e != cudaSuccess) return e;
    int logG = 0;
    while ((1 << logG) < G) ++logG;
    return direction < 0 ? grid_fft_g<-1>(logG, grid, planes, tw, corr, status, lost, st)
                         : grid_fft_g<1>(logG, grid, planes, tw, corr, status, lost, st);
}

} // namespace idg

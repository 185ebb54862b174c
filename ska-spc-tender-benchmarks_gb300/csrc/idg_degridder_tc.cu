// idg_degridder_tc.cu -- the degridder on the tensor cores.
//
// With the factors of idg_tc.cuh a visibility is
//   V = sum_y conj(Q(y)) H(y),   H(y) = sum_x conj(P(x)) S'(x, y)  (+ first order),
// S' the subgrid's pixels after taper, A-terms and the per-pixel phase factor.
// H for a tile of 128 visibilities is a matrix product: visibilities x (cos,
// sin of the x-factors) times the (x, pixel row and polarisation) matrix S'.
//  * M = 128 visibilities: thread i of a warpgroup owns visibility i.  Two
//    factor warpgroups take tiles in turn: they form the x-factors and store
//    them, split into fp16 hi + lo, as the A operand into their own lanes of
//    tensor memory; nothing is exchanged between threads.
//  * N = (row, polarisation, re | im): S' as fp16 hi and lo in shared memory,
//    made once per subgrid and block, in three groups of rows Sr | Si | -Sr, so
//    that cos times (Sr, Si) and sin times (Si, -Sr) give Hr and Hi side by
//    side in one product of N = 128 (16 rows).
//  * Two result warpgroups take tiles in turn, thread = visibility again: they
//    read H and finish the sum over y in fp32 registers with their own
//    y-factors: no reduction across threads.
//  * One warp issues the products: the rows of a block in two halves, each with
//    an accumulator of its own, so that one fills while the other is read.
//  * One warp runs ahead: it fetches the next subgrid, checks it and asks for
//    its pixels and A-terms; the factor warps, which have time to spare, stage
//    its S' into the other of two buffers while the tensor core works on the
//    current one.
// One CTA of 18 warps per SM: all of its tensor memory (448 of the 512 columns that
// an allocation has to be are used), 147 KB of operands.
// Measured on GB300, 4,416 subgrids of 128 x 16 visibilities at S = 32: 0.90 ms
// (24.6 SM cycles per visibility beyond a fixed 7 us per subgrid and SM), against
// 5.27 ms for the mirror-quad kernel.  The products alone take 16 cycles per
// visibility; the rest is the issue slots of the factor and result warps, which
// share the SM's four schedulers.  28 subgrids of 64 x 16 in one call: 25 us
// against 115 us.
// Subgrids larger than 32 are done in blocks of at most 32 x 32 pixels, the
// later blocks adding to the visibilities written by the first, once all results
// of the block before are stored.
#include "idg_tc.cuh"
#include "idg_internal.h"

namespace idg {

namespace {

constexpr int kGen = 256;                 // factor threads (two warpgroups)
constexpr int kThreads = 2 * kGen + 64;   // + two result warpgroups, the issuing and the scouting warp
constexpr int kTile = 128;                // visibilities per tile
constexpr int kGroup = 4, kSegTiles = 16; // subgrids sharing their long ones, least tiles of a segment
constexpr int kAcc = 2;                   // accumulators of 128 columns: (re | im) x ROWS x 4 polarisations
constexpr uint32_t kColA = 256, kColsA = 96, kTmemCols = 512;

// A subgrid found by the scouting warp.
struct Item {
    int stop, s, row0, c0, nc, nvis, t_begin, t_end;
    unsigned st1, st2;
    int aterm;
    TcSubgrid sg;
};

// One subgrid block on its way through the roles.
struct Job {
    int stop, nc, t_begin, t_end, c0, row0, y0, add;
    int nvis;
    TcSubgrid sg;
    float4 inv; // per polarisation
};

struct Head {
    uint64_t a_full[2], a_free[2];           // per factor warpgroup
    uint64_t d_full[2][kAcc], d_free[2][kAcc]; // per result warpgroup and row group of its tile
    uint64_t job_full[2], job_free[2], b_free[2];
    uint64_t item_full, item_free;
    uint64_t drain;
    uint32_t tmem;
    TcWatch watch;
    int gen_stop;
    uint4 max_bits; // per polarisation
    unsigned scratch[kTcScratch];
    Item item;
    Job job[2];
};

// Blocks of a subgrid and the operand layout.
struct Shape {
    int nb, bs; // blocks per axis, pixels per block (even)
    int kx;     // x extent of a block padded to 16: the K of the product
    int rows;   // rows per accumulator: 8, 12 or 16 (the kernel's ROWS)
    int nq;     // accumulators' worth of rows in a block
};
__host__ __device__ inline Shape tc_shape(int S) {
    Shape s;
    s.nb = S > 32 ? 2 : 1;
    s.bs = s.nb == 1 ? S : 2 * ((S + 3) / 4);
    s.kx = s.bs <= 16 ? 16 : 32;
    s.nq = s.bs <= 16 ? 1 : 2;
    s.rows = (s.bs / s.nq + 3) & ~3;
    return s;
}
template <int ROWS>
struct Op { // one accumulator's operand, for one of hi, lo, first order
    static constexpr uint32_t ks = 12 * ROWS * 16 + 16; // bytes between 8-wide k groups (16: conflict-free stores)
    static constexpr uint32_t bytes = (4 * ks + 127u) & ~127u;
};

struct Layout {
    size_t b, axis, ntab, chan, total;
    uint32_t bset; // bytes of one operand set: hi, lo, first order
};
template <int ROWS>
__host__ __device__ inline Layout tc_layout(int S, int C) {
    const Shape s = tc_shape(S);
    Layout L;
    size_t off = (sizeof(Head) + 127) & ~size_t(127);
    L.bset = 3u * Op<ROWS>::bytes * (uint32_t)s.nq;
    L.b = off;    off += 2 * (size_t)L.bset;
    L.axis = off; off += (size_t)(s.nb * s.bs / 2 + 16) * 32;
    L.ntab = off; off += (size_t)(S / 2) * (S / 2) * 8;
    off = (off + 15) & ~size_t(15);
    L.chan = off; off += (size_t)C * 16;
    L.total = off;
    return L;
}

// One visibility's row: u, v, w and the wavenumber factors.
struct Vis {
    float u, v, w;
    float4 k;
};
__device__ __forceinline__ Vis load_vis(const KernelArgs &a, const float4 *chan, int row0, int c0, int nc, int i) {
    const int t = i / nc, c = c0 + i - t * nc;
    const float *p = a.uvw + 3 * ((int64_t)row0 + t);
    return {p[0], p[1], p[2], chan[c]};
}

__device__ __forceinline__ void gen_sync() { named_sync<1, kGen>(); }

// Row of a row group's operand for (row y of the group, polarisation p): four rows
// y of one polarisation next to each other, so that the results of a row pair
// come out of tensor memory as register pairs.
__device__ __forceinline__ uint32_t op_row(int y, int p) { return (uint32_t)(16 * (y >> 2) + 4 * p + (y & 3)); }

// S' of the block's pixels (x0 + x, y0 + y) into the operand layout: first the
// largest magnitude of each polarisation (cross-hands may be far below the
// others), then scaled and split.  inv: the reciprocal scales.
template <int ROWS>
__device__ __forceinline__ void stage_block(const KernelArgs &a, const Item &si, Head *head, const Shape &sh, int x0,
                                             int y0, unsigned char *bh, const float4 *axis, const float2 *ntab,
                                             float4 &inv) {
    const TcSubgrid &sg = si.sg;
    const int s = si.s;
    const int tid = threadIdx.x, S = a.S, S2 = S * S, Sh = S / 2;
    const bool refcpu = (a.flags & IDG_FLAG_DEGRID_ATERM_REFCPU) != 0;
    const bool taper = (a.flags & IDG_FLAG_NO_TAPER) == 0;
    const size_t jones = (size_t)S2 * 2;
    const float4 *a1 = a.aterms + ((size_t)si.aterm * a.nr_stations + si.st1) * jones;
    const float4 *a2 = a.aterms + ((size_t)si.aterm * a.nr_stations + si.st2) * jones;
    const int kp = sh.kx / 2, items = kp * sh.nq * ROWS;
    unsigned char *bl = bh + Op<ROWS>::bytes * sh.nq, *b1 = bl + Op<ROWS>::bytes * sh.nq;
    gen_sync(); // the previous block's readers of max_bits are past it
    if (tid < 4) (&head->max_bits.x)[tid] = 0u;
    gen_sync();
    constexpr int kIter = 2; // at most 512 pixel pairs
    cf v[kIter][2][4];
    unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int it = 0; it < kIter; ++it) {
        const int i = tid + it * kGen;
        const int y = i / kp, x = 2 * (i - y * kp);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int gx = x0 + x + e, gy = y0 + y;
            const bool in = i < items && x + e < sh.bs && y < sh.bs && gx < S && gy < S;
            if (in) {
                const int q = gy * S + gx;
                const float2 n = ntab[(gy < Sh ? gy : S - 1 - gy) * Sh + (gx < Sh ? gx : S - 1 - gx)];
                cf j1[4], j2[4];
                load_jones(a1 + 2 * q, j1);
                load_jones(a2 + 2 * q, j2);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 w = a.subgrids[((size_t)s * 4 + p) * S2 + q];
                    v[it][e][p] = {w.x, w.y};
                }
                const cf f = cscale(cconj(tc_pixel_factor(sg.g0h, sg.g0l, n)), taper ? a.taper[q] : 1.f);
                if (refcpu)
                    aterm_gridder(v[it][e], j1, j2);
                else
                    aterm_adjoint(v[it][e], j1, j2);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    v[it][e][p] = cmul(f, v[it][e][p]);
                    m[p] = max(m[p], max(__float_as_uint(fabsf(v[it][e][p].re)), __float_as_uint(fabsf(v[it][e][p].im))));
                }
            } else {
#pragma unroll
                for (int p = 0; p < 4; ++p) v[it][e][p] = {0.f, 0.f};
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) m[p] = __reduce_max_sync(0xffffffffu, m[p]);
    if ((tid & 31) < 4) atomicMax(&head->max_bits.x + (tid & 3), (tid & 2) ? (tid & 1) ? m[3] : m[2] : (tid & 1) ? m[1] : m[0]);
    gen_sync();
    const uint4 most = head->max_bits;
    const float scale[4] = {tc_scale(most.x, inv.x), tc_scale(most.y, inv.y), tc_scale(most.z, inv.z), tc_scale(most.w, inv.w)};
#pragma unroll
    for (int it = 0; it < kIter; ++it) {
        const int i = tid + it * kGen;
        if (i >= items) continue;
        const int y = i / kp, x = 2 * (i - y * kp), h = y / ROWS, yl = y % ROWS;
        const float4 ax = axis[2 * ((y0 + y) >> 1) + 1]; // cx of the row pair
        const float cy = ((y0 + y) & 1) ? ax.y : ax.x;
        const uint32_t base = (uint32_t)h * Op<ROWS>::bytes + (uint32_t)(x >> 3) * Op<ROWS>::ks + (uint32_t)(x & 7) * 2u;
        constexpr uint32_t g = ROWS * 64u; // from a row of Sr to its row of Si, and on to -Sr
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const f2 re = fmul2(pack2(v[it][0][p].re, v[it][1][p].re), pack2(scale[p], scale[p]));
            const f2 im = fmul2(pack2(v[it][0][p].im, v[it][1][p].im), pack2(scale[p], scale[p]));
            uint32_t rh, rl, ih, il;
            tc_split(re, rh, rl);
            tc_split(im, ih, il);
            const uint32_t o = base + op_row(yl, p) * 16u;
            *reinterpret_cast<uint32_t *>(bh + o) = rh;
            *reinterpret_cast<uint32_t *>(bh + o + g) = ih;
            *reinterpret_cast<uint32_t *>(bh + o + 2u * g) = rh ^ 0x80008000u;
            *reinterpret_cast<uint32_t *>(bl + o) = rl;
            *reinterpret_cast<uint32_t *>(bl + o + g) = il;
            *reinterpret_cast<uint32_t *>(bl + o + 2u * g) = rl ^ 0x80008000u;
            if (sg.cross) {
                const uint32_t cr = tc_half2(fmul2(re, pack2(cy, cy))), ci = tc_half2(fmul2(im, pack2(cy, cy)));
                *reinterpret_cast<uint32_t *>(b1 + o) = cr;
                *reinterpret_cast<uint32_t *>(b1 + o + g) = ci;
                *reinterpret_cast<uint32_t *>(b1 + o + 2u * g) = cr ^ 0x80008000u;
            }
        }
    }
    fence_proxy_async(); // the tensor core reads the operand through the asynchronous proxy
}

// x-factors of one tile into the A operand (columns Ch | Cl | Sh | Sl | A1c | A1s).
__device__ __forceinline__ void store_factors(uint32_t tm, const Shape &sh, const float4 *axis, float hi, float lo,
                                              float d, bool cross) {
    const f2 H = pack2(hi, hi), L = pack2(lo, lo), D = pack2(d, d);
    const uint32_t w = (uint32_t)(sh.kx / 2);
    for (int p0 = 0; p0 < sh.kx / 2; p0 += 4) {
        uint32_t ch[4], cl[4], sn[4], sl[4], c1[4], s1[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 g = axis[2 * (p0 + i)];
            f2 c, s;
            tc_sincos(H, L, D, pack2(g.x, g.y), pack2(g.z, g.w), c, s);
            tc_split(c, ch[i], cl[i]);
            tc_split(s, sn[i], sl[i]);
            if (cross) {
                const float4 x = axis[2 * (p0 + i) + 1];
                const f2 e = fmul2(D, pack2(x.x, x.y));
                c1[i] = tc_half2(fmul2(e, c));
                s1[i] = tc_half2(fmul2(e, s));
            }
        }
        tmem_st4(tm + p0, ch);
        tmem_st4(tm + w + p0, cl);
        tmem_st4(tm + 2 * w + p0, sn);
        tmem_st4(tm + 3 * w + p0, sl);
        if (cross) {
            tmem_st4(tm + 4 * w + p0, c1);
            tmem_st4(tm + 5 * w + p0, s1);
        }
    }
}

// The products of one row group: D = Hr | Hi of its rows.  The accumulator is
// truncated after every product: the small ones (lo parts, first-order term)
// come first, the hi hi products last.  bh, bl, b1: descriptors of the group's
// operands.
template <int ROWS, int KJ, bool CROSS>
__device__ __forceinline__ void issue_rows(uint32_t d, uint32_t am, uint32_t bh, uint32_t bl, uint32_t b1) {
    constexpr uint32_t id = umma_idesc_f16(128, 8 * ROWS), hi = umma_desc_hi(128);
    constexpr uint32_t w = 8 * KJ, dk = (2 * Op<ROWS>::ks) >> 4, off = (ROWS * 64) >> 4; // next 16 x; rows Si | -Sr
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
        const uint32_t c = am + 8u * (uint32_t)j, k = j * dk;
        if (j == 0)
            umma_f16_ts<false, id, hi>(d, c, bl + k);
        else
            umma_f16_ts<true, id, hi>(d, c, bl + k);
        umma_f16_ts<true, id, hi>(d, c + w, bh + k);
        umma_f16_ts<true, id, hi>(d, c + 2 * w, bl + k + off);
        umma_f16_ts<true, id, hi>(d, c + 3 * w, bh + k + off);
        if (CROSS) {
            umma_f16_ts<true, id, hi>(d, c + 4 * w, b1 + k + off);
            umma_f16_ts<true, (id | kUmmaNegateA), hi>(d, c + 5 * w, b1 + k);
        }
    }
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
        const uint32_t c = am + 8u * (uint32_t)j, k = j * dk;
        umma_f16_ts<true, id, hi>(d, c, bh + k);
        umma_f16_ts<true, id, hi>(d, c + 2 * w, bh + k + off);
    }
}

// The scouting warp: takes work from the counter, leaves out what the
// expansion does not hold for, and asks L2 for the pixels and A-terms of the
// others.
//  * nseg > 0 (fewer subgrids than CTAs): a claim is one of nseg equal segments
//    of a subgrid's tiles.
//  * nseg = 0: a claim is one of kGroup subgrids of a group, shared like this: a
//    subgrid of 2 kSegTiles tiles or more is cut into up to kGroup segments
//    (as many as the group has members), and claim q of a group takes segment
//    q - j modulo the members of its subgrid j.
//    So there are as many claims as subgrids, a short subgrid (one segment) is
//    one claim, and a long one is spread over its neighbours' claims: one of
//    16,384 visibilities at S = 48 held its SM for 0.75 ms at the end of the
//    call.  Degridding steps, whole and shared: 1,500 subgrids of 128 to 16,384
//    visibilities at S = 48 2.01 and 1.59 ms, 600 at S = 32 408 and 271 us, 1,500
//    at S = 24 539 and 446; for 4,416 even ones the look at the neighbours costs
//    5 of 880 us, of one tile each 6 of 228.  Claims for every segment, the empty
//    ones too, made that last call 299 us.
__device__ __forceinline__ void scout_role(const KernelArgs &a, int nseg, Head *head) {
    volatile TcWatch *watch = &head->watch;
    const int lane = threadIdx.x & 31;
    const size_t jones = (size_t)a.S * a.S * 2; // float4 per matrix plane
    uint32_t k = 0;
    auto publish = [&](const Item &it) {
        if (k > 0) tc_wait(&head->item_free, (k - 1) & 1, watch, a.status);
        // a wait that was given up leaves the item to those who may be reading it
        if (__any_sync(0xffffffffu, watch->abort)) return;
        if (lane == 0) {
            head->item = it;
            mbar_arrive(&head->item_full);
        }
        ++k;
    };
    for (;;) {
        int item = 0;
        if (lane == 0) item = watch->abort ? INT32_MAX : atomicAdd(a.work_counter, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        Item it{};
        if (item >= a.nr_subgrids * (nseg > 0 ? nseg : 1)) {
            it.stop = 1;
            publish(it);
            return;
        }
        // the claim's own subgrid, and on lane j how subgrid j of its group is cut
        const int q = nseg > 0 ? 0 : item % kGroup, first = nseg > 0 ? item / nseg : item - q;
        auto subgrid = [&](int j) { return a.work_list ? a.work_list[first + j] : first + j; };
        SubgridInfo si = load_subgrid(a, subgrid(q));
        const int members = nseg > 0 ? 1 : (int)min((int64_t)kGroup, a.nr_subgrids - first); // the last group may be short
        int parts = nseg;
        if (nseg == 0 && lane < members) {
            const int s = subgrid(lane), nc = a.ext ? a.ext[s].channel_end - a.ext[s].channel_begin : a.C;
            const int64_t ntiles = (int64_t)a.md[s].nr_timesteps * nc / kTile;
            parts = (int)max((int64_t)1, min((int64_t)members, ntiles / kSegTiles));
        }
        const int seg = nseg > 0 ? item - first * nseg : q - lane + (q < lane ? members : 0);
        unsigned todo = __ballot_sync(0xffffffffu, seg < parts && lane < members); // q among them
        for (int j = q; todo != 0; todo &= ~(1u << j)) {
            if ((todo >> j & 1u) == 0) { // after the claim's own
                j = __ffs((int)todo) - 1;
                si = load_subgrid(a, subgrid(j));
            }
            if (lane == 0) watch->looked = global_timer_ns();
            const int sj = subgrid(j), segj = __shfl_sync(0xffffffffu, seg, j), partsj = __shfl_sync(0xffffffffu, parts, j);
            if (!si.ok) {
                if (lane == 0) flag_status(a.status, kStatusBadPlan);
                continue;
            }
            const int nc = si.c1 - si.c0;
            if (nc == 0 || si.T == 0) continue;
            if (!tc_fits<32>(a, si, head->scratch, &it.sg, [] { __syncwarp(); })) {
                if (lane == 0) atomicAdd(a.fallback, 1);
                continue;
            }
            const char *px = reinterpret_cast<const char *>(a.subgrids + (size_t)sj * 4 * a.S * a.S);
            const char *j1 = reinterpret_cast<const char *>(a.aterms + ((size_t)si.aterm * a.nr_stations + si.st1) * jones);
            const char *j2 = reinterpret_cast<const char *>(a.aterms + ((size_t)si.aterm * a.nr_stations + si.st2) * jones);
            for (size_t o = (size_t)lane * 128; o < jones * 16; o += 32 * 128) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(px + o));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(j1 + o));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(j2 + o));
            }
            it.s = sj;
            it.row0 = si.row0;
            it.c0 = si.c0;
            it.nc = nc;
            it.nvis = si.T * nc; // tc_fits bounds it
            it.st1 = si.st1;
            it.st2 = si.st2;
            it.aterm = si.aterm;
            const int ntiles = (it.nvis + kTile - 1) / kTile;
            it.t_begin = (int)((int64_t)ntiles * segj / partsj);
            it.t_end = (int)((int64_t)ntiles * (segj + 1) / partsj);
            if (it.t_begin < it.t_end) publish(it);
        }
    }
}

// Factor warps: subgrid after subgrid, its staging, then this warpgroup's tiles.
template <int ROWS, bool BLOCKS>
__device__ __forceinline__ void factor_role(const KernelArgs &a, Head *head, const Shape &sh, const Layout &L,
                                            unsigned char *smem, uint32_t tl) {
    const float4 *axis = reinterpret_cast<const float4 *>(smem + L.axis);
    const float2 *ntab = reinterpret_cast<const float2 *>(smem + L.ntab);
    const float4 *chan = reinterpret_cast<const float4 *>(smem + L.chan);
    volatile TcWatch *watch = &head->watch;
    const int tid = threadIdx.x, wg = tid >> 7, lane = tid & 127;
    uint32_t n = 0, uses = 0, j = 0; // tiles so far, this warpgroup's, jobs so far
    for (uint32_t k = 0;; ++k) {
        tc_wait(&head->item_full, k & 1, watch, a.status);
        if (tid == 0) head->gen_stop = head->item.stop || watch->abort; // one answer for all
        gen_sync();
        const Item it = head->item;
        const bool stop = head->gen_stop != 0;
        gen_sync();
        mbar_arrive(&head->item_free);
        if (stop) break;

        for (int block = 0; block < (BLOCKS ? 4 : 1); ++block, ++j) {
            const int x0 = (block & 1) * sh.bs, y0 = (block >> 1) * sh.bs;
            const uint32_t buf = j & 1;
            if (j >= 2) {
                tc_wait(&head->b_free[buf], ((j >> 1) - 1) & 1, watch, a.status);
                tc_wait(&head->job_free[buf], ((j >> 1) - 1) & 1, watch, a.status);
            }
            float4 inv;
            stage_block<ROWS>(a, it, head, sh, x0, y0, smem + L.b + buf * L.bset, axis, ntab, inv);
            if (tid == 0 && !watch->abort) // after a wait that was given up others may be reading the last one
                head->job[buf] = Job{0, it.nc, it.t_begin, it.t_end, it.c0, it.row0, y0, block > 0, it.nvis, it.sg,
                                     make_float4(inv.x * kTcTruncation, inv.y * kTcTruncation, inv.z * kTcTruncation,
                                                 inv.w * kTcTruncation)};
            gen_sync();
            if (tid == 0) mbar_arrive(&head->job_full[buf]);

            // this warpgroup's tiles, the next one's row loaded ahead
            int tile = it.t_begin + (int)((n ^ (uint32_t)wg) & 1u);
            n += (uint32_t)(it.t_end - it.t_begin);
            if (tile >= it.t_end) continue;
            Vis nv = load_vis(a, chan, it.row0, it.c0, it.nc, min(tile * kTile + lane, it.nvis - 1));
            for (; tile < it.t_end; tile += 2, ++uses) {
                const Vis v = nv;
                if (tile + 2 < it.t_end)
                    nv = load_vis(a, chan, it.row0, it.c0, it.nc, min((tile + 2) * kTile + lane, it.nvis - 1));
                float hi, lo;
                tc_slope(v.k.x, v.k.y, v.u, it.sg.xh, it.sg.xl, hi, lo);
                const float d = kTwoPiF * tc_delta(v.k.z, v.k.w, v.w, it.sg.mid);
                if (uses > 0) tc_wait(&head->a_free[wg], (uses - 1) & 1, watch, a.status);
                __syncwarp();
                tmem_fence_after();
                store_factors(tl + kColA + kColsA * wg, sh, axis + x0, hi, lo * kTwoPiF, d, it.sg.cross != 0);
                tmem_wait_st();
                tmem_fence_before();
                mbar_arrive(&head->a_full[wg]);
            }
        }
    }
    // the end, for the other roles
    const uint32_t buf = j & 1;
    if (j >= 2) tc_wait(&head->job_free[buf], ((j >> 1) - 1) & 1, watch, a.status);
    gen_sync();
    if (tid == 0) {
        head->job[buf].stop = 1;
        mbar_arrive(&head->job_full[buf]);
    }
}

// Result warps: H times the y-factors, summed over the rows.
template <int ROWS, bool BLOCKS>
__device__ __forceinline__ void result_role(const KernelArgs &a, Head *head, const Shape &sh, const Layout &L,
                                            unsigned char *smem, uint32_t tl) {
    const float4 *axis = reinterpret_cast<const float4 *>(smem + L.axis);
    const float4 *chan = reinterpret_cast<const float4 *>(smem + L.chan);
    volatile TcWatch *watch = &head->watch;
    const int wg = (threadIdx.x >> 7) & 1, lane = threadIdx.x & 127;
    uint32_t n = 0, uses = 0;
    for (uint32_t j = 0;; ++j) {
        const uint32_t buf = j & 1;
        tc_wait(&head->job_full[buf], (j >> 1) & 1, watch, a.status);
        __syncwarp();
        if (__any_sync(0xffffffffu, watch->abort)) return;
        const Job job = head->job[buf];
        if (job.stop) return;
        // With an odd number of tiles the block before had a tile in the other
        // warpgroup: its stores come before this one's reads.  (Its threads are past that
        // job or ahead of this one in the products' order, so they never wait for this
        // one.)
        if (BLOCKS && job.add) tc_wait(&head->job_free[buf ^ 1], ((j - 1) >> 1) & 1, watch, a.status);
        const int nvis = job.nvis;
        const uint32_t n0 = n;
        int tile = job.t_begin + (int)((n ^ (uint32_t)wg) & 1u);
        n += (uint32_t)(job.t_end - job.t_begin);
        if (tile < job.t_end) {
            Vis nv = load_vis(a, chan, job.row0, job.c0, job.nc, min(tile * kTile + lane, nvis - 1));
            for (; tile < job.t_end; tile += 2, ++uses) {
                const Vis v = nv;
                if (tile + 2 < job.t_end)
                    nv = load_vis(a, chan, job.row0, job.c0, job.nc, min((tile + 2) * kTile + lane, nvis - 1));
                float hi, lo;
                tc_slope(v.k.x, v.k.y, v.v, job.sg.yh, job.sg.yl, hi, lo);
                const float d = kTwoPiF * tc_delta(v.k.z, v.k.w, v.w, job.sg.mid);
                lo *= kTwoPiF;
                const f2 H = pack2(hi, hi), Lo = pack2(lo, lo), D = pack2(d, d);
                f2 vr[4], vi[4]; // per polarisation, even and odd rows
#pragma unroll
                for (int p = 0; p < 4; ++p) vr[p] = vi[p] = 0ull;
                const uint32_t r0 = (n0 + (uint32_t)(tile - job.t_begin)) * (uint32_t)sh.nq;
                for (int h = 0; h < sh.nq; ++h) {
                    const float4 *ax = axis + job.y0 + h * ROWS;
                    const uint32_t col = tl + ((r0 + h) % kAcc) * 128u;
                    tc_wait(&head->d_full[wg][h], uses & 1, watch, a.status);
                    __syncwarp();
                    tmem_fence_after();
#pragma unroll
                    for (int q = 0; q < ROWS; q += 4) { // four rows: 16 columns of Hr, 16 of Hi
                        f2 hr[8], hm[8], qc[2], qs[2];
                        tmem_ld16x2(col + 4 * q, col + 4 * ROWS + 4 * q, hr, hm);
                        if (q + 4 >= ROWS) {
                            tmem_fence_before();
                            mbar_arrive(&head->d_free[wg][h]);
                        }
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const float4 g = ax[q + 2 * r];
                            tc_sincos(H, Lo, D, pack2(g.x, g.y), pack2(g.z, g.w), qc[r], qs[r]);
                        }
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const f2 ms = qs[r] ^ 0x8000000080000000ull;
#pragma unroll
                            for (int p = 0; p < 4; ++p) {
                                const f2 x = hr[2 * p + r], y = hm[2 * p + r];
                                vr[p] = ffma2(y, qs[r], ffma2(x, qc[r], vr[p]));
                                vi[p] = ffma2(x, ms, ffma2(y, qc[r], vi[p]));
                            }
                        }
                    }
                }
                const int i = tile * kTile + lane;
                if (i < nvis) {
                    const int t = i / job.nc, c = job.c0 + i - t * job.nc;
                    float4 *dst = a.vis + (((int64_t)job.row0 + t) * a.C + c) * 2;
                    const float4 i4 = head->job[buf].inv;
                    float o[8];
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float inv = p == 0 ? i4.x : p == 1 ? i4.y : p == 2 ? i4.z : i4.w;
                        float e, f;
                        unpack2(vr[p], e, f);
                        o[2 * p] = (e + f) * inv;
                        unpack2(vi[p], e, f);
                        o[2 * p + 1] = (e + f) * inv;
                    }
                    if (BLOCKS && job.add) {
                        const float4 e = dst[0], f = dst[1];
                        o[0] += e.x, o[1] += e.y, o[2] += e.z, o[3] += e.w;
                        o[4] += f.x, o[5] += f.y, o[6] += f.z, o[7] += f.w;
                    }
                    dst[0] = make_float4(o[0], o[1], o[2], o[3]);
                    dst[1] = make_float4(o[4], o[5], o[6], o[7]);
                }
            }
        }
        mbar_arrive(&head->job_free[buf]);
    }
}

// The tiles of one job.  n, r: tiles and row halves before them; b0: descriptor
// of the operand set.
template <int ROWS, int KJ, bool CROSS>
__device__ __forceinline__ void issue_job(const KernelArgs &a, Head *head, const Shape &sh, uint32_t t0, uint32_t b0,
                                          uint32_t n, int tiles, uint32_t lead) {
    volatile TcWatch *watch = &head->watch;
    const uint32_t group = Op<ROWS>::bytes >> 4, set = group * (uint32_t)sh.nq;
    const uint32_t back = kAcc / (uint32_t)sh.nq; // tiles to an accumulator's last user
#pragma unroll 1
    for (int i = 0; i < tiles; ++i, ++n) {
        const uint32_t w = n & 1, am = t0 + kColA + kColsA * w;
        tc_wait(&head->a_full[w], (n >> 1) & 1, watch, a.status);
#pragma unroll 1
        for (uint32_t h = 0; h < (uint32_t)sh.nq; ++h) {
            if (n >= back) tc_wait(&head->d_free[(n - back) & 1][h], ((n - back) >> 1) & 1, watch, a.status);
            tmem_fence_after();
            if (lead) {
                const uint32_t bh = b0 + h * group;
                issue_rows<ROWS, KJ, CROSS>(t0 + (sh.nq == 1 ? w : h) * 128u, am, bh, bh + set, bh + 2 * set);
                umma_commit(&head->d_full[w][h]);
                if (h + 1 == (uint32_t)sh.nq) umma_commit(&head->a_free[w]);
            }
            __syncwarp();
        }
    }
}

// One warp issues every product, tile by tile.
template <int ROWS>
__device__ __forceinline__ void issue_role(const KernelArgs &a, Head *head, const Shape &sh, const Layout &L,
                                           unsigned char *smem, uint32_t tm) {
    volatile TcWatch *watch = &head->watch;
    const uint32_t lead = elect_lane(), t0 = warp_uniform(tm);
    uint32_t n = 0;
    for (uint32_t j = 0;; ++j) {
        const uint32_t buf = j & 1;
        tc_wait(&head->job_full[buf], (j >> 1) & 1, watch, a.status);
        __syncwarp();
        if (__any_sync(0xffffffffu, watch->abort) || warp_uniform(head->job[buf].stop)) break;
        const uint32_t b0 = warp_uniform(umma_desc_lo(smem_addr(smem + L.b + buf * L.bset), Op<ROWS>::ks));
        const int tiles = (int)warp_uniform(head->job[buf].t_end - head->job[buf].t_begin);
        const bool cross = warp_uniform(head->job[buf].sg.cross) != 0;
        if (sh.kx == 32) {
            if (cross)
                issue_job<ROWS, 2, true>(a, head, sh, t0, b0, n, tiles, lead);
            else
                issue_job<ROWS, 2, false>(a, head, sh, t0, b0, n, tiles, lead);
        } else if (cross) {
            issue_job<ROWS, 1, true>(a, head, sh, t0, b0, n, tiles, lead);
        } else {
            issue_job<ROWS, 1, false>(a, head, sh, t0, b0, n, tiles, lead);
        }
        n += (uint32_t)tiles;
        if (lead) umma_commit(&head->b_free[buf]);
        __syncwarp();
    }
    if (lead && n > 0) { // products in flight end (bounded) before their memory goes, also where a reader gave up
        umma_commit(&head->drain);
        mbar_wait_bounded(&head->drain, 0, kTcWaitNs);
    }
    __syncwarp();
}

// BLOCKS: subgrids larger than 32, in four blocks.
template <int ROWS, bool BLOCKS>
__global__ void __launch_bounds__(kThreads, 1) degridder_tc_kernel(KernelArgs a, int nseg) {
    extern __shared__ __align__(128) unsigned char smem[];
    const Shape sh = tc_shape(a.S);
    const Layout L = tc_layout<ROWS>(a.S, a.C);
    Head *head = reinterpret_cast<Head *>(smem);
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 16) {
        tmem_alloc(&head->tmem, kTmemCols);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&head->a_full[i], 128);
            mbar_init(&head->a_free[i], 1);
            for (int h = 0; h < kAcc; ++h) {
                mbar_init(&head->d_full[i][h], 1);
                mbar_init(&head->d_free[i][h], 128);
            }
            mbar_init(&head->job_full[i], 1);
            mbar_init(&head->job_free[i], 256);
            mbar_init(&head->b_free[i], 1);
        }
        mbar_init(&head->item_full, 1);
        mbar_init(&head->item_free, kGen);
        mbar_init(&head->drain, 1);
        mbar_init_fence();
        head->watch = TcWatch{0, 0};
    }
    tc_axis_table(a, reinterpret_cast<float4 *>(smem + L.axis), sh.nb * sh.bs / 2 + 16, tid, kThreads);
    tc_n_table(a, reinterpret_cast<float2 *>(smem + L.ntab), tid, kThreads);
    tc_channel_table(a, reinterpret_cast<float4 *>(smem + L.chan), tid, kThreads);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tm = head->tmem;
    const uint32_t tl = tm + ((uint32_t)(warp & 3) << 21); // this warp's lane quarter

    if (warp < 8)
        factor_role<ROWS, BLOCKS>(a, head, sh, L, smem, tl);
    else if (warp < 16)
        result_role<ROWS, BLOCKS>(a, head, sh, L, smem, tl);
    else if (warp == 16)
        issue_role<ROWS>(a, head, sh, L, smem, tm);
    else
        scout_role(a, nseg, head);
    __syncthreads();
    if (warp == 16) tmem_free(tm, kTmemCols);
}

template <int ROWS, bool BLOCKS>
cudaError_t launch(const KernelArgs &args, cudaStream_t stream) {
    auto kern = degridder_tc_kernel<ROWS, BLOCKS>;
    KernelArgs a = args;
    a.tc = tc_const(a.S, a.image_size);
    const size_t smem = tc_layout<ROWS>(a.S, a.C).total;
    static std::atomic<uint64_t> allowed{0};
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kern), &allowed);
    if (e != cudaSuccess) return e;
    int64_t blocks = launch_device().sms;
    if (a.share_den > 1) blocks = blocks / a.share_den > 0 ? blocks / a.share_den : 1;
    if (a.max_ctas > 0 && blocks > a.max_ctas) blocks = a.max_ctas;
    // few subgrids: their tiles are shared out over the CTAs; see scout_role
    const int nseg = a.nr_subgrids >= blocks ? 0 : (int)(blocks / a.nr_subgrids < 16 ? blocks / a.nr_subgrids : 16);
    if (nseg > 0 && blocks > a.nr_subgrids * nseg) blocks = a.nr_subgrids * nseg;
    kern<<<(unsigned)blocks, kThreads, smem, stream>>>(a, nseg);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return launch_degridder_unfit(a, stream); // what the expansion does not hold for
}

} // namespace

bool degridder_tc_supported(int S, double image_size) {
    return S >= 8 && S <= 64 && S % 2 == 0 && tc_image_fits(image_size);
}

cudaError_t launch_degridder_tc(const KernelArgs &a, cudaStream_t stream) {
    const bool blocks = a.S > 32;
    switch (tc_shape(a.S).rows) {
    case 8: return launch<8, false>(a, stream); // S = 8
    case 12: return blocks ? launch<12, true>(a, stream) : launch<12, false>(a, stream);
    default: return blocks ? launch<16, true>(a, stream) : launch<16, false>(a, stream);
    }
}

} // namespace idg

// idg_gridder_tc.cu -- the gridder on the tensor cores.
//
// With the factors of idg_tc.cuh the sum over visibilities of a pixel is
//   G(x, y, p) = sum_v A_v(y, p) P_v(x),   A_v(y, p) = V_v(p) Q_v(y)  (+ first order),
// a matrix product of (row, polarisation) x visibilities with visibilities x
// columns; the per-pixel phase factor, A-terms and taper follow once per pixel.
//  * M = 128: (row, polarisation) of a block of at most 32 x 32 pixels.  A goes
//    into tensor memory, split into fp16 hi + lo.  A thread of a factor
//    warpgroup owns one row and, of every 16 visibilities, four: it forms their
//    y-factors once, uses them for the four polarisations and stores all of it
//    with the 16-lane store shape, so no y-factor is computed twice or exchanged.
//  * N = (re | im) x columns: cos and sin of the x-factors as fp16 in shared
//    memory.  Two operands, one for Re A with rows cos | sin and one for -Im A
//    with rows sin | -cos, add up Re G and Im G side by side; each holds the
//    hi parts, the lo parts and the first-order rows d cx (-sin | cos) one
//    after the other, so that one product of N = 192 takes A's hi part to all
//    three, and a second of N = 64 its lo part to the hi rows.  Few large
//    products matter: a product costs its warp some 70 cycles to issue beside
//    the other warps' work.  The first-order sum's factor cx(y) is a factor of
//    the whole row and is applied when the sum is read.
//  * Visibilities come in chunks of 256, each scaled by a power of two to the
//    fp16 range, and go through in stages of 32.  Correlations far below the
//    others (cross-hands) have powers of their own, put in by the loading warps
//    only then: for every chunk it would cost the 4,416 subgrids 4 %, the check 1 %.
//    The tensor core truncates its accumulator after every product, so the
//    full-size and the small products have accumulators of their own and after
//    each chunk their sum is added in fp32 to the block's sums in shared memory,
//    while the next chunk fills the other buffer.
//  * Roles: four factor warpgroups that take stages in turn, both operands of
//    one (an own half stage of A, an own stage of B each); a fifth for the sums
//    and the epilogue; two warps that bring in the chunks, one that issues the
//    products, one that looks for the next subgrid.
// One CTA of 24 warps per SM and all of its tensor memory.
// Measured on GB300, 4,416 subgrids of 128 x 16 visibilities at S = 32: 1.27 ms
// (41 SM cycles per visibility) against 5.02 ms for the mirror-quad kernel.  The
// products take 16 of those cycles.  The rest is the traffic of factors between
// the roles: with the factors' arithmetic left out, or the loads, or the stores,
// it stays near 30.  What helped: one warpgroup doing both operands of a stage
// (one barrier less per stage, and the row and column factors of a warpgroup
// overlap) in place of two for A and one for B, 1.31 against 1.37 ms, a fourth
// such warpgroup, 1.26, and products issued by one thread inside one branch
// instead of a predicate on each.  The roles run five different loops on one SM,
// so these are kept small: with the half stages unrolled and two stages of
// x-factors at a time, the same work missed the instruction cache (1.47 ms).
// 28 subgrids of 64 x 16 in one call: 40 us against 213 us.
#include "idg_tc.cuh"
#include "idg_internal.h"

namespace idg {

namespace {

constexpr int kWorkers = 4; // factor warpgroups
constexpr int kThreads = (kWorkers + 1) * 128 + 4 * 32, kLoadThread = kThreads - 64;
constexpr int kChunk = 256, kStage = 32; // visibilities
constexpr float kShort = 512.f;          // visibilities of a subgrid whose checks take as long as its sums
constexpr uint32_t kColsD = 192, kColA = 384, kColsA = 32, kTmemCols = 512;
constexpr uint32_t kAccStride = 128 * 16 + 16; // one group of four columns of the sums, padded

// A subgrid block found by the scouting warp.
struct Item {
    int stop, s, row0, c0, nc, nvis, x0, y0;
    unsigned st1, st2;
    int aterm;
    TcSubgrid sg;
};

struct Chunk {
    int stop, stages, first, last;
    float scale, inv[4]; // per polarisation
    Item it;
};

struct Head {
    uint64_t a_full[kWorkers], a_free[kWorkers];
    uint64_t c_full[2], c_free[2]; // chunks
    uint64_t d_full[2], d_free[2]; // accumulators
    uint64_t item_full, item_free, drain;
    uint32_t tmem;
    TcWatch watch;
    int load_stop;
    unsigned scratch[kTcScratch];
    uint4 wmax[2][2]; // per polarisation
    Item item;
    Chunk chunk[2];
};

// What a chunk's stages read: visibilities by polarisation and part, slopes.
struct ChunkData {
    float v[8][kChunk];
    float ah[kChunk], al[kChunk], bh[kChunk], bl[kChunk], d[kChunk];
};

struct Shape {
    int nb, bs; // blocks per axis, pixels per block (even)
};
__host__ __device__ inline Shape tc_shape(int S) {
    Shape s;
    s.nb = S > 32 ? 2 : 1;
    s.bs = s.nb == 1 ? S : 2 * ((S + 3) / 4);
    return s;
}

// XR: columns per block, rounded up to 16, 24 or 32.
template <int XR>
struct Op { // one stage of B
    static constexpr uint32_t ks = 12 * XR * 16; // bytes between 8-wide k groups: rows for Re A, then for -Im A
    static constexpr uint32_t bytes = 4 * ks;
};

struct Layout {
    size_t b, data, acc, axis, ntab, total;
};
template <int XR>
__host__ __device__ inline Layout tc_layout(int S) {
    const Shape s = tc_shape(S);
    Layout L;
    size_t off = (sizeof(Head) + 127) & ~size_t(127);
    L.b = off;    off += (size_t)kWorkers * Op<XR>::bytes;
    L.data = off; off += 2 * sizeof(ChunkData);
    L.acc = off;  off += (size_t)(2 * XR / 4) * kAccStride;
    L.axis = off; off += (size_t)(s.nb * s.bs / 2 + 16) * 32;
    L.ntab = off; off += (size_t)(S / 2) * (S / 2) * 8;
    L.total = off;
    return L;
}

__device__ __forceinline__ void load_sync() { named_sync<1, 64>(); }

// The subgrid of a claim.  More items than CTAs go longest first, or a long one
// claimed late would be all that runs at the end.  A work list is in that order
// already and is taken as it is; otherwise not by a sort, but the warp
// ranks 32 neighbours by their visibilities, and the claims take the longest of
// every 32 first, then the second longest of every 32, and so on.  From the
// first short one on, a claim and its neighbours' lengths are asked for while the
// previous item is checked: there the scout is what the others wait for.  (With
// long ones that would bind work to an SM too early.)  Gridding steps: 2,500
// subgrids of 128 to 16,384 visibilities at S = 24 1.26 ms in the plan's order, 0.95
// this way and 0.93 by a sorted list (1.29 when that was ranked once more, which
// made 32 sweeps of it), 600 at S = 32 0.64 to 0.72, 0.43 and 0.44; groups of 8
// instead of 32: 1.02 and 0.53.  4,416 subgrids of 128 visibilities pay 4 of 178 us
// for it, even ones being told apart from others by one vote.
struct Claim {
    int item, s, rank;  // work item; on each lane a neighbour of its subgrid (ranked), or that subgrid
    float length;       // the neighbour's visibilities; -1: none
};
__device__ __forceinline__ float length_of(const KernelArgs &a, int s) {
    const int nc = a.ext ? a.ext[s].channel_end - a.ext[s].channel_begin : a.C;
    return (float)max(a.md[s].nr_timesteps, 0) * (float)max(nc, 0);
}
__device__ __forceinline__ Claim look_up(const KernelArgs &a, int item, int nblocks, bool many, bool ranked) {
    Claim c{item, 0, 0, -1.f};
    const int idx = item / nblocks, n = (int)a.nr_subgrids;
    if (idx >= n) return c;
    if (!ranked) {
        c.s = a.work_list ? a.work_list[idx] : idx;
        if (many) c.length = length_of(a, c.s);
        return c;
    }
    const int groups = (n + 31) / 32, last = n - 32 * (groups - 1); // the last group has no ranks from `last` on
    const int late = idx - last * groups;
    c.rank = late < 0 ? idx / groups : last + late / (groups - 1);
    const int group = late < 0 ? idx - c.rank * groups : late - (c.rank - last) * (groups - 1);
    const int i = 32 * group + (int)(threadIdx.x & 31);
    if (i < n) {
        c.s = i;
        c.length = length_of(a, i);
    }
    return c;
}
__device__ __forceinline__ int subgrid_of(const Claim &c, bool ranked, float *length) {
    *length = c.length;
    if (!ranked) return c.s;
    const float first = __shfl_sync(0xffffffffu, c.length, 0);
    int who = c.rank;
    if (!__all_sync(0xffffffffu, c.length < 0.f || c.length == first)) {
        const int lane = threadIdx.x & 31;
        int mine = 0;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const float other = __shfl_sync(0xffffffffu, c.length, j);
            mine += other > c.length || (other == c.length && j < lane);
        }
        who = __ffs((int)__ballot_sync(0xffffffffu, mine == c.rank)) - 1;
    }
    *length = __shfl_sync(0xffffffffu, c.length, who);
    return __shfl_sync(0xffffffffu, c.s, who);
}

// Takes (subgrid, block) items from the work counter; leaves out what the
// expansion does not hold for.
__device__ __forceinline__ void scout_role(const KernelArgs &a, Head *head, const Shape &sh) {
    volatile TcWatch *watch = &head->watch;
    const int lane = threadIdx.x & 31, nblocks = sh.nb * sh.nb, S2 = a.S * a.S;
    const size_t jones = (size_t)S2 * 2;
    const bool many = a.nr_subgrids * nblocks > (int64_t)gridDim.x, ranked = many && !a.work_list;
    auto claim = [&] { return lane > 0 ? 0 : watch->abort ? INT32_MAX : atomicAdd(a.work_counter, 1); };
    auto look = [&](int c) { return look_up(a, __shfl_sync(0xffffffffu, c, 0), nblocks, many, ranked); };
    Claim next{};
    int ahead = 0;      // the claim after the next one
    bool eager = false; // down to the short ones
    for (uint32_t k = 0;;) {
        const Claim now = eager ? next : look(claim());
        if (lane == 0) watch->looked = global_timer_ns();
        float length;
        const int item = now.item, s = subgrid_of(now, ranked, &length);
        if (many && (eager || length < kShort)) {
            next = look(eager ? ahead : claim());
            ahead = claim();
            eager = true;
        }
        Item it{};
        it.stop = item >= a.nr_subgrids * nblocks;
        if (!it.stop) {
            const int block = item % nblocks;
            const SubgridInfo si = load_subgrid(a, s);
            if (!si.ok) {
                if (lane == 0) flag_status(a.status, kStatusBadPlan);
                if (block == 0)
                    for (int i = lane; i < 4 * S2; i += 32) a.subgrids[(size_t)s * 4 * S2 + i] = make_float2(0.f, 0.f);
                continue;
            }
            if (!tc_fits<32>(a, si, head->scratch, &it.sg, [] { __syncwarp(); })) {
                if (lane == 0) atomicAdd(a.fallback, 1);
                continue;
            }
            const char *j1 = reinterpret_cast<const char *>(a.aterms + ((size_t)si.aterm * a.nr_stations + si.st1) * jones);
            const char *j2 = reinterpret_cast<const char *>(a.aterms + ((size_t)si.aterm * a.nr_stations + si.st2) * jones);
            for (size_t o = (size_t)lane * 128; o < jones * 16; o += 32 * 128) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(j1 + o));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(j2 + o));
            }
            it.s = s;
            it.row0 = si.row0;
            it.c0 = si.c0;
            it.nc = si.c1 - si.c0;
            it.nvis = si.T * it.nc; // tc_fits bounds it, and it is not zero
            it.x0 = (block % sh.nb) * sh.bs;
            it.y0 = (block / sh.nb) * sh.bs;
            it.st1 = si.st1;
            it.st2 = si.st2;
            it.aterm = si.aterm;
        }
        if (k > 0) tc_wait(&head->item_free, (k - 1) & 1, watch, a.status);
        // a wait that was given up leaves the item to those who may be reading it
        if (__any_sync(0xffffffffu, watch->abort)) return;
        if (lane == 0) {
            head->item = it;
            mbar_arrive(&head->item_full);
        }
        ++k;
        if (it.stop) return;
    }
}

// The raw inputs of one visibility.
struct Raw {
    float4 v0, v1;
    float u, v, w, k;
};
__device__ __forceinline__ Raw load_raw(const KernelArgs &a, const Item &it, int i) {
    Raw r;
    const int j = min(i, it.nvis - 1);
    const int t = j / it.nc, c = it.c0 + j - t * it.nc;
    const float4 *src = a.vis + (((int64_t)it.row0 + t) * a.C + c) * 2;
    r.v0 = r.v1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < it.nvis) {
        r.v0 = src[0];
        r.v1 = src[1];
    }
    const float *p = a.uvw + 3 * ((int64_t)it.row0 + t);
    r.u = p[0];
    r.v = p[1];
    r.w = p[2];
    r.k = a.wavenumbers[c];
    return r;
}

// x-factors of one stage: thread (x = lane, eight visibilities of warp w).
template <int XR>
__device__ __forceinline__ void make_b(unsigned char *slot, const ChunkData &cd, int v0, f2 H, f2 F, f2 CX, bool cross,
                                       int lane, int w) {
    uint32_t ch[4], cl[4], sh[4], sl[4], c1[4], s1[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float4 hi = *reinterpret_cast<const float4 *>(&cd.ah[v0 + 4 * q]);
        const float4 lo = *reinterpret_cast<const float4 *>(&cd.al[v0 + 4 * q]);
        const float4 d = *reinterpret_cast<const float4 *>(&cd.d[v0 + 4 * q]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * q + e;
            const f2 D = e ? pack2(d.z, d.w) : pack2(d.x, d.y);
            f2 c, s;
            tc_sincos(e ? pack2(hi.z, hi.w) : pack2(hi.x, hi.y), e ? pack2(lo.z, lo.w) : pack2(lo.x, lo.y), D, H, F, c,
                      s);
            tc_split(c, ch[i], cl[i]);
            tc_split(s, sh[i], sl[i]);
            if (cross) {
                const f2 x = fmul2(D, CX);
                c1[i] = tc_half2(fmul2(c, x));
                s1[i] = tc_half2(fmul2(s, x));
            }
        }
    }
    if (lane >= XR) return;
    const auto vec = [](const uint32_t (&r)[4], uint32_t flip) {
        return make_uint4(r[0] ^ flip, r[1] ^ flip, r[2] ^ flip, r[3] ^ flip);
    };
    constexpr uint32_t neg = 0x80008000u;
    uint4 *o = reinterpret_cast<uint4 *>(slot + (uint32_t)w * Op<XR>::ks + (uint32_t)lane * 16u);
    o[0] = vec(ch, 0u);
    o[XR] = o[6 * XR] = vec(sh, 0u);
    o[2 * XR] = vec(cl, 0u);
    o[3 * XR] = o[8 * XR] = vec(sl, 0u);
    o[7 * XR] = vec(ch, neg);
    o[9 * XR] = vec(cl, neg);
    if (cross) {
        o[4 * XR] = vec(s1, neg);
        o[5 * XR] = o[10 * XR] = vec(c1, 0u);
        o[11 * XR] = vec(s1, 0u);
    }
}

// Chunks (two warps; a thread takes two visibilities at a time).  The next
// inputs are on their way while these are made ready.
__device__ __forceinline__ void load_role(const KernelArgs &a, Head *head, const Layout &L, unsigned char *smem) {
    ChunkData *data = reinterpret_cast<ChunkData *>(smem + L.data);
    volatile TcWatch *watch = &head->watch;
    const int lane = (int)threadIdx.x - kLoadThread;
    uint32_t cn = 0; // chunks so far
    for (uint32_t k = 0;; ++k) {
        tc_wait(&head->item_full, k & 1, watch, a.status);
        load_sync();
        if (lane == 0) head->load_stop = head->item.stop || watch->abort; // one answer for all
        load_sync();
        const Item it = head->item;
        const bool stop = head->load_stop != 0;
        load_sync();
        mbar_arrive(&head->item_free);
        const int nchunks = stop ? 1 : (it.nvis + kChunk - 1) / kChunk;
        Raw r0{}, r1{};
        if (!stop) {
            r0 = load_raw(a, it, lane);
            r1 = load_raw(a, it, lane + 64);
        }
        for (int chunk = 0; chunk < nchunks; ++chunk, ++cn) {
            const uint32_t buf = cn & 1;
            const int v0 = chunk * kChunk, stages = stop ? 0 : (min(it.nvis - v0, kChunk) + kStage - 1) / kStage;
            if (cn >= 2) tc_wait(&head->c_free[buf], ((cn >> 1) - 1) & 1, watch, a.status);
            ChunkData &cd = data[buf];
            unsigned m[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
            for (int o = 0; o < stages * kStage; o += 64) {
                const Raw r = r0;
                const int n = o + lane;
                r0 = r1;
                if (v0 + o + 128 < it.nvis) r1 = load_raw(a, it, v0 + n + 128);
                const float v[8] = {r.v0.x, r.v0.y, r.v0.z, r.v0.w, r.v1.x, r.v1.y, r.v1.z, r.v1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    cd.v[i][n] = v[i];
                    m[i >> 1] = max(m[i >> 1], __float_as_uint(fabsf(v[i])));
                }
                const float ph = __fmul_rn(r.k, a.tc.d2h), pl = fmaf(r.k, a.tc.d2l, fmaf(r.k, a.tc.d2h, -ph));
                const float qh = __fmul_rn(r.k, a.tc.i2h), ql = fmaf(r.k, a.tc.i2l, fmaf(r.k, a.tc.i2h, -qh));
                float hi, lo;
                tc_slope(ph, pl, r.u, it.sg.xh, it.sg.xl, hi, lo);
                cd.ah[n] = hi;
                cd.al[n] = kTwoPiF * lo;
                tc_slope(ph, pl, r.v, it.sg.yh, it.sg.yl, hi, lo);
                cd.bh[n] = hi;
                cd.bl[n] = kTwoPiF * lo;
                cd.d[n] = kTwoPiF * tc_delta(qh, ql, r.w, it.sg.mid);
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) m[p] = __reduce_max_sync(0xffffffffu, m[p]);
            if ((lane & 31) == 0) head->wmax[buf][lane >> 5] = make_uint4(m[0], m[1], m[2], m[3]);
            load_sync();
            const uint4 o = head->wmax[buf][(lane >> 5) ^ 1];
            const unsigned w[4] = {max(m[0], o.x), max(m[1], o.y), max(m[2], o.z), max(m[3], o.w)};
            unsigned most = 0u, least = 0xffffffffu;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                most = max(most, w[p]);
                least = min(least, w[p] - 1u); // a correlation of zeros counts as large
            }
            // Down to 2^-12 of the largest a correlation's lo part keeps its bits under
            // one scale (fp16 goes down to 2^-24, 2^-36 of it).
            const bool own = most > least && most - least > (12u << 23);
            const auto of = [&](int p) { return p == 0 ? w[0] : p == 1 ? w[1] : p == 2 ? w[2] : w[3]; };
            if (own && 4 * lane < stages * kStage) {
#pragma unroll 1
                for (int i = 0; i < 8; ++i) {
                    float unused;
                    const float f = tc_scale(of(i >> 1), unused);
                    float4 &q = *reinterpret_cast<float4 *>(&cd.v[i][4 * lane]);
                    q = make_float4(q.x * f, q.y * f, q.z * f, q.w * f);
                }
            }
            Chunk &c = head->chunk[buf];
            if (lane < 4) {
                float inv;
                const float scale = tc_scale(own ? of(lane) : most, inv);
                // the accumulator is truncated after each of 4 products per stage: see kTcTruncation
                c.inv[lane] = inv * (1.f + kTcTruncationPerStage * (float)stages);
                if (lane == 0) c.scale = own ? 1.f : scale;
            }
            if (lane == 32) {
                c.stop = stop;
                c.stages = stages;
                c.first = chunk == 0;
                c.last = chunk == nchunks - 1;
                c.it = it;
            }
            mbar_arrive(&head->c_full[buf]);
        }
        if (stop) return;
    }
}

__device__ __forceinline__ void tmem_st_16x256_x4(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]));
}
// A of 16 visibilities: thread (row of the block t / 4 + 8 w, visibilities
// 4 (t % 4) .. + 3).  Of the 16-lane store shape a thread holds lanes t / 4 and
// t / 4 + 8, columns 2 (t % 4) and + 1: two polarisations of its row, two pairs
// of visibilities; r[0] for polarisations 0, 1 (lanes 0 .. 15 of the warp's
// quarter), r[1] for 2, 3 (16 .. 31).  Columns: Re hi | Re lo | Im hi | Im lo,
// eight each.
__device__ __forceinline__ void make_a(uint32_t (&r)[2][16], const ChunkData &cd, int v0, f2 H, f2 F, f2 SC) {
    const float4 hi = *reinterpret_cast<const float4 *>(&cd.bh[v0]);
    const float4 lo = *reinterpret_cast<const float4 *>(&cd.bl[v0]);
    const float4 d = *reinterpret_cast<const float4 *>(&cd.d[v0]);
    f2 c[2], s[2], n[2];
    tc_sincos(pack2(hi.x, hi.y), pack2(lo.x, lo.y), pack2(d.x, d.y), H, F, c[0], s[0]);
    tc_sincos(pack2(hi.z, hi.w), pack2(lo.z, lo.w), pack2(d.z, d.w), H, F, c[1], s[1]);
#pragma unroll
    for (int b = 0; b < 2; ++b) { // the chunk's power of two goes in here
        c[b] = fmul2(c[b], SC);
        s[b] = fmul2(s[b], SC);
        n[b] = s[b] ^ 0x8000000080000000ull;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float4 vr = *reinterpret_cast<const float4 *>(&cd.v[2 * p][v0]);
        const float4 vi = *reinterpret_cast<const float4 *>(&cd.v[2 * p + 1][v0]);
        uint32_t(&o)[16] = r[p >> 1];
        const int e = 2 * (p & 1);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const f2 x = b ? pack2(vr.z, vr.w) : pack2(vr.x, vr.y), y = b ? pack2(vi.z, vi.w) : pack2(vi.x, vi.y);
            const f2 ar = ffma2(y, n[b], fmul2(x, c[b])), ai = ffma2(y, c[b], fmul2(x, s[b]));
            tc_split(ar, o[e + b], o[4 + e + b]);
            tc_split(ai, o[8 + e + b], o[12 + e + b]);
        }
    }
}

// Factor warpgroups: both factors of every kWorkers-th stage.
template <int XR>
__device__ __forceinline__ void factor_role(const KernelArgs &a, Head *head, const Layout &L, unsigned char *smem,
                                            uint32_t tl) {
    const float4 *axis = reinterpret_cast<const float4 *>(smem + L.axis);
    const ChunkData *data = reinterpret_cast<const ChunkData *>(smem + L.data);
    volatile TcWatch *watch = &head->watch;
    const int wg = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3, t = threadIdx.x & 31, row = 8 * warp + (t >> 2);
    uint32_t turn = (uint32_t)wg, uses = 0; // stages until this warpgroup's next one; those it has done
    for (uint32_t cn = 0;; ++cn) {
        const uint32_t buf = cn & 1;
        tc_wait(&head->c_full[buf], (cn >> 1) & 1, watch, a.status);
        __syncwarp();
        if (__any_sync(0xffffffffu, watch->abort)) return;
        const Chunk &c = head->chunk[buf];
        if (c.stop) return;
        const uint32_t stages = (uint32_t)c.stages;
        const int y = c.it.y0 + row, x0 = c.it.x0;
        const bool cross = c.it.sg.cross != 0;
        const float scale = c.scale;
        for (; turn < stages; turn += kWorkers, ++uses) {
            const int v0 = (int)turn * kStage;
            const float4 g = axis[2 * (y >> 1)];
            const float h = y & 1 ? g.y : g.x, f = y & 1 ? g.w : g.z;
#pragma unroll 1
            for (uint32_t kb = 0; kb < 2; ++kb) {
                uint32_t r[2][16];
                make_a(r, data[buf], v0 + 16 * (int)kb + 4 * (t & 3), pack2(h, h), pack2(f, f), pack2(scale, scale));
                // the products of this warpgroup's previous half stage, and all before it, have read A and B
                if (uses > 0 || kb > 0) tc_wait(&head->a_free[wg], (kb + 1) & 1, watch, a.status);
                __syncwarp();
                tmem_fence_after();
                tmem_st_16x256_x4(tl + kColA + kColsA * wg, r[0]);
                tmem_st_16x256_x4(tl + kColA + kColsA * wg + (16u << 16), r[1]);
                if (kb == 0) {
                    const float4 g0 = axis[x0 + 2 * (t >> 1)], g1 = axis[x0 + 2 * (t >> 1) + 1];
                    const float hx = t & 1 ? g0.y : g0.x, fx = t & 1 ? g0.w : g0.z, cx = t & 1 ? g1.y : g1.x;
                    make_b<XR>(smem + L.b + wg * Op<XR>::bytes, data[buf], v0 + 8 * warp, pack2(hx, hx), pack2(fx, fx),
                               pack2(cx, cx), cross, t, warp);
                    fence_proxy_async();
                }
                tmem_wait_st();
                tmem_fence_before();
                mbar_arrive(&head->a_full[wg]);
            }
        }
        turn -= stages;
        mbar_arrive(&head->c_free[buf]);
    }
}

// Sums and epilogue (one warpgroup; thread = lane of tensor memory).
template <int XR>
__device__ __forceinline__ void sum_role(const KernelArgs &a, Head *head, const Layout &L, unsigned char *smem,
                                         uint32_t tl, const Shape &sh) {
    const float2 *ntab = reinterpret_cast<const float2 *>(smem + L.ntab);
    const float4 *axis = reinterpret_cast<const float4 *>(smem + L.axis);
    volatile TcWatch *watch = &head->watch;
    const int lane = threadIdx.x & 127, w = lane >> 5, t = lane & 31;
    const int S = a.S, S2 = S * S, Sh = S / 2;
    unsigned char *acc = smem + L.acc;
    for (uint32_t cn = 0;; ++cn) {
        const uint32_t buf = cn & 1;
        tc_wait(&head->c_full[buf], (cn >> 1) & 1, watch, a.status);
        __syncwarp();
        if (__any_sync(0xffffffffu, watch->abort)) return;
        const Chunk c = head->chunk[buf];
        const float inv = head->chunk[buf].inv[t >> 3]; // of this lane of tensor memory
        mbar_arrive(&head->c_free[buf]);
        if (c.stop) return;
        tc_wait(&head->d_full[buf], (cn >> 1) & 1, watch, a.status);
        __syncwarp();
        tmem_fence_after();
        const f2 K = pack2(inv, inv);
        const bool cross = c.it.sg.cross != 0;
        const int row = c.it.y0 + 8 * w + (t & 7); // of this lane of tensor memory
        const float4 g1 = axis[2 * (row >> 1) + 1];
        const float cy = row & 1 ? g1.y : g1.x;
        const f2 CY = pack2(cy, cy);
#pragma unroll 1
        for (int g = 0; g < 2 * XR / 16; ++g) {
            f2 vh[8], vl[8];
            const uint32_t col = tl + kColsD * buf + 16 * g;
            tmem_ld16x2(col, col + 2 * XR, vh, vl);
#pragma unroll
            for (int q = 0; q < 8; ++q) vh[q] = fadd2(vh[q], vl[q]);
            if (cross) {
                tmem_ld16(col + 4 * XR, vl);
#pragma unroll
                for (int q = 0; q < 8; ++q) vh[q] = ffma2(vl[q], CY, vh[q]);
            }
            if (g == 2 * XR / 16 - 1) {
                tmem_fence_before();
                mbar_arrive(&head->d_free[buf]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ulonglong2 *p = reinterpret_cast<ulonglong2 *>(acc + (uint32_t)(4 * g + q) * kAccStride + lane * 16);
                const f2 s0 = vh[2 * q], s1 = vh[2 * q + 1];
                ulonglong2 o;
                if (c.first) {
                    o.x = fmul2(s0, K);
                    o.y = fmul2(s1, K);
                } else {
                    o = *p;
                    o.x = ffma2(s0, K, o.x);
                    o.y = ffma2(s1, K, o.y);
                }
                *p = o;
            }
        }
        if (!c.last) continue;

        // ---- epilogue: this warp's eight rows, lane = column
        __syncwarp();
        const bool taper = (a.flags & IDG_FLAG_NO_TAPER) == 0;
        const size_t jones = (size_t)S2 * 2;
        const float4 *a1 = a.aterms + ((size_t)c.it.aterm * a.nr_stations + c.it.st1) * jones;
        const float4 *a2 = a.aterms + ((size_t)c.it.aterm * a.nr_stations + c.it.st2) * jones;
        const int gx = c.it.x0 + t;
        const int rows = min(8, min(sh.bs, S - c.it.y0) - 8 * w);
        if (t < sh.bs && gx < S && rows > 0) {
            const int q0 = (c.it.y0 + 8 * w) * S + gx;
            cf n1[4], n2[4]; // the next pixel's, on their way while this one is worked on
            load_jones(a1 + 2 * q0, n1);
            load_jones(a2 + 2 * q0, n2);
#pragma unroll 1
            for (int yy = 0; yy < rows; ++yy) {
                const int gy = c.it.y0 + 8 * w + yy, q = q0 + yy * S, nq = q0 + min(yy + 1, rows - 1) * S;
                cf j1[4], j2[4], px[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    j1[p] = n1[p];
                    j2[p] = n2[p];
                }
                load_jones(a1 + 2 * nq, n1);
                load_jones(a2 + 2 * nq, n2);
                const float2 n = ntab[(gy < Sh ? gy : S - 1 - gy) * Sh + (gx < Sh ? gx : S - 1 - gx)];
                const cf f = cscale(tc_pixel_factor(c.it.sg.g0h, c.it.sg.g0l, n), taper ? a.taper[q] : 1.f);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const uint32_t o = (uint32_t)(32 * w + 8 * p + yy) * 16u;
                    const uint32_t ci = (uint32_t)(XR + t);
                    px[p].re = *reinterpret_cast<const float *>(acc + (uint32_t)(t >> 2) * kAccStride + o + (t & 3) * 4);
                    px[p].im = *reinterpret_cast<const float *>(acc + (ci >> 2) * kAccStride + o + (ci & 3u) * 4u);
                }
                aterm_gridder(px, j1, j2);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const cf v = cmul(f, px[p]);
                    a.subgrids[((size_t)c.it.s * 4 + p) * S2 + q] = make_float2(v.re, v.im);
                }
            }
        }
        __syncwarp();
    }
}

// The products of 16 visibilities (one thread).
template <int XR, bool CROSS>
__device__ __forceinline__ void issue_step(uint32_t d, uint32_t c, uint32_t k, uint32_t acc) {
    constexpr uint32_t hi = umma_desc_hi(128);
    constexpr uint32_t id = umma_idesc_f16(128, (CROSS ? 6 : 4) * XR), idl = umma_idesc_f16(128, 2 * XR);
    umma_f16_ts_if<id, hi>(d, c, k, acc);
    umma_f16_ts<true, (id | kUmmaNegateA), hi>(d, c + 16, k + 6 * XR);
    umma_f16_ts<true, idl, hi>(d + 2 * XR, c + 8, k);
    umma_f16_ts<true, (idl | kUmmaNegateA), hi>(d + 2 * XR, c + 24, k + 6 * XR);
}

// The stages of one chunk: the warpgroups' first half stages, then their second
// ones, so that each is formed while the others' are multiplied.  gs: stages
// before this chunk; c0, b0: the warpgroups' first A columns and B descriptor.
template <int XR, bool CROSS>
__device__ __forceinline__ void issue_chunk(const KernelArgs &a, Head *head, uint32_t d, uint32_t c0, uint32_t b0,
                                            uint32_t gs, int stages, uint32_t lead) {
    volatile TcWatch *watch = &head->watch;
    uint32_t acc = 0;
    for (int st = 0; st < stages; st += kWorkers, gs += kWorkers) {
        const uint32_t n = (uint32_t)min(kWorkers, stages - st);
#pragma unroll 1
        for (uint32_t kb = 0; kb < 2; ++kb) {
            uint32_t w = gs % kWorkers;
#pragma unroll 1
            for (uint32_t i = 0; i < n; ++i) {
                tc_wait(&head->a_full[w], kb, watch, a.status); // with kb = 0, B too
                tmem_fence_after();
                if (lead) {
                    issue_step<XR, CROSS>(d, c0 + kColsA * w,
                                          b0 + (Op<XR>::bytes >> 4) * w + ((2 * Op<XR>::ks) >> 4) * kb, acc);
                    umma_commit(&head->a_free[w]);
                }
                __syncwarp();
                acc = 1;
                w = w + 1 == kWorkers ? 0 : w + 1;
            }
        }
    }
}

template <int XR>
__device__ __forceinline__ void issue_role(const KernelArgs &a, Head *head, const Layout &L, unsigned char *smem,
                                           uint32_t tm) {
    volatile TcWatch *watch = &head->watch;
    const uint32_t lead = elect_lane();
    const uint32_t t0 = warp_uniform(tm), b0 = warp_uniform(umma_desc_lo(smem_addr(smem + L.b), Op<XR>::ks));
    uint32_t gs = 0;
    for (uint32_t cn = 0;; ++cn) {
        const uint32_t buf = cn & 1;
        tc_wait(&head->c_full[buf], (cn >> 1) & 1, watch, a.status);
        __syncwarp();
        if (__any_sync(0xffffffffu, watch->abort)) break;
        const bool stop = warp_uniform(head->chunk[buf].stop) != 0, cross = warp_uniform(head->chunk[buf].it.sg.cross) != 0;
        const int stages = (int)warp_uniform(head->chunk[buf].stages);
        mbar_arrive(&head->c_free[buf]);
        if (stop) break;
        if (cn >= 2) tc_wait(&head->d_free[buf], ((cn >> 1) - 1) & 1, watch, a.status);
        __syncwarp();
        if (cross)
            issue_chunk<XR, true>(a, head, t0 + kColsD * buf, t0 + kColA, b0, gs, stages, lead);
        else
            issue_chunk<XR, false>(a, head, t0 + kColsD * buf, t0 + kColA, b0, gs, stages, lead);
        gs += (uint32_t)stages;
        if (lead) umma_commit(&head->d_full[buf]);
        __syncwarp();
    }
    if (lead && gs > 0) { // products in flight end (bounded) before their memory goes, also where a reader gave up
        umma_commit(&head->drain);
        mbar_wait_bounded(&head->drain, 0, kTcWaitNs);
    }
    __syncwarp();
}

template <int XR>
__global__ void __launch_bounds__(kThreads, 1) gridder_tc_kernel(KernelArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const Shape sh = tc_shape(a.S);
    const Layout L = tc_layout<XR>(a.S);
    Head *head = reinterpret_cast<Head *>(smem);
    const int tid = threadIdx.x, warp = tid >> 5;

    constexpr int kSum = 4 * kWorkers, kIssue = kSum + 4; // first warps of the roles behind the factor warpgroups
    if (warp == kIssue) {
        tmem_alloc(&head->tmem, kTmemCols);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < kWorkers; ++i) {
            mbar_init(&head->a_full[i], 128);
            mbar_init(&head->a_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&head->c_full[i], 64);
            mbar_init(&head->c_free[i], 128 * kWorkers + 128 + 32);
            mbar_init(&head->d_full[i], 1);
            mbar_init(&head->d_free[i], 128);
        }
        mbar_init(&head->item_full, 1);
        mbar_init(&head->item_free, 64);
        mbar_init(&head->drain, 1);
        mbar_init_fence();
        head->watch = TcWatch{0, 0};
    }
    tc_axis_table(a, reinterpret_cast<float4 *>(smem + L.axis), sh.nb * sh.bs / 2 + 16, tid, kThreads);
    tc_n_table(a, reinterpret_cast<float2 *>(smem + L.ntab), tid, kThreads);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tm = head->tmem;
    const uint32_t tl = tm + ((uint32_t)(warp & 3) << 21); // this warp's lane quarter

    if (warp < kSum)
        factor_role<XR>(a, head, L, smem, tl);
    else if (warp < kIssue)
        sum_role<XR>(a, head, L, smem, tl, sh);
    else if (warp == kIssue)
        issue_role<XR>(a, head, L, smem, tm);
    else if (warp == kIssue + 1)
        scout_role(a, head, sh);
    else
        load_role(a, head, L, smem);
    __syncthreads();
    if (warp == kIssue) tmem_free(tm, kTmemCols);
}

template <int XR>
cudaError_t launch(const KernelArgs &args, cudaStream_t stream, bool load_only) {
    auto kern = gridder_tc_kernel<XR>;
    if (load_only) {
        cudaFuncAttributes fa;
        return cudaFuncGetAttributes(&fa, kern);
    }
    KernelArgs a = args;
    a.tc = tc_const(a.S, a.image_size);
    const size_t smem = tc_layout<XR>(a.S).total;
    static std::atomic<uint64_t> allowed{0};
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kern), &allowed);
    if (e != cudaSuccess) return e;
    int64_t blocks = launch_device().sms;
    if (a.share_den > 1) blocks = blocks / a.share_den > 0 ? blocks / a.share_den : 1;
    if (a.max_ctas > 0 && blocks > a.max_ctas) blocks = a.max_ctas;
    const Shape sh = tc_shape(a.S);
    if (blocks > a.nr_subgrids * sh.nb * sh.nb) blocks = a.nr_subgrids * sh.nb * sh.nb;
    kern<<<(unsigned)blocks, kThreads, smem, stream>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return launch_gridder_unfit(a, stream, false); // what the expansion does not hold for
}

cudaError_t dispatch(const KernelArgs &a, cudaStream_t stream, bool load_only) {
    const int bs = tc_shape(a.S).bs;
    if (bs <= 16) return launch<16>(a, stream, load_only);
    if (bs <= 24) return launch<24>(a, stream, load_only);
    return launch<32>(a, stream, load_only);
}

} // namespace

bool gridder_tc_supported(int S, double image_size) {
    return S >= 8 && S <= 64 && S % 2 == 0 && tc_image_fits(image_size);
}

cudaError_t launch_gridder_tc(const KernelArgs &a, cudaStream_t stream) { return dispatch(a, stream, false); }

cudaError_t load_gridder_tc() {
    KernelArgs a{};
    for (int S : {16, 24, 32}) {
        a.S = S;
        if (cudaError_t e = dispatch(a, nullptr, true)) return e;
    }
    return launch_gridder_unfit(a, nullptr, true);
}

} // namespace idg

// idg_tiles.cu -- the adder with a fixed summation order ("tile bins").
//
// The adder's job is grid[z][pol][y0+j][x0+i] += F[s][pol][j][i] over all
// subgrids s (with the Hermitian mirror for -W <= z < 0; see idg_adder.cu).
// Footprints overlap heavily -- consecutive time slices of a baseline land on
// nearly the same cells, and short baselines crowd the centre of the grid -- so
// idg_adder() accumulates with floating-point atomics, whose order (and so the
// last bits of the result) changes from run to run.  Here the order is fixed:
//
//  * On the host, once per plan, the subgrids are binned into tiles of 32 x 32
//    cells of their target plane (a counting sort in subgrid order, so each
//    tile's list is ascending).  Each list is cut into chunks of at most
//    kChunk subgrids.
//  * Pass 1, two CTAs per chunk: the chunk's plan entries are staged in shared
//    memory; every thread owns one cell of the tile (all four correlations) and
//    adds the chunk's subgrids into registers, in list order.  A tile with one
//    chunk is then added into the grid with plain loads and stores -- no other
//    CTA touches its cells; a tile with several chunks writes each chunk's sum
//    to a partial tile.
//  * Pass 2, one CTA per correlation of a tile with several chunks: grid +=
//    partial 0, then partial 1, ... in chunk order.
// No atomics; the result depends on the plan only.  Loads of a subgrid row
// coalesce across the warp (consecutive lanes, consecutive cells).  Cells that
// fall outside the grid and entries outside [-W, W) are skipped, as in
// idg_adder().
#include <algorithm>
#include <vector>

#include "idg_device.cuh"
#include "idg_host.h"
#include "idg_internal.h"
#include "idg_ptx.cuh"
#include "idg_tiles.h"

namespace idg {
namespace {

constexpr int kTile = 32;       // tile edge in cells (one warp lane per column)
constexpr int kWarps = 16;      // warps of a CTA, one row of a tile at a time
constexpr int kChunk = 128;     // subgrids per pass-1 work item (at most 256: their places are bytes)

// The chunk's plan entries (x, y, z, subgrid) are staged in shared memory
// first.  A footprint rarely fits a tile, so every tile an entry touches sees
// only part of it: a warp owns one row and first lists the entries that reach
// it, in order; the entry loop then issues predicated loads (columns outside an
// entry's footprint load nothing and add zero), kStep entries at a time, so
// that all their loads are in flight before any is added.  The adds stay in
// list order.  A work item takes two CTAs, one for either half of the rows.  The
// grid's cells are asked for before the entries, into shared memory: on a large grid
// a tile has two or three entries, and asked for last the cells were what it waited
// for (8,000 subgrids of 32^2 spread over 4096^2: 490 us, this way 330, with the
// cells in registers 353; over 2048^2 185, 136 and 144).
// Measured on GB300, 9,180 subgrids of 32^2 added to a cleared 2048^2 grid (20 us of
// clearing included): 105 us, where one CTA per item with every warp going
// through all entries, two rows 16 apart per thread, took 157 (73 % of the issue
// slots busy, half of them with cells outside the footprint); with two
// neighbouring rows per warp 115.  365 MB are read, 54 us at the copy rate; 412
// items of up to 128 entries are what is left for balance.
__global__ void __launch_bounds__(32 * kWarps, 2)
    tile_add_kernel(const TileItem *items, const int *entries, const idg_metadata *md, int S, int G, int ntx,
                    const float2 *subgrids, float2 *grid, float2 *partials) {
    constexpr int kStep = 4;
    __shared__ int4 smd[kChunk];
    __shared__ unsigned char listed[kWarps][kChunk];
    __shared__ float2 before[4][32 * kWarps]; // each thread's own cells
    const TileItem it = items[blockIdx.x >> 1];
    const int n = it.end - it.begin;
    for (int e = threadIdx.x; e < n; e += 32 * kWarps) {
        const int s = entries[it.begin + e];
        const idg_metadata m = md[s];
        smd[e] = make_int4(m.x, m.y, m.z, s);
    }
    const int per_plane = ntx * ntx;
    const int plane = it.tile / per_plane, r = it.tile - plane * per_plane, ty = r / ntx, tx = r - ty * ntx;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = kWarps * (blockIdx.x & 1) + warp;
    const int gx = tx * kTile + lane, gy = ty * kTile + row;
    const int S2 = S * S;
    const bool mine = gx < G && gy < G;
    float2 *cell = grid + (((int64_t)plane * 4) * G + gy) * G + gx;
    const int64_t next = (int64_t)G * G; // to the next correlation
    float2 acc[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        acc[p] = make_float2(0.f, 0.f);
        if (it.slot < 0 && mine) // on its way beside the entries, and in no registers
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(&before[p][threadIdx.x])),
                         "l"(cell + p * next)
                         : "memory");
    }
    __syncthreads();
    if (gy >= G) return;

    int nl = 0; // entries of this warp
    for (int e0 = 0; e0 < n; e0 += 32) {
        const int e = e0 + lane;
        bool hit = false;
        if (e < n) {
            const int4 m = smd[e];
            hit = (unsigned)(m.z < 0 ? G - gy - m.y : gy - m.y) < (unsigned)S;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (hit) listed[warp][nl + __popc(hits & ((1u << lane) - 1u))] = (unsigned char)e;
        nl += __popc(hits);
    }
    __syncwarp();

    for (int l = 0; l < nl; l += kStep) {
        float2 v[kStep][4];
        float sign[kStep];
#pragma unroll
        for (int h = 0; h < kStep; ++h) {
            const bool live = l + h < nl;
            const int4 m = smd[listed[warp][live ? l + h : l]];
            const bool mir = m.z < 0;
            sign[h] = mir ? -1.f : 1.f; // mirrored: conjugated
            const int i = mir ? G - gx - m.x : gx - m.x, j = mir ? G - gy - m.y : gy - m.y;
            const bool in = live && (unsigned)i < (unsigned)S && gx < G;
            // grid correlation p takes subgrid correlation p, or its swap when mirrored
            const int q1 = mir ? 2 * S2 : S2, q2 = 3 * S2 - q1;
            const float2 *src = subgrids + ((int64_t)m.w * 4 * S2 + (in ? j * S + i : 0));
#pragma unroll
            for (int p = 0; p < 4; ++p)
                v[h][p] = in ? __ldg(src + (p == 0 ? 0 : p == 1 ? q1 : p == 2 ? q2 : 3 * S2)) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < kStep; ++h)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                acc[p].x += v[h][p].x;
                acc[p].y = fmaf(sign[h], v[h][p].y, acc[p].y);
            }
    }

    if (gx >= G) return;
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        if (it.slot < 0) {
            const float2 g = before[p][threadIdx.x];
            cell[p * next] = make_float2(g.x + acc[p].x, g.y + acc[p].y);
        } else {
            partials[(((int64_t)it.slot * 4 + p) * kTile + row) * kTile + lane] = acc[p];
        }
    }
}

// One CTA per tile and correlation; four partial sums in flight.
__global__ void __launch_bounds__(kTile * kWarps)
    tile_combine_kernel(const TileMulti *multi, int G, int ntx, const float2 *partials, float2 *grid) {
    const TileMulti t = multi[blockIdx.x];
    const int p = blockIdx.y;
    const int per_plane = ntx * ntx;
    const int plane = t.tile / per_plane, r = t.tile - plane * per_plane, ty = r / ntx, tx = r - ty * ntx;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gx = tx * kTile + lane;
    if (gx >= G) return;
#pragma unroll
    for (int k = 0; k < kTile / kWarps; ++k) {
        const int row = warp + kWarps * k, gy = ty * kTile + row;
        if (gy >= G) continue;
        float2 *c = grid + (((int64_t)plane * 4 + p) * G + gy) * G + gx;
        const float2 *src = partials + (((int64_t)t.first_slot * 4 + p) * kTile + row) * kTile + lane;
        float2 g = *c;
#pragma unroll 4
        for (int q = 0; q < t.nslots; ++q) {
            const float2 v = src[(int64_t)q * 4 * kTile * kTile];
            g.x += v.x;
            g.y += v.y;
        }
        *c = g;
    }
}

// The footprint of entry m in grid cells of its target plane, [lo, hi) per
// axis after clipping to the grid; false when empty or outside [-W, W).
bool footprint(const idg_metadata &m, int S, int G, int W, int *plane, int *xlo, int *xhi, int *ylo, int *yhi) {
    if (m.z < -W || m.z >= W) return false;
    const bool mirror = m.z < 0;
    *plane = mirror ? -m.z - 1 : m.z;
    // direct: cells x .. x+S-1; mirrored: cells G-x-S+1 .. G-x
    const int64_t x0 = mirror ? (int64_t)G - m.x - S + 1 : m.x, y0 = mirror ? (int64_t)G - m.y - S + 1 : m.y;
    *xlo = (int)std::max<int64_t>(x0, 0);
    *xhi = (int)std::min<int64_t>(x0 + S, G);
    *ylo = (int)std::max<int64_t>(y0, 0);
    *yhi = (int)std::min<int64_t>(y0 + S, G);
    return *xlo < *xhi && *ylo < *yhi;
}

} // namespace

size_t TileBinsHost::partial_bytes() const { return (size_t)nslots * 4 * kTile * kTile * sizeof(float2); }

int bin_tiles(const idg_params *params, int64_t nr_subgrids, const idg_metadata *metadata, TileBinsHost *out) {
    const int S = params->subgrid_size, G = params->grid_size, W = params->nr_w_planes > 0 ? params->nr_w_planes : 1;
    const int ntx = (G + kTile - 1) / kTile;
    const int64_t per_plane = (int64_t)ntx * ntx, ntiles = per_plane * W;
    if (ntiles > INT32_MAX) return fail(IDG_ERR_UNSUPPORTED, "grid of %d planes of %d^2 cells has too many tiles", W, G);
    // counting sort of (tile, subgrid) pairs by tile, in subgrid order
    std::vector<int64_t> count(ntiles, 0);
    auto each_tile = [&](int64_t s, auto &&fn) {
        int pl, xlo, xhi, ylo, yhi;
        if (!footprint(metadata[s], S, G, W, &pl, &xlo, &xhi, &ylo, &yhi)) return;
        for (int ty = ylo / kTile; ty <= (yhi - 1) / kTile; ++ty)
            for (int tx = xlo / kTile; tx <= (xhi - 1) / kTile; ++tx) fn(pl * per_plane + (int64_t)ty * ntx + tx);
    };
    for (int64_t s = 0; s < nr_subgrids; ++s) each_tile(s, [&](int64_t t) { ++count[t]; });
    std::vector<int64_t> offset(ntiles + 1, 0);
    for (int64_t t = 0; t < ntiles; ++t) offset[t + 1] = offset[t] + count[t];
    const int64_t nentries = offset[ntiles];
    if (nentries > INT32_MAX)
        return fail(IDG_ERR_UNSUPPORTED, "%lld (tile, subgrid) pairs: too many for one bin set", (long long)nentries);
    TileBinsHost &b = *out;
    b = TileBinsHost{};
    b.S = S;
    b.G = G;
    b.W = W;
    b.ntx = ntx;
    b.entries.assign(std::max<int64_t>(nentries, 1), 0);
    std::vector<int64_t> fill(offset.begin(), offset.end() - 1);
    for (int64_t s = 0; s < nr_subgrids; ++s) each_tile(s, [&](int64_t t) { b.entries[fill[t]++] = (int)s; });
    for (int64_t t = 0; t < ntiles; ++t) {
        const int64_t n = count[t];
        if (n == 0) continue;
        const int64_t nch = (n + kChunk - 1) / kChunk;
        if (nch == 1) {
            b.items.push_back({(int)t, (int)offset[t], (int)(offset[t] + n), -1});
            continue;
        }
        b.multi.push_back({(int)t, b.nslots, (int)nch, 0});
        for (int64_t c = 0; c < nch; ++c) {
            const int64_t lo = offset[t] + c * kChunk, hi = std::min(offset[t] + n, lo + kChunk);
            b.items.push_back({(int)t, (int)lo, (int)hi, b.nslots++});
        }
    }
    // longest work items first, so that the short ones fill in at the end
    std::stable_sort(b.items.begin(), b.items.end(),
                     [](const TileItem &x, const TileItem &y) { return x.end - x.begin > y.end - y.begin; });
    return IDG_OK;
}

cudaError_t launch_binned_adder(const TileBinsDev &b, const float2 *subgrids, float2 *grid, cudaStream_t stream) {
    if (b.nitems > 0) {
        tile_add_kernel<<<2u * (unsigned)b.nitems, 32 * kWarps, 0, stream>>>(b.items, b.entries, b.md, b.S, b.G, b.ntx,
                                                                         subgrids, grid, b.partials);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (b.nmulti > 0) {
        tile_combine_kernel<<<dim3((unsigned)b.nmulti, 4), kTile * kWarps, 0, stream>>>(b.multi, b.G, b.ntx, b.partials, grid);
        return cudaGetLastError();
    }
    return cudaSuccess;
}

} // namespace idg

// Bins on the device: the public handle owns the device copies.
struct idg_tile_bins {
    int device = 0;
    int64_t nr_subgrids = 0;
    int64_t info[4] = {0, 0, 0, 0};
    void *mem = nullptr; // metadata, entries, items, multi, partial tiles (one allocation)
    idg::TileBinsDev dev;
};

namespace idg {

// One device allocation holding the plan's metadata and its bins (256-byte
// aligned parts); `mem` receives it, `view` points into it.
int upload_tile_bins(const TileBinsHost &h, int64_t nr_subgrids, const idg_metadata *metadata, void **mem,
                     TileBinsDev *view) {
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t b_md = up(sizeof(idg_metadata) * std::max<int64_t>(nr_subgrids, 1)),
                 b_en = up(sizeof(int) * h.entries.size()),
                 b_it = up(sizeof(TileItem) * std::max<size_t>(h.items.size(), 1)),
                 b_mu = up(sizeof(TileMulti) * std::max<size_t>(h.multi.size(), 1)), b_pa = up(h.partial_bytes());
    char *base = nullptr;
    IDG_CUDA(cudaMalloc(reinterpret_cast<void **>(&base), b_md + b_en + b_it + b_mu + b_pa));
    TileBinsDev &v = *view;
    v.md = reinterpret_cast<const idg_metadata *>(base);
    v.entries = reinterpret_cast<const int *>(base + b_md);
    v.items = reinterpret_cast<const TileItem *>(base + b_md + b_en);
    v.multi = reinterpret_cast<const TileMulti *>(base + b_md + b_en + b_it);
    v.partials = h.nslots ? reinterpret_cast<float2 *>(base + b_md + b_en + b_it + b_mu) : nullptr;
    v.S = h.S;
    v.G = h.G;
    v.ntx = h.ntx;
    v.nitems = (int)h.items.size();
    v.nmulti = (int)h.multi.size();
    cudaError_t e = cudaSuccess;
    if (nr_subgrids > 0)
        e = cudaMemcpy(base, metadata, sizeof(idg_metadata) * nr_subgrids, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(base + b_md, h.entries.data(), sizeof(int) * h.entries.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !h.items.empty())
        e = cudaMemcpy(base + b_md + b_en, h.items.data(), sizeof(TileItem) * h.items.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !h.multi.empty())
        e = cudaMemcpy(base + b_md + b_en + b_it, h.multi.data(), sizeof(TileMulti) * h.multi.size(),
                       cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(base);
        return cuda_fail(e, "tile bins upload");
    }
    *mem = base;
    return IDG_OK;
}

} // namespace idg

extern "C" {

IDG_API int idg_tile_bins_create(const idg_params *params, int64_t nr_subgrids, const idg_metadata *metadata,
                                 idg_tile_bins **bins) {
    using namespace idg;
    if (!bins) return fail(IDG_ERR_INVALID_ARGUMENT, "bins output is NULL");
    *bins = nullptr;
    if (!params) return fail(IDG_ERR_INVALID_ARGUMENT, "params is NULL");
    if (params->subgrid_size < 1 || params->grid_size < 1) return fail(IDG_ERR_INVALID_ARGUMENT, "bad sizes");
    if (nr_subgrids < 0 || nr_subgrids > INT32_MAX) return fail(IDG_ERR_INVALID_ARGUMENT, "nr_subgrids");
    if (nr_subgrids > 0 && !metadata) return fail(IDG_ERR_INVALID_ARGUMENT, "metadata is NULL");
    TileBinsHost h;
    if (int rc = bin_tiles(params, nr_subgrids, metadata, &h)) return rc;
    auto *b = new idg_tile_bins;
    cudaGetDevice(&b->device);
    b->nr_subgrids = nr_subgrids;
    b->info[0] = (int64_t)h.items.size();
    b->info[1] = (int64_t)h.multi.size();
    b->info[2] = h.nslots;
    b->info[3] = (int64_t)h.partial_bytes();
    if (int rc = upload_tile_bins(h, nr_subgrids, metadata, &b->mem, &b->dev)) {
        delete b;
        return rc;
    }
    *bins = b;
    return IDG_OK;
}

IDG_API int idg_tile_bins_destroy(idg_tile_bins *bins) {
    if (!bins) return IDG_OK;
    if (bins->mem) cudaFree(bins->mem);
    delete bins;
    return IDG_OK;
}

IDG_API int idg_tile_bins_info(const idg_tile_bins *bins, int64_t *sizes) {
    using namespace idg;
    if (!bins || !sizes) return fail(IDG_ERR_INVALID_ARGUMENT, "NULL argument");
    for (int i = 0; i < 4; ++i) sizes[i] = bins->info[i];
    return IDG_OK;
}

IDG_API int idg_adder_binned(const idg_tile_bins *bins, const void *subgrids, void *grid, void *stream) {
    using namespace idg;
    if (!bins) return fail(IDG_ERR_INVALID_ARGUMENT, "bins is NULL");
    if (bins->nr_subgrids == 0) return IDG_OK;
    if (!subgrids || !grid) return fail(IDG_ERR_INVALID_ARGUMENT, "NULL device pointer");
    int dev = 0;
    IDG_CUDA(cudaGetDevice(&dev));
    if (dev != bins->device)
        return fail(IDG_ERR_INVALID_ARGUMENT, "bins belong to device %d, current is %d", bins->device, dev);
    cudaError_t e = launch_binned_adder(bins->dev, reinterpret_cast<const float2 *>(subgrids),
                                        reinterpret_cast<float2 *>(grid), reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return cuda_fail(e, "binned adder launch");
    return IDG_OK;
}

} // extern "C"

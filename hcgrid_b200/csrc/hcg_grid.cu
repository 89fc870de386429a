// Gather gridding on the device (replaces the `hcgrid` kernel,
// HCGrid/gridding.cu:277-403, and the host normalisation,
// HCGrid/gmap.cpp:306-312).
//
// Selection follows the reference exactly: per target pixel the ring range
// [uring, dring] from the disc around its centre, per ring the HEALPix pixel
// window [lpix, rpix] at phi -/+ disc_size (not scaled by 1/cos(dec)), the
// polar whole-ring rule, the first-used-ring skip of the reference's search
// (start_int - 1 underflow) and a strict distance < sphere_radius cutoff.
// Rings whose window edge falls outside the ring -- where the reference's
// loop would never advance -- are skipped and counted instead.
//
// Geometry (ring windows, great-circle distance, cutoff, Gaussian weight)
// is FP64. Channel sums are FP32 (multi-channel) or FP64 (single channel);
// weight sums are FP64.
//
// Kernels
//   k_pixel_prep     per pixel: ring range and the phi half of loc2pix
//   k_grid_1chan     one warp per 2x2 pixel group, candidates spread over
//                    lanes, FP64
//   k_tile_rings     one block per 16x8-pixel tile: windows, the tile's union,
//                    candidate counts and entry offsets
//   k_group          one block (or a half, a quarter) per tile, a warp per 2x2
//                    group in turn: FP64 weights written as compact
//                    (sample, w[4]) entries
//   k_group_accum    one warp per group: FP32 channel accumulation from the
//                    entries, 4 channels per lane, normalised on store
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "hcg_internal.h"
#include "hcg_kernels.cuh"
#include "hcg_wcs.cuh"

namespace hcg {
namespace {

// ---------------------------------------------------------------------------
// Single-job kernels: one launch per phase, thread/warp/block indices map
// directly onto pixels, groups and tiles.

__global__ void k_pixel_prep(HpxParams h, uint64_t firstring, uint64_t usedrings, double disc, uint64_t npixmap,
                             const double *__restrict__ X, const double *__restrict__ Y, PixPrep *__restrict__ out,
                             DevStats *stats) {
    uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p < npixmap) prep_item(h, firstring, usedrings, disc, X, Y, out, stats, p);
}

template <int MODE, bool TABLES>  // as pair_weights, group_windows_any
__global__ void __launch_bounds__(kGroupThreads, MODE >= kPairEllipse ? 4 : kGroupCtas) k_grid_1chan(const __grid_constant__ GridArgs a, uint32_t nx, uint32_t ny, uint64_t ngroups,
                                                        const float *__restrict__ data, uint32_t cstride,
                                                        float *__restrict__ out, float *__restrict__ wout) {
    __shared__ GroupShared S[kGroupWarps];
    PairCounts pc;
    const int warp = threadIdx.x >> 5;
    constexpr int kGroups = kGroupWarps / kGrid1Parts<MODE>;  // of a block
    const uint64_t grp = blockIdx.x * (uint64_t)kGroups + warp % kGroups;
    if (grp < ngroups) grid1_item<MODE, TABLES>(a, nx, ny, data, cstride, out, wout, grp, S[warp], pc);
    flush_counts(pc, a.stats);
}

// The weight pass, a block per 16x8-pixel tile. MODE as pair_weights; PACK:
// entries as 16-bit hi/lo pairs for the tensor-core builders (1) or as FP32
// weights (0)
template <int MODE, int PACK>
__global__ void __launch_bounds__(kWeightThreads, MODE == kPairUnit ? kWeightCtas : 4)
    k_group(const __grid_constant__ GridArgs a, GroupArgs g, const unsigned long long *__restrict__ off, uint32_t *__restrict__ e_idx,
            float4 *__restrict__ e_w, uint32_t *__restrict__ cnt, double *__restrict__ wsum, TileArgs tiles, bool tiled) {
    __shared__ TileGroupShared S;
    PairCounts pc;
    group_tile_item<MODE, PACK>(a, g, off, e_idx, e_w, cnt, wsum, tiles, tiled, tiles.t0 + blockIdx.x, blockIdx.y,
                                gridDim.y, S, pc);
    flush_counts(pc, a.stats);
}

// Candidate counts of the groups whose tile's ring span exceeds the tile table.
__global__ void __launch_bounds__(kGroupThreads) k_group_count(const __grid_constant__ GridArgs a, GroupArgs g, uint32_t *__restrict__ cap) {
    __shared__ GroupShared S[kGroupWarps];
    const int warp = threadIdx.x >> 5;
    for (uint64_t grp = blockIdx.x * (uint64_t)kGroupWarps + warp; grp < g.ngroups; grp += gridDim.x * (uint64_t)kGroupWarps)
        group_count_item(a, g, cap, grp, S[warp]);
}

__global__ void __launch_bounds__(256) k_group_accum(GroupArgs g, const unsigned long long *__restrict__ off,
                                                     const uint32_t *__restrict__ cnt,
                                                     const uint32_t *__restrict__ e_idx,
                                                     const float4 *__restrict__ e_w, const double *__restrict__ wsum,
                                                     const float *__restrict__ spec, uint32_t nchan,
                                                     uint32_t cstride, float *__restrict__ out, uint32_t ostride,
                                                     float *__restrict__ wout) {
    uint64_t grp = g.g0 + blockIdx.x * 8ull + (threadIdx.x >> 5);
    if (grp < g.g1)
        group_accum_item(g, off, cnt, e_idx, e_w, wsum, spec, nchan, cstride, out, ostride, wout, grp);
}

template <int W, bool TABLES>
__global__ void __launch_bounds__(32 * W, W == 4 ? kRingCtas : 2) k_tile_rings(const __grid_constant__ GridArgs a, GroupArgs g, TileArgs T) {
    tile_rings_item<W, TABLES>(a, g, T, T.t0 + blockIdx.x);
}

__global__ void __launch_bounds__(kTileThreads, 1) k_tile_accum(GroupArgs g, TileArgs T,
                                                            const unsigned long long *__restrict__ off,
                                                            const uint32_t *__restrict__ cnt,
                                                            const uint32_t *__restrict__ e_slot,
                                                            const float4 *__restrict__ e_w,
                                                            const double *__restrict__ wsum,
                                                            const float *__restrict__ spec, uint32_t nchan,
                                                            uint32_t cstride, float *__restrict__ out,
                                                            uint32_t ostride, float *__restrict__ wout,
                                                            unsigned long long *timeouts) {
    // slices of a tile are adjacent blocks: they run together and share the
    // tile's entries through L2
    tile_accum_item(g, T, off, cnt, e_slot, e_w, wsum, spec, nchan, cstride, out, ostride, wout, T.t0 + blockIdx.y,
                    blockIdx.x * kAccumSlice, timeouts);
}

// Exclusive scan of n uint32 counts into uint64 offsets (out[n] = total),
// one block of 1024 threads.
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const uint32_t *__restrict__ in, uint64_t n,
                                                            uint32_t parts, unsigned long long *__restrict__ psum) {
    scan_sums_item(in, n, parts, psum, blockIdx.x);
}
__global__ void __launch_bounds__(kScanThreads) k_scan_psum(unsigned long long *__restrict__ psum, uint32_t parts) {
    scan_psum_item(psum, parts);
}
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint32_t *__restrict__ in, uint64_t n,
                                                             uint32_t parts, const unsigned long long *__restrict__ psum,
                                                             unsigned long long *__restrict__ out) {
    scan_apply_item(in, n, parts, psum, out, blockIdx.x);
}


// Entry offsets at the first group of every tile row (and the total).
__global__ void k_row_offsets(const unsigned long long *__restrict__ off, uint64_t ngroups, uint64_t groups_per_row,
                              uint32_t nrows, unsigned long long *__restrict__ out) {
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r > nrows) return;
    uint64_t g0 = min((uint64_t)r * groups_per_row, ngroups);
    out[r] = off[g0];
}

// Coarsening: pixel p of row-run [lead, lead + factor) takes the ring range,
// the phi halves of its windows and the polar rule of the run's first pixel
// (HCGrid/gridding.cu:284-308: the disc of l1[0], b1[0]); its own l1, b1,
// cb1 stay for distance and weight. Leaders are only read, so in place.
__global__ void k_coarsen(PixPrep *__restrict__ prep, uint32_t nx, uint64_t npix, uint32_t factor) {
    const uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= npix) return;
    const uint32_t x = (uint32_t)(p % nx), back = x % factor;
    if (back == 0) return;
    const PixPrep L = prep[p - back];
    PixPrep &P = prep[p];
    for (int e = 0; e < 2; ++e) P.tt[e] = L.tt[e];
    P.ur = L.ur;
    P.nr = L.nr;
    P.polar = L.polar;
}

// Target pixel centres of a SIN header, one thread per pixel.
__global__ void k_sin_coords(SinWcs w, uint32_t nx, uint64_t npix, double *__restrict__ X, double *__restrict__ Y) {
    uint64_t o = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (o >= npix) return;
    double x, y;
    sin_pix2world(w, (double)(o % nx) + 1.0, (double)(o / nx) + 1.0, x, y);
    X[o] = x;
    Y[o] = y;
}

}  // namespace

cudaError_t coarsen_prep(PixPrep *prep, uint32_t nx, uint64_t npix, uint32_t factor, cudaStream_t s) {
    if (factor <= 1 || npix == 0) return cudaSuccess;
    k_coarsen<<<(unsigned)((npix + 255) / 256), 256, 0, s>>>(prep, nx, npix, factor);
    return cudaGetLastError();
}

cudaError_t sin_coords_device(const SinWcs &w, uint32_t nx, uint32_t ny, double *d_x, double *d_y, cudaStream_t s) {
    uint64_t n = (uint64_t)nx * ny;
    k_sin_coords<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, nx, n, d_x, d_y);
    return cudaGetLastError();
}

cudaError_t grid_field(hcg_context *ctx, const hcg_field *f, const hcg_target *t, float *d_cube, int layout,
                       float *d_wts, int engine, std::string &why) {
    // engine: HCG_ENGINE_FP32 or a tensor-core engine whose split the field holds
    const bool tc = (engine == HCG_ENGINE_TC_BF16 || engine == HCG_ENGINE_TC_F16) && f->nchan > 1;
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    const uint64_t P = (uint64_t)t->nx * t->ny;
    // the counters of this grid pass: overflow, timeouts, tc_macs, ustat, entries
    if ((e = cudaMemsetAsync(&ctx->d_stats->overflow, 0, sizeof(DevStats) - offsetof(DevStats, overflow), s)) !=
        cudaSuccess)
        return e;
    PixPrep *prep = (PixPrep *)ctx->scratch.get(0, P * sizeof(PixPrep), s, e);
    if (e != cudaSuccess) return e;
    cudaEventRecord(ctx->ev0, s);
    k_pixel_prep<<<(unsigned)((P + 255) / 256), 256, 0, s>>>(f->hpx, f->firstring, f->usedrings, f->disc_size, P,
                                                              t->d_x, t->d_y, prep, ctx->d_stats);
    if ((e = coarsen_prep(prep, t->nx, P, ctx->factor, s)) != cudaSuccess) return e;
    cudaEventRecord(ctx->evp[0], s);
    const GridArgs a = grid_args(f, prep, ctx->d_stats);
    if (f->nchan == 1) {
        cudaEventRecord(ctx->evp[1], s);
        cudaEventRecord(ctx->evp[2], s);
        const uint64_t ngroups = (uint64_t)((t->nx + 1) / 2) * ((t->ny + 1) / 2);
        const int mode = pair_mode1(f, a);
        const unsigned nblk = (unsigned)(mode == kPairSlow ? ngroups : (ngroups + kGroupWarps - 1) / kGroupWarps);
        const bool tab = table_windows(a);
        auto pick = [&](auto table, auto any) { return tab ? table : any; };
        auto grid1 = mode == kPairSlow      ? k_grid_1chan<kPairSlow, false>
                     : mode == kPairEllipse ? pick(k_grid_1chan<kPairEllipse, true>, k_grid_1chan<kPairEllipse, false>)
                     : mode == kPairSinc    ? pick(k_grid_1chan<kPairSinc, true>, k_grid_1chan<kPairSinc, false>)
                     : mode == kPairUnit    ? pick(k_grid_1chan<kPairUnit, true>, k_grid_1chan<kPairUnit, false>)
                                            : pick(k_grid_1chan<kPairGeneral, true>, k_grid_1chan<kPairGeneral, false>);
        grid1<<<nblk, kGroupThreads, 0, s>>>(a, t->nx, t->ny, ngroups, f->d_spec, f->cstride, d_cube, d_wts);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    } else {
        GroupArgs g;
        g.nx = t->nx;
        g.ny = t->ny;
        g.gx = (t->nx + 1) / 2;
        g.ngroups = (uint64_t)g.gx * ((t->ny + 1) / 2);
        uint32_t *cap = (uint32_t *)ctx->scratch.get(1, g.ngroups * sizeof(uint32_t), s, e);
        unsigned long long *off =
            (unsigned long long *)ctx->scratch.get(2, (g.ngroups + 1) * sizeof(unsigned long long), s, e);
        uint32_t *cnt = (uint32_t *)ctx->scratch.get(3, g.ngroups * sizeof(uint32_t), s, e);
        double *wsum = (double *)ctx->scratch.get(4, P * sizeof(double), s, e);
        if (e != cudaSuccess) return e;
        g.g0 = 0;
        g.g1 = g.ngroups;
        g.ebase = 0;
        unsigned gblocks = (unsigned)((g.ngroups + kGroupWarps - 1) / kGroupWarps);
        // tile table (union of ring windows per 16x8-pixel tile)
        TileArgs T{};
        T.ntx = (t->nx + kTileX - 1) / kTileX;
        T.nty = (t->ny + kTileY - 1) / kTileY;
        T.t0 = 0;
        const uint64_t ntiles = (uint64_t)T.ntx * T.nty;
        T.r0 = (int *)ctx->scratch.get(8, ntiles * sizeof(int), s, e);
        T.nr = (int *)ctx->scratch.get(9, ntiles * sizeof(int), s, e);
        T.U = (uint32_t *)ctx->scratch.get(10, ntiles * sizeof(uint32_t), s, e);
        T.ulo = (uint32_t *)ctx->scratch.get(11, ntiles * kTileMaxRings * sizeof(uint32_t), s, e);
        T.base = (uint32_t *)ctx->scratch.get(12, ntiles * (kTileMaxRings + 1) * sizeof(uint32_t), s, e);
        T.ring_idx = (uint16_t *)ctx->scratch.get(14, ntiles * kTileMaxSpan * sizeof(uint16_t), s, e);
        T.cap = cap;  // the tile pass counts each group's candidates
        {
            // the tile pass keeps each group's windows for the weight pass (up to 4 GiB of them)
            const size_t wbytes = (size_t)ntiles * kWinSpan * kTileGroups * 2 * sizeof(uint4);
            cudaError_t ew = cudaSuccess;
            T.win = wbytes <= (4ull << 30) ? (uint4 *)ctx->scratch.get(18, wbytes, s, ew) : nullptr;
            if (ew != cudaSuccess) {
                cudaGetLastError();
                T.win = nullptr;
            }
        }
        T.overflow = &ctx->d_stats->overflow;
        T.pad = tc ? 8 : 1;  // the tensor-core engine loads ring runs as boxes of 8 samples
        T.ustat = ctx->d_stats->ustat;
        T.off = off;
        T.entries = &ctx->d_stats->entries;
        if (e != cudaSuccess) return e;
        if (ntiles <= 148 * 4)
            (table_windows(a) ? k_tile_rings<8, true> : k_tile_rings<8, false>)<<<(unsigned)ntiles, 256, 0, s>>>(a, g, T);
        else
            (table_windows(a) ? k_tile_rings<4, true> : k_tile_rings<4, false>)<<<(unsigned)ntiles, 128, 0, s>>>(a, g, T);
        cudaEventRecord(ctx->evp[1], s);
        if ((e = cudaMemcpyAsync(ctx->h_stats, ctx->d_stats, sizeof(DevStats), cudaMemcpyDeviceToHost, s)) !=
                cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        const DevStats tp = *ctx->h_stats;
        const unsigned long long budget = ctx->entry_budget / (sizeof(uint32_t) + sizeof(float4));
        const uint64_t groups_per_row = (uint64_t)(kTileY / 2) * g.gx;
        // The entries lie in the order the tile pass counted them when they fit
        // the entry budget; else, and with tiles beyond the ring table (whose
        // groups are counted now), the groups' counts are scanned and the work is
        // split into runs of tile rows that fit it.
        std::vector<unsigned long long> ro(T.nty + 1, 0);
        ro[T.nty] = tp.entries;
        const bool whole = tp.overflow == 0 && tp.entries <= budget;
        if (!whole) {
            unsigned long long *rowoff =
                (unsigned long long *)ctx->scratch.get(13, (T.nty + 1) * sizeof(unsigned long long), s, e);
            const uint32_t parts = (uint32_t)std::min<uint64_t>(1024, (g.ngroups + 4095) / 4096 + 1);
            unsigned long long *psum =
                (unsigned long long *)ctx->scratch.get(15, (parts + 1) * sizeof(unsigned long long), s, e);
            if (e != cudaSuccess) return e;
            if (tp.overflow) k_group_count<<<std::min(gblocks, 148u * 3), kGroupThreads, 0, s>>>(a, g, cap);
            k_scan_sums<<<parts, kScanThreads, 0, s>>>(cap, g.ngroups, parts, psum);
            k_scan_psum<<<1, kScanThreads, 0, s>>>(psum, parts);
            k_scan_apply<<<parts, kScanThreads, 0, s>>>(cap, g.ngroups, parts, psum, off);
            k_row_offsets<<<(T.nty + 1 + 255) / 256, 256, 0, s>>>(off, g.ngroups, groups_per_row, T.nty, rowoff);
            if ((e = cudaMemcpyAsync(ro.data(), rowoff, ro.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                     s)) != cudaSuccess ||
                (e = cudaStreamSynchronize(s)) != cudaSuccess)
                return e;
        }
        const bool tiled = tp.overflow == 0;  // every tile's ring span fits the tile table
        if (tc && !tiled && !f->d_spec) {
            why = "a tile spans more than " + std::to_string(kTileMaxSpan) + " rings or holds samples in more than " +
                  std::to_string(kTileMaxRings) + ": the FP32 fallback needs the FP32 spectra";
            return cudaErrorInvalidValue;
        }
        const uint32_t ostride = layout == HCG_LAYOUT_CHANNEL_MAJOR ? 0 : f->nchan;  // 0: [channel][pixel]
        if (tc && tiled && tc_use_weights(ctx, f, tp.ustat[0], ro[T.nty], ntiles)) {
            // dense tiles: the tensor-core kernel evaluates the weights itself (no entries)
            cudaEventRecord(ctx->evp[2], s);
            if ((e = tc_weights(ctx, f, a, g, T, ntiles, d_cube, ostride, d_wts, why)) != cudaSuccess) return e;
            cudaEventRecord(ctx->ev1, s);
            return cudaGetLastError();
        }
        std::vector<std::pair<uint32_t, uint32_t>> chunks;
        unsigned long long most = whole ? std::max(tp.entries, 1ULL) : 1;
        for (uint32_t ra = 0; ra < T.nty;) {
            uint32_t rb = ra + 1;
            // a run fits the entry budget and the 65535 limit of the grid's y dimension
            while (rb < T.nty && (whole || ro[rb + 1] - ro[ra] <= budget) && (uint64_t)(rb + 1 - ra) * T.ntx <= 65535)
                ++rb;
            chunks.push_back({ra, rb});
            if (!whole) most = std::max(most, ro[rb] - ro[ra]);
            ra = rb;
        }
        uint32_t *e_idx = (uint32_t *)ctx->scratch.get(5, (most + 1) * sizeof(uint32_t), s, e);
        float4 *e_w = (float4 *)ctx->scratch.get(6, (most + 1) * sizeof(float4), s, e);
        if (e != cudaSuccess) {
            why = "entry buffer of " + std::to_string(most) + " candidates";
            return e;
        }
        float *dst = d_cube;
        const int smem = kAccumSmem;
        static bool attr_set = false;
        if (tiled && !attr_set) {
            if ((e = cudaFuncSetAttribute(k_tile_accum, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) !=
                cudaSuccess)
                return e;
            attr_set = true;
        }
        bool first = true;
        for (auto &ch : chunks) {
            GroupArgs gc = g;
            if (tiled && tc) {  // the tensor-core builders take packed hi/lo weights
                gc.pack = 1;
                tc_entry_format(f, gc.fmt, gc.wscale);
            }
            gc.g0 = std::min<uint64_t>((uint64_t)ch.first * groups_per_row, g.ngroups);
            gc.g1 = std::min<uint64_t>((uint64_t)ch.second * groups_per_row, g.ngroups);
            gc.ebase = whole ? 0 : ro[ch.first];
            if (gc.g1 <= gc.g0) continue;
            unsigned cb = (unsigned)((gc.g1 - gc.g0 + 7) / 8), gb = (ch.second - ch.first) * T.ntx;
            TileArgs tt = T;
            tt.t0 = (uint64_t)ch.first * T.ntx;
            const int mode = pair_mode(f, a);
            auto pick = [&](auto packed, auto fp32) { return gc.pack ? packed : fp32; };
            auto weights = mode == kPairSlow      ? pick(k_group<kPairSlow, 1>, k_group<kPairSlow, 0>)
                           : mode == kPairEllipse ? pick(k_group<kPairEllipse, 1>, k_group<kPairEllipse, 0>)
                           : mode == kPairSinc    ? pick(k_group<kPairSinc, 1>, k_group<kPairSinc, 0>)
                           : mode == kPairUnit    ? pick(k_group<kPairUnit, 1>, k_group<kPairUnit, 0>)
                                                  : pick(k_group<kPairGeneral, 1>, k_group<kPairGeneral, 0>);
            // two waves of blocks or more: a tile's groups are shared by up to four blocks
            const unsigned parts = gb >= 148 * kWeightCtas * 2 ? 1 : gb >= 148 * kWeightCtas ? 2 : 4;
            weights<<<dim3(gb, parts), kWeightThreads, 0, s>>>(a, gc, off, e_idx, e_w, cnt, wsum, tt, tiled);
            if (first) cudaEventRecord(ctx->evp[2], s);  // phase marks are exact for a single chunk
            first = false;
            if (tiled && tc) {
                TileArgs Tc = T;
                Tc.t0 = (uint64_t)ch.first * T.ntx;
                e = tc_accum(ctx, f, gc, Tc, (uint64_t)(ch.second - ch.first) * T.ntx, off, cnt, e_idx, e_w, wsum, dst,
                             ostride, d_wts, tp.ustat[1], why);
                if (e != cudaSuccess) return e;
            } else if (tiled) {
                TileArgs Tc = T;
                Tc.t0 = (uint64_t)ch.first * T.ntx;
                dim3 grid((f->cstride + kAccumSlice - 1) / kAccumSlice,
                          (unsigned)((uint64_t)(ch.second - ch.first) * T.ntx));
                k_tile_accum<<<grid, kTileThreads, smem, s>>>(gc, Tc, off, cnt, e_idx, e_w, wsum, f->d_spec,
                                                               f->nchan, f->cstride, dst, ostride, d_wts,
                                                               &ctx->d_stats->timeouts);
            } else {
                k_group_accum<<<cb, 256, 0, s>>>(gc, off, cnt, e_idx, e_w, wsum, f->d_spec, f->nchan, f->cstride,
                                                 dst, ostride, d_wts);
            }
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
        if (first) cudaEventRecord(ctx->evp[2], s);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    cudaEventRecord(ctx->ev1, s);
    return cudaGetLastError();
}

}  // namespace hcg

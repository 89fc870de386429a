// Field construction on the device: HEALPix keys of the samples, a stable
// LSD radix sort of (key, original index), the permuted sample geometry,
// the two-level ring lookup table and the per-ring window table.
//
// Reference path replaced (HCGrid/gridding.cu:70-136, all host code there):
//   keys      theta = pi/2 - lat*D2R, phi = lon*D2R, h_ang2pix  (77-82)
//   sort      boost parallel_stable_sort of (hpx, inx) by hpx     (86-92)
//   permute   lons/lats/data gathered by the sorted order          (96-114)
//   LUT       h_start_ring[k] = first sample of ring firstring+k  (118-136)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "hcg_internal.h"

namespace hcg {
namespace {

constexpr int kSortThreads = 256;

// Range of the keys as two maxima that start at zero: of ~key and of key.
struct KeyRange {
    unsigned long long nmin, kmax;
};

// A resident grid of blocks sweeps the samples, so that the range costs two
// atomics a block: one pair per warp (125,000 on one address for 4,000,000
// samples) held the kernel at 175 us.
__global__ void __launch_bounds__(256) k_sample_keys(HpxParams h, uint64_t n, const double *__restrict__ lon,
                                                     const double *__restrict__ lat, uint64_t *__restrict__ keys,
                                                     KeyRange *range, unsigned long long *invalid, DevStats *stats) {
    __shared__ unsigned long long s_nmin[8], s_kmax[8];
    unsigned long long nmin = 0, kmax = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double lo = lon[i], la = lat[i];
        if (!isfinite(lo) || !isfinite(la) || fabs(la) > 90.0) atomicAdd(invalid, 1ULL);
        const double theta = dsub(kHalfPi, dmul(kDeg2Rad, la));
        const double phi = dmul(kDeg2Rad, lo);
        int hard;
        const uint64_t k = ang2pix_quick(h, theta, phi, hard);
        if (hard) atomicAdd(&stats->hard_roundings, 1ULL);
        keys[i] = k;
        nmin = max(nmin, ~(unsigned long long)k);
        kmax = max(kmax, (unsigned long long)k);
    }
    for (int o = 16; o; o >>= 1) {
        nmin = max(nmin, __shfl_xor_sync(0xffffffffu, nmin, o));
        kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_nmin[threadIdx.x >> 5] = nmin;
        s_kmax[threadIdx.x >> 5] = kmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            nmin = max(nmin, s_nmin[w]);
            kmax = max(kmax, s_kmax[w]);
        }
        atomicMax(&range->nmin, nmin);
        atomicMax(&range->kmax, kmax);
    }
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, input index), 8 bits a pass over the bits in
// which the keys differ (key - kmin; 32-bit words whenever they fit, which they
// do for every field smaller than about a quarter of the sky at nside 8192).
// Per pass: k_rs_hist (digit counts of each tile), k_rs_scan (a block per digit
// scans the tiles' counts) and k_rs_scatter. What bounds a pass is the
// scattered writes; sorting a tile by digit in shared memory first makes them
// runs of consecutive positions. 4,000,000 keys in four passes: 0.23 ms
// (1.17 ms with a one-block scan of the 250,000 counts and four block barriers
// per 256 keys).
//
// One tile: each warp ranks kItems x 32 consecutive items with
// ballots against its own digit counters (no block barrier inside),
// then the warps' counts are scanned per digit. Item order is (warp, round,
// lane) = input order, so equal digits keep it.
constexpr int kSortWarps = kSortThreads / 32;

// rank of this lane's digit among the warp's items so far; `cnt` is the warp's
// counter row. Inactive lanes have no counter.
template <typename CNT>
__device__ __forceinline__ uint32_t warp_rank(CNT *cnt, uint32_t d, bool valid) {
    const int lane = threadIdx.x & 31;
    // lanes with the same digit, by its bits: eight votes that overlap (a
    // match instruction takes a turn per distinct digit)
    unsigned peers = __ballot_sync(0xffffffffu, valid);
    if (!valid) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const unsigned bal = __ballot_sync(0xffffffffu, (d >> b) & 1u);
        peers &= (d >> b) & 1u ? bal : ~bal;
    }
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if (valid && lane == leader) {
        old = cnt[d];
        cnt[d] = (CNT)(old + __popc(peers));
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, old, leader) + __popc(peers & ((1u << lane) - 1u));
}

// exclusive scan of one value per thread over the first 256 threads of a
// block; every thread of the block calls it
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t *s_w) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31 && w < 8) s_w[w] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (int i = 0; i < w && i < 8; ++i) before += s_w[i];
    __syncthreads();  // s_w may be written again
    return before + incl - v;
}

// Digit counts of each tile, digit-major (hist[d * nblocks + b]), and of all
// tiles (total[d]).
template <typename KIn, int kItems>
__global__ void __launch_bounds__(kSortThreads) k_rs_hist(const KIn *__restrict__ keys, uint64_t n, int shift,
                                                         uint64_t kmin, uint32_t *__restrict__ hist, uint32_t nblocks,
                                                         unsigned long long *__restrict__ total) {
    __shared__ uint32_t h[kSortWarps][256];
    const int warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < 256 * kSortWarps; d += kSortThreads) (&h[0][0])[d] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * (kSortThreads * kItems);
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint64_t i = base + (uint64_t)j * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[warp][(uint32_t)(((uint64_t)keys[i] - kmin) >> shift) & 255u], 1u);
    }
    __syncthreads();
    const int d = threadIdx.x;
    uint32_t s = 0;
    for (int w = 0; w < kSortWarps; ++w) s += h[w][d];
    hist[(uint64_t)d * nblocks + blockIdx.x] = s;
    if (s) atomicAdd(total + d, (unsigned long long)s);
}

// Block d: the tiles' counts of digit d -> their first output positions.
__global__ void __launch_bounds__(256) k_rs_scan(uint32_t *__restrict__ hist, uint32_t nblocks,
                                                 const unsigned long long *__restrict__ total) {
    __shared__ uint32_t s_w[8];
    __shared__ uint32_t s_tot;
    const int tid = threadIdx.x;
    const uint32_t d = blockIdx.x;
    uint32_t run = 0;
    {
        const uint32_t ex = scan256((uint32_t)total[tid], s_w);
        if (tid == (int)d) s_tot = ex;
        __syncthreads();
        run = s_tot;
    }
    uint32_t *row = hist + (uint64_t)d * nblocks;
    for (uint32_t c = 0; c < nblocks; c += 256) {
        const uint32_t i = c + tid;
        const uint32_t v = i < nblocks ? row[i] : 0u;
        const uint32_t ex = scan256(v, s_w);
        if (i < nblocks) row[i] = run + ex;
        if (tid == 255) s_tot = ex + v;
        __syncthreads();
        run += s_tot;
        __syncthreads();
    }
}

// Input keys are kin[i] - kmin (the first pass reads the samples' keys, and
// their indices are i: vin null); output keys are kout = that + kadd (the last
// pass writes the samples' keys).
template <typename KIn, typename KOut, int kItems>
__global__ void __launch_bounds__(kSortThreads) k_rs_scatter(const KIn *__restrict__ kin,
                                                            const uint32_t *__restrict__ vin,
                                                            KOut *__restrict__ kout, uint32_t *__restrict__ vout,
                                                            uint64_t n, int shift, uint64_t kmin, uint64_t kadd,
                                                            const uint32_t *__restrict__ offs, uint32_t nblocks) {
    using K = typename std::conditional<sizeof(KIn) == 4 || sizeof(KOut) == 4, uint32_t, uint64_t>::type;
    constexpr int kTile = kSortThreads * kItems;
    __shared__ uint32_t s_cnt[kSortWarps][256];
    __shared__ uint32_t s_base[256], s_w[8];
    __shared__ K s_key[kTile];
    __shared__ uint32_t s_val[kTile];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int d = tid; d < kSortWarps * 256; d += kSortThreads) (&s_cnt[0][0])[d] = 0;
    const uint64_t base = (uint64_t)blockIdx.x * kTile, first = base + (uint64_t)warp * (32 * kItems) + lane;
    K key[kItems];
    uint32_t val[kItems], rank[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint64_t i = first + 32 * j;
        key[j] = i < n ? (K)((uint64_t)kin[i] - kmin) : 0;
        val[j] = i < n ? (vin ? vin[i] : (uint32_t)i) : 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const bool valid = first + 32 * j < n;
        rank[j] = warp_rank(s_cnt[warp], (uint32_t)(key[j] >> shift) & 255u, valid);
    }
    __syncthreads();
    uint32_t cnt = 0;
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = s_cnt[w][tid];
        s_cnt[w][tid] = cnt;
        cnt += c;
    }
    const uint32_t start = scan256(cnt, s_w);
    for (int w = 0; w < kSortWarps; ++w) s_cnt[w][tid] += start;
    s_base[tid] = offs[(uint64_t)tid * nblocks + blockIdx.x] - start;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (first + 32 * j < n) {
            const uint32_t p = s_cnt[warp][(uint32_t)(key[j] >> shift) & 255u] + rank[j];
            s_key[p] = key[j];
            s_val[p] = val[j];
        }
    }
    __syncthreads();
    const uint32_t m = n - base < (uint64_t)kTile ? (uint32_t)(n - base) : (uint32_t)kTile;
    for (uint32_t p = tid; p < m; p += kSortThreads) {
        const K k = s_key[p];
        const uint32_t dst = s_base[(uint32_t)(k >> shift) & 255u] + p;
        kout[dst] = (KOut)((uint64_t)k + kadd);
        vout[dst] = s_val[p];
    }
}

// The whole sort of at most kSmallSort keys in one block: the items stay in
// registers between passes and cross shared memory once a pass. Latency is all
// there is at this size: 10,000 keys in three passes take 35 us here against
// 84 us in nine launches of three blocks each.
constexpr int kSmallThreads = 1024, kSmallItems = 16;
constexpr uint64_t kSmallSort = (uint64_t)kSmallThreads * kSmallItems;
constexpr size_t kSmallSmem = kSmallSort * 8 + (kSmallThreads / 32) * 256 * sizeof(uint16_t);
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(const uint64_t *__restrict__ kin,
                                                              uint64_t *__restrict__ kout,
                                                              uint32_t *__restrict__ vout, uint32_t n, int passes,
                                                              uint64_t kmin) {
    extern __shared__ uint32_t s_small[];
    uint32_t *s_key = s_small, *s_val = s_key + kSmallSort;
    uint16_t(*s_cnt)[256] = reinterpret_cast<uint16_t(*)[256]>(s_val + kSmallSort);
    __shared__ uint32_t s_w[8], s_start[256], s_part[4][256];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // rounds a warp takes: its items are consecutive, so unused rounds are skipped for every warp
    const uint32_t rounds = (n + kSmallThreads - 1) / kSmallThreads, first = warp * 32 * rounds + lane;
    uint32_t key[kSmallItems], val[kSmallItems], rank[kSmallItems];
#pragma unroll
    for (int j = 0; j < kSmallItems; ++j) {
        const uint32_t i = first + 32 * j;
        key[j] = j < (int)rounds && i < n ? (uint32_t)(kin[i] - kmin) : 0;
        val[j] = i;
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        for (int d = tid; d < (kSmallThreads / 32) * 256; d += kSmallThreads) (&s_cnt[0][0])[d] = 0;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSmallItems; ++j) {
            if (j >= (int)rounds) break;
            const bool valid = first + 32 * j < n;
            rank[j] = warp_rank(s_cnt[warp], (key[j] >> shift) & 255u, valid);
        }
        __syncthreads();
        // per digit, the warps' counts in four quarters of eight warps
        const uint32_t d = tid & 255, w0 = (tid >> 8) * 8;
        uint32_t cnt = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) cnt += s_cnt[w0 + w][d];
        s_part[tid >> 8][d] = cnt;
        __syncthreads();
        uint32_t start = scan256(tid < 256 ? s_part[0][d] + s_part[1][d] + s_part[2][d] + s_part[3][d] : 0u, s_w);
        if (tid < 256) s_start[d] = start;
        __syncthreads();
        start = s_start[d];
        for (int q = 0; q < (tid >> 8); ++q) start += s_part[q][d];
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = s_cnt[w0 + w][d];
            s_cnt[w0 + w][d] = (uint16_t)start;
            start += c;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSmallItems; ++j) {
            if (j < (int)rounds && first + 32 * j < n) {
                const uint32_t q = s_cnt[warp][(key[j] >> shift) & 255u] + rank[j];
                s_key[q] = key[j];
                s_val[q] = val[j];
            }
        }
        __syncthreads();
        if (p + 1 < passes) {
#pragma unroll
            for (int j = 0; j < kSmallItems; ++j) {
                const uint32_t i = first + 32 * j;
                if (j < (int)rounds && i < n) {
                    key[j] = s_key[i];
                    val[j] = s_val[i];
                }
            }
        }
    }
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        kout[i] = kmin + s_key[i];
        vout[i] = s_val[i];
    }
}

// One pass on the host side: counts, scan, scatter.
template <typename KIn, typename KOut, int kItems>
cudaError_t sort_pass(const KIn *kin, const uint32_t *vin, KOut *kout, uint32_t *vout, uint64_t n, int shift,
                      uint64_t kmin, uint64_t kadd, uint32_t *hist, unsigned long long *total, cudaStream_t s) {
    const uint32_t nblocks = (uint32_t)((n + kSortThreads * kItems - 1) / (kSortThreads * kItems));
    k_rs_hist<KIn, kItems><<<nblocks, kSortThreads, 0, s>>>(kin, n, shift, kmin, hist, nblocks, total);
    k_rs_scan<<<256, 256, 0, s>>>(hist, nblocks, total);
    k_rs_scatter<KIn, KOut, kItems>
        <<<nblocks, kSortThreads, 0, s>>>(kin, vin, kout, vout, n, shift, kmin, kadd, hist, nblocks);
    return cudaGetLastError();
}

// All passes with keys of type K between them; `keys` (the samples' keys) is
// read by the first pass, out_k / out_v written by the last one.
template <typename K, int kItems>
cudaError_t sort_passes(const uint64_t *keys, uint64_t n, int passes, uint64_t kmin, K *t0, K *t1, uint32_t *v0,
                        uint32_t *v1, uint64_t *out_k, uint32_t *out_v, uint32_t *hist, unsigned long long *total,
                        cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    K *a = t0, *b = t1;
    uint32_t *va = v0, *vb = v1;
    for (int p = 0; p < passes && e == cudaSuccess; ++p, total += 256) {
        const bool first = p == 0, last = p + 1 == passes;
        if (first && last)
            e = sort_pass<uint64_t, uint64_t, 8>(keys, nullptr, out_k, out_v, n, 8 * p, kmin, kmin, hist, total, s);
        else if (first)
            e = sort_pass<uint64_t, K, kItems>(keys, nullptr, a, va, n, 8 * p, kmin, 0, hist, total, s);
        else if (last)
            e = sort_pass<K, uint64_t, kItems>(a, va, out_k, out_v, n, 8 * p, 0, kmin, hist, total, s);
        else {
            e = sort_pass<K, K, kItems>(a, va, b, vb, n, 8 * p, 0, 0, hist, total, s);
            std::swap(a, b);
            std::swap(va, vb);
        }
    }
    return e;
}

// Bounds of a ring's samples, kept as maxima of order-preserving 32-bit codes
// (a code of 0 is below every value): |phi| distance from the pixel centre,
// -cos(lat), -lat and lat, each rounded so that the bound holds.
struct RingAcc {
    uint32_t dphi, ncb, nb, b;
};
__device__ __forceinline__ uint32_t order_code(float x) {
    const uint32_t u = __float_as_uint(x);
    return u >> 31 ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float order_value(uint32_t c) {
    return c >> 31 ? __uint_as_float(c & 0x7fffffffu) : __uint_as_float(~c);
}

// Ring half of loc2pix at each used ring's first pixel centre
// (gridding.cu:330-334: ring info, pix2ang of startpix, then the theta used
// by ang2pix for lpix and rpix).
__global__ void k_ring_table(HpxParams h, uint64_t firstring, uint64_t usedrings, const uint32_t *__restrict__ lut,
                             const uint64_t *__restrict__ keys, const RingAcc *__restrict__ acc,
                             RingRec *__restrict__ rings, DevStats *stats) {
    uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k >= usedrings) return;
    RingRec R;
    uint64_t ring = firstring + k;
    ring_info(h, ring, R.startpix, R.npr);
    double z, phi, sth;
    bool have;
    pix2loc(h, R.startpix, z, phi, sth, have);
    double theta = have ? atan2(sth, z) : acos(z);
    // ang2pix(theta, phi) as the kernel calls it: cos (and sin near the poles) of theta
    double s, c;
    int hard;
    sincos_cr(theta, s, c, hard);
    if (hard) atomicAdd(&stats->hard_roundings, 1ULL);
    bool use_sin = (theta < 0.01) || (theta > kPiMinus001);
    double za = fabs(c);
    double ns = u2d(h.nside);
    R.eq = za <= kTwoThird;
    R.zpos = c > 0;
    if (R.eq)
        R.t2 = dmul(dmul(ns, c), 0.75);
    else if ((za < 0.99) || !use_sin)
        R.t2 = dmul(ns, dsqrt(dmul(3., dsub(1., za))));
    else
        R.t2 = ddiv(dmul(ns, s), dsqrt(ddiv(dadd(1., za), 3.)));
    R.lut_lo = lut[k];
    R.lut_hi = lut[k + 1];
    R.phi0 = phi;
    R.dphi = 0.0;
    R.cbmin = 1.0;
    R.bmin = 0.0;
    R.bmax = 0.0;
    if (R.lut_hi > R.lut_lo) {
        const RingAcc A = acc[k];
        R.dphi = order_value(A.dphi);
        R.cbmin = -order_value(A.ncb);
        R.bmin = -order_value(A.nb);
        R.bmax = order_value(A.b);
    }
    // pixel range of the ring's samples; the table offsets follow (k_ring_offsets)
    R.pmin = 0;
    R.span = 0;
    R.tbl = 0;
    if (R.lut_lo != 0 && R.lut_hi > R.lut_lo) {
        R.pmin = (uint32_t)(keys[R.lut_lo] - R.startpix);
        R.span = (uint32_t)(keys[R.lut_hi - 1] - keys[R.lut_lo] + 1);
    }
    rings[k] = R;
}

// Table offset of each ring (span + 1 entries where it holds samples) and the
// total; one block.
__global__ void __launch_bounds__(1024) k_ring_offsets(RingRec *__restrict__ rings, uint64_t usedrings,
                                                       unsigned long long *__restrict__ total) {
    __shared__ unsigned long long s_w[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned long long run = 0;
    for (uint64_t c = 0; c < usedrings; c += 1024) {
        const uint64_t k = c + tid;
        const uint32_t span = k < usedrings ? rings[k].span : 0;
        const unsigned long long v = span ? span + 1ULL : 0ULL;
        unsigned long long incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_w[w] = incl;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (int i = 0; i < 32; ++i) {
            if (i == w) before = all;
            all += s_w[i];
        }
        __syncthreads();
        if (k < usedrings) rings[k].tbl = run + before + incl - v;
        run += all;
    }
    if (tid == 0) *total = run;
}

// A field whose tables are too large: no ring has one.
__global__ void k_ring_no_tables(RingRec *__restrict__ rings, uint64_t usedrings) {
    const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k < usedrings) rings[k].span = 0, rings[k].tbl = 0;
}

// The rings' window records (before k_ring_no_tables).
__global__ void k_ring_windows(HpxParams h, uint64_t firstring, uint64_t usedrings, const RingRec *__restrict__ rings,
                               bool tables, RingWin *__restrict__ out) {
    const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k >= usedrings) return;
    const RingRec R = rings[k];
    const uint64_t r = firstring + k;
    RingWin w;
    w.t2 = R.t2;
    w.bmin = R.bmin;
    w.bmax = R.bmax;
    w.inv_dp = u2d(R.npr) * (0.5 / kPi);
    w.icb = __double2float_ru(1.0 / R.cbmin);
    w.dphi = __double2float_ru(R.dphi + 2e-9);
    w.lut_lo = R.lut_lo;
    w.lut_hi = R.lut_hi;
    w.pmin = R.pmin;
    w.span = R.span;
    const bool centred = r >= h.nside && r <= 3 * h.nside && ((r + h.nside) & 1);
    w.tbl = (tables ? R.tbl : (uint32_t)R.startpix) | (R.eq ? kRingEq : 0) | (centred ? 0 : kRingHalf);
    out[k] = w;
}

// t[0 .. count) = v for each lane of a warp (count 0: nothing): a lane's few
// entries by itself, a long run by the whole warp. Warp-collective. Where samples
// are far apart, a run is most of a ring: a field of 10,000 samples at RA 0, whose
// rings' samples lie at both ends of the circle, took 335 us with a lane a run and
// 126 us so (311 with a search an entry).
__device__ __forceinline__ void warp_fill(uint32_t *t, uint32_t count, uint32_t v) {
    constexpr uint32_t kLong = 16;
    const int lane = threadIdx.x & 31;
    if (count <= kLong)
        for (uint32_t q = 0; q < count; ++q) t[q] = v;
    for (unsigned todo = __ballot_sync(0xffffffffu, count > kLong); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        uint32_t *const at =
            reinterpret_cast<uint32_t *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(t), src));
        const uint32_t m = __shfl_sync(0xffffffffu, count, src), x = __shfl_sync(0xffffffffu, v, src);
#pragma unroll 4
        for (uint32_t q = lane; q < m; q += 32) at[q] = x;
    }
}

// Per-ring pixel tables: entry q of ring k is the first sorted sample of the
// ring whose pixel is >= startpix + pmin + q (entry span: the end of the ring).
// Each sample fills the entries after its predecessor's pixel up to its own,
// so an entry costs one store instead of a binary search (4,000,000 samples:
// 70 us with the searches).
__global__ void __launch_bounds__(256) k_ring_ptab(HpxParams h, uint64_t n, uint64_t firstring,
                                                   const RingRec *__restrict__ rings,
                                                   const uint64_t *__restrict__ keys, uint32_t *__restrict__ ptab) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t *t = ptab;
    uint32_t count = 0;
    if (j < n) {
        const uint64_t key = keys[j];
        const RingRec &R = rings[pix2ring(h, key) - firstring];
        const uint32_t span = R.span;
        if (span) {
            const uint64_t p0 = R.startpix + R.pmin, q = j > R.lut_lo ? keys[j - 1] - p0 + 1 : 0;
            t += R.tbl + q;
            count = (uint32_t)(key - p0 + 1 - q);  // 0: the predecessor's pixel
            if (j + 1 == R.lut_hi) ptab[R.tbl + span] = (uint32_t)(j + 1);
        }
    }
    warp_fill(t, count, (uint32_t)j);
}

// One thread per sorted sample: the permuted geometry, the inverse
// permutation, the ring table's entries at ring changes, and the bounds of
// the sample's ring (one atomic per ring and warp). One pass over the samples
// instead of five (searches per ring, inverse, geometry, a block per ring for
// the bounds). Also the largest |w| of the per-sample weights (when given)
// into *wbits as the bits of a non-negative double, whose order as integers is
// the order of the values; NaN sorts above infinity.
__global__ void __launch_bounds__(256) k_sample_geometry(
    HpxParams h, uint64_t n, uint64_t firstring, uint64_t usedrings, uint64_t *__restrict__ keys,
    const uint32_t *__restrict__ perm, const double *__restrict__ lon, const double *__restrict__ lat,
    const double *__restrict__ w, double *__restrict__ l2, double *__restrict__ b2, double *__restrict__ cb2,
    double *__restrict__ wout, double2 *__restrict__ half, uint32_t *__restrict__ inv, uint32_t *__restrict__ lut,
    RingAcc *__restrict__ acc, unsigned long long *__restrict__ wbits) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool act = j < n;
    unsigned long long wb = 0;
    uint32_t ring = 0xffffffffu;
    RingAcc A{};
    if (act) {
        const uint32_t i = perm[j];
        const double b = dmul(lat[i], kDeg2Rad);
        const double l = dmul(lon[i], kDeg2Rad);
        const double cb = cos(b);
        l2[j] = l;
        b2[j] = b;
        cb2[j] = cb;
        inv[i] = (uint32_t)j;
        const double wi = w ? w[i] : 1.0;
        wout[j] = wi;
        wb = (unsigned long long)__double_as_longlong(fabs(wi));
        double2 q;
        sincos(l * 0.5, &q.x, &q.y);
        const double rc = sqrt(fmax(cb, 0.0));
        q.x *= rc;
        q.y *= rc;
        half[j] = q;
        sincos(b * 0.5, &q.x, &q.y);
        half[n + j] = q;
        const uint64_t key = keys[j], r = pix2ring(h, key);
        ring = (uint32_t)(r - firstring);
        uint64_t start, npr;
        ring_info(h, r, start, npr);
        const bool centred = r >= h.nside && r <= 3 * h.nside && ((r + h.nside) & 1);  // first centre at phi 0
        double d = l - (u2d(key - start) + (centred ? 0.0 : 0.5)) * (2.0 * kPi / u2d(npr));
        d -= 2.0 * kPi * rint(d * (0.5 / kPi));
        A.dphi = order_code(__double2float_ru(fabs(d)));
        A.ncb = order_code(-__double2float_rd(cb));
        A.nb = order_code(-__double2float_rd(b));
        A.b = order_code(__double2float_ru(b));
    }
    uint32_t prev = __shfl_up_sync(0xffffffffu, ring, 1), rings = 0;
    if (act) {
        if (j == 0) {
            keys[n] = h.npix;  // sentinel (gridding.cu:100)
            lut[0] = 0;
        } else {
            if (lane == 0) prev = (uint32_t)(pix2ring(h, keys[j - 1]) - firstring);
            rings = ring - prev;
        }
        if (j + 1 == n) lut[usedrings] = (uint32_t)n;
    }
    warp_fill(lut + (rings ? prev + 1 : 0), rings, (uint32_t)j);  // gridding.cu:118-136
    const unsigned peers = __match_any_sync(0xffffffffu, ring);
    if (act) {
        A.dphi = __reduce_max_sync(peers, A.dphi);
        A.ncb = __reduce_max_sync(peers, A.ncb);
        A.nb = __reduce_max_sync(peers, A.nb);
        A.b = __reduce_max_sync(peers, A.b);
        if (lane == __ffs(peers) - 1) {
            RingAcc *p = acc + ring;
            atomicMax(&p->dphi, A.dphi);
            atomicMax(&p->ncb, A.ncb);
            atomicMax(&p->nb, A.nb);
            atomicMax(&p->b, A.b);
        }
    }
    if (!w) return;
#pragma unroll
    for (int o = 16; o; o >>= 1) wb = max(wb, __shfl_xor_sync(0xffffffffu, wb, o));
    if (lane == 0 && wb) atomicMax(wbits, wb);
}

// One row of nchan values to a row of cstride (a multiple of 4, zero padded),
// by the `tpr` threads that share it (a power of two up to 32; `t` is the
// thread's place): 16 bytes a thread and step.
__device__ __forceinline__ void copy_row(const float *__restrict__ src, float *__restrict__ dst, uint32_t nchan,
                                         uint32_t cstride, uint32_t t, uint32_t tpr) {
    if ((nchan & 3) == 0 && ((uintptr_t)src & 15) == 0) {
        for (uint32_t c = t * 4; c < nchan; c += tpr * 4)
            *reinterpret_cast<float4 *>(dst + c) = __ldg(reinterpret_cast<const float4 *>(src + c));
    } else {
        for (uint32_t c = t * 4; c < cstride; c += tpr * 4) {
            float4 v;
            v.x = __ldg(src + c);
            v.y = c + 1 < nchan ? __ldg(src + c + 1) : 0.f;
            v.z = c + 2 < nchan ? __ldg(src + c + 2) : 0.f;
            v.w = c + 3 < nchan ? __ldg(src + c + 3) : 0.f;
            *reinterpret_cast<float4 *>(dst + c) = v;
        }
    }
}
// threads that share a row: one per 16 bytes, so that short rows (a single
// channel above all: 470 us for 4,000,000 with a warp each) do not leave most
// of a warp idle
inline uint32_t row_threads(uint32_t cstride) {
    uint32_t t = 1;
    while (t < 32 && 4 * t < cstride) t *= 2;
    return t;
}

// out[j][0..cstride) = in[perm[j]][0..nchan), zero padded, and the channels'
// largest finite magnitudes and the count of non-finite values on the way (the
// split needs them; a pass of its own reads the spectra once more, 90 us for
// 500,000 x 256). Block (x, y) takes `rows` rows of channels [128 y, 128 y +
// 128); a thread keeps one channel quad, so its maxima stay in registers and a
// channel costs one atomic a block.
__global__ void __launch_bounds__(256) k_permute_rows(uint64_t n, uint32_t nchan, uint32_t cstride, uint32_t tpr,
                                                      uint32_t rows,
                                                      const uint32_t *__restrict__ perm, const float *__restrict__ in,
                                                      float *__restrict__ out, unsigned int *__restrict__ amax,
                                                      unsigned long long *__restrict__ nonfinite) {
    __shared__ uint4 s_m[256];
    const uint32_t c = blockIdx.y * 128 + 4 * (threadIdx.x % tpr), step = 256 / tpr;
    const bool vec = (nchan & 3) == 0 && ((uintptr_t)in & 15) == 0;
    uint32_t m[4] = {0, 0, 0, 0}, bad = 0;
    if (c < cstride) {
        const uint64_t j0 = blockIdx.x * (uint64_t)rows, j1 = min(n, j0 + rows);
        auto row = [&](uint64_t j) {
            const float *src = in + (uint64_t)__ldg(perm + j) * nchan + c;
            if (vec) return __ldg(reinterpret_cast<const float4 *>(src));
            return make_float4(__ldg(src), c + 1 < nchan ? __ldg(src + 1) : 0.f, c + 2 < nchan ? __ldg(src + 2) : 0.f,
                               c + 3 < nchan ? __ldg(src + 3) : 0.f);
        };
        auto put = [&](uint64_t j, const float4 &v) {
            *reinterpret_cast<float4 *>(out + j * cstride + c) = v;
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t u = __float_as_uint(x[i]) & 0x7fffffffu;
                const bool fin = u < 0x7f800000u;
                m[i] = max(m[i], fin ? u : 0u);
                bad += !fin;
            }
        };
        uint64_t j = j0 + threadIdx.x / tpr;
        for (; j + 3 * step < j1; j += 4 * step) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = row(j + u * step);
#pragma unroll
            for (int u = 0; u < 4; ++u) put(j + u * step, v[u]);
        }
        for (; j < j1; j += step) put(j, row(j));
    }
    if (nchan == 1) return;  // a single channel is not split
    s_m[threadIdx.x] = make_uint4(m[0], m[1], m[2], m[3]);
    if (bad) atomicAdd(nonfinite, (unsigned long long)bad);
    __syncthreads();
    if (threadIdx.x < tpr && c < cstride) {
        for (uint32_t t = threadIdx.x + tpr; t < 256; t += tpr) {
            const uint4 o = s_m[t];
            m[0] = max(m[0], o.x);
            m[1] = max(m[1], o.y);
            m[2] = max(m[2], o.z);
            m[3] = max(m[3], o.w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c + i < nchan && m[i]) atomicMax(amax + c + i, m[i]);
    }
}

// out[j][c] = in[c][perm[j]]: 32x32 tiles through shared memory.
__global__ void k_permute_cols(uint64_t n, uint32_t nchan, uint32_t cstride, const uint32_t *__restrict__ perm,
                               const float *__restrict__ in, float *__restrict__ out) {
    __shared__ float tile[32][33];
    uint64_t j0 = (uint64_t)blockIdx.x * 32;
    uint32_t c0 = blockIdx.y * 32;
    int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        uint64_t j = j0 + tx;
        uint32_t c = c0 + r;
        tile[r][tx] = (j < n && c < nchan) ? in[(uint64_t)c * n + perm[j]] : 0.f;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        uint64_t j = j0 + r;
        uint32_t c = c0 + tx;
        if (j < n && c < cstride) out[j * cstride + c] = tile[tx][r];
    }
}

// One uploaded chunk of sample-major spectra (input rows [r0, r0 + rows))
// scattered to its sorted rows, zero padding to cstride.
__global__ void __launch_bounds__(256) k_scatter_rows(uint64_t r0, uint64_t rows, uint32_t nchan, uint32_t cstride,
                                                      uint32_t tpr, const uint32_t *__restrict__ inv,
                                                      const float *__restrict__ in, float *__restrict__ out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, r = i / tpr;
    if (r >= rows) return;
    copy_row(in + r * nchan, out + (uint64_t)__ldg(inv + r0 + r) * cstride, nchan, cstride, (uint32_t)(i % tpr), tpr);
}

// One uploaded chunk of channel-major spectra (planes [c0, c1) of n samples)
// scattered to the sorted sample-major rows: 32 samples x 32 channels per
// block through shared memory; the last chunk also writes the zero padding
// channels up to cstride.
__global__ void k_scatter_cols(uint64_t n, uint32_t c0, uint32_t c1, uint32_t cend, uint32_t cstride,
                               const uint32_t *__restrict__ inv, const float *__restrict__ in,
                               float *__restrict__ out) {
    __shared__ float tile[32][33];
    const uint64_t j0 = (uint64_t)blockIdx.x * 32;
    const uint32_t cb = c0 + blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const uint64_t j = j0 + tx;
        const uint32_t c = cb + r;
        tile[r][tx] = (j < n && c < c1) ? in[(uint64_t)(c - c0) * n + j] : 0.f;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const uint64_t j = j0 + r;
        const uint32_t c = cb + tx;
        if (j < n && c < cend) out[(uint64_t)__ldg(inv + j) * cstride + c] = tile[tx][r];
    }
}

}  // namespace

cudaError_t build_field(hcg_context *ctx, hcg_field *f, const double *d_lon, const double *d_lat,
                        const double *d_w, std::string &why) {
    cudaStream_t s = ctx->stream;
    const uint64_t n = f->n;
    cudaError_t e;
    uint64_t *k0 = nullptr;  // the samples' keys, then the words read back (one buffer)
    uint32_t *v0 = nullptr;  // the sort's buffers
    uint8_t *mem = nullptr;
    // device words read back: the keys' range and invalid samples, then the pixel tables' total and the largest weight
    struct Back {
        KeyRange range;
        unsigned long long invalid, total, wbits;
    };
    static_assert(sizeof(Back) <= kHostBack, "read back through the context's host words");
    Back *back = nullptr, *hb = reinterpret_cast<Back *>(ctx->h_stats);
    RingAcc *acc = nullptr;
    // the next `count` elements of an allocation, 256-byte aligned; with a null
    // `at` only the offset advances
    size_t used = 0;
    auto carve = [&](auto *&p, uint64_t count) {
        using E = std::remove_reference_t<decltype(*p)>;
        used = (used + 255) & ~(size_t)255;
        p = reinterpret_cast<E *>(mem + used);
        used += count * sizeof(E);
    };
    auto samples = [&]() {
        used = 0;
        carve(f->d_keys, n + 1);
        carve(f->d_l2, n);
        carve(f->d_b2, n);
        carve(f->d_cb2, n);
        carve(f->d_w, n);
        carve(f->d_half, 2 * n);
        carve(f->d_perm, n);
        carve(f->d_inv, n);
    };
    auto ringmem = [&]() {
        used = 0;
        carve(f->d_rings, f->usedrings);
        carve(f->d_rwin, f->usedrings);
        carve(acc, f->usedrings);
        carve(f->d_lut, f->usedrings + 1);
    };
    // The sort's buffers are the context's for up to 2^23 samples (about 250 MB):
    // a buffer that comes and goes between the field's own leaves holes that the
    // spectra (larger than all the others) do not fit, and a program that makes a
    // field a scan waited milliseconds for 0.5 GB to be mapped again.
    const bool keep = n <= (1u << 23);
    auto temp = [&](auto *&p, int slot, size_t bytes) -> cudaError_t {
        if (!keep) return dalloc(&p, bytes, s, ctx->pool);
        cudaError_t te = cudaSuccess;
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(ctx->scratch.get(slot, bytes, s, te));
        return te;
    };
    const size_t key_bytes = ((n + 1) * sizeof(uint64_t) + 255) & ~(size_t)255;
#define TRY(x)                         \
    do {                               \
        e = (x);                       \
        if (e != cudaSuccess) goto fail; \
    } while (0)
    samples();
    TRY(dalloc(&f->d_samples, used, s, ctx->pool));
    mem = static_cast<uint8_t *>(f->d_samples);
    samples();
    TRY(temp(k0, kScratchKeys, key_bytes + sizeof(Back)));
    back = reinterpret_cast<Back *>(reinterpret_cast<uint8_t *>(k0) + key_bytes);
    TRY(cudaMemsetAsync(back, 0, sizeof(Back), s));
    k_sample_keys<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(
        f->hpx, n, d_lon, d_lat, k0, &back->range, &back->invalid, ctx->d_stats);
    TRY(cudaGetLastError());
    {
        TRY(cudaMemcpyAsync(hb, back, sizeof *hb, cudaMemcpyDeviceToHost, s));
        TRY(cudaStreamSynchronize(s));
        if (hb->invalid) {
            why = "non-finite coordinates or |lat| > 90 in " + std::to_string(hb->invalid) + " samples";
            e = cudaErrorInvalidValue;
            goto fail;
        }
        const uint64_t kmin = ~hb->range.nmin, kmax = hb->range.kmax;
        f->firstring = pix2ring(f->hpx, kmin);
        f->usedrings = 1 + pix2ring(f->hpx, kmax) - f->firstring;
        const uint64_t span_bits = 64 - (kmax == kmin ? 64 : __builtin_clzll(kmax - kmin));
        const int passes = span_bits ? (int)((span_bits + 7) / 8) : 1;
        const bool wide = span_bits > 32;
        if (n <= kSmallSort && !wide) {
            TRY(cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
            k_sort_small<<<1, kSmallThreads, kSmallSmem, s>>>(k0, f->d_keys, f->d_perm, (uint32_t)n, passes, kmin);
            TRY(cudaGetLastError());
        } else {
            // tiles of 16 x 256 keys write the longest runs; below about two
            // tiles an SM, and for 64-bit keys (shared memory), smaller ones
            const bool small = n < (1u << 20);
            const size_t word = wide ? 8 : 4, tile = kSortThreads * (wide ? 8 : small ? 4 : 16);
            const size_t nblocks = (n + std::min<size_t>(tile, kSortThreads * 8) - 1) / std::min<size_t>(tile, kSortThreads * 8);
            const size_t pairs = (2 * n * (word + 4) + 255) & ~(size_t)255;
            TRY(temp(v0, kScratchSort, pairs + 256 * nblocks * sizeof(uint32_t) + 8 * 256 * sizeof(unsigned long long)));
            unsigned long long *total = (unsigned long long *)((uint8_t *)v0 + pairs);
            uint32_t *counts = (uint32_t *)(total + 8 * 256), *va = v0 + 2 * n * (word / 4), *vb = va + n;
            uint64_t *const k1 = f->d_keys;
            uint32_t *const perm = f->d_perm;
            TRY(cudaMemsetAsync(total, 0, passes * 256 * sizeof(unsigned long long), s));
            if (wide)
                TRY((sort_passes<uint64_t, 8>(k0, n, passes, kmin, (uint64_t *)v0, (uint64_t *)v0 + n, va, vb, k1,
                                              perm, counts, total, s)));
            else if (small)
                TRY((sort_passes<uint32_t, 4>(k0, n, passes, kmin, v0, v0 + n, va, vb, k1, perm, counts, total, s)));
            else
                TRY((sort_passes<uint32_t, 16>(k0, n, passes, kmin, v0, v0 + n, va, vb, k1, perm, counts, total, s)));
        }
    }
    mem = nullptr;
    ringmem();
    TRY(dalloc(&f->d_ringmem, used, s, ctx->pool));
    mem = static_cast<uint8_t *>(f->d_ringmem);
    ringmem();
    TRY(cudaMemsetAsync(acc, 0, f->usedrings * sizeof(RingAcc), s));
    {
        const unsigned rblocks = (unsigned)((f->usedrings + 255) / 256), nblk = (unsigned)((n + 255) / 256);
        k_sample_geometry<<<nblk, 256, 0, s>>>(f->hpx, n, f->firstring, f->usedrings, f->d_keys, f->d_perm, d_lon,
                                               d_lat, d_w, f->d_l2, f->d_b2, f->d_cb2, f->d_w, f->d_half, f->d_inv,
                                               f->d_lut, acc, &back->wbits);
        k_ring_table<<<rblocks, 256, 0, s>>>(f->hpx, f->firstring, f->usedrings, f->d_lut, f->d_keys, acc, f->d_rings,
                                             ctx->d_stats);
        k_ring_offsets<<<1, 1024, 0, s>>>(f->d_rings, f->usedrings, &back->total);
        TRY(cudaGetLastError());
        TRY(cudaMemcpyAsync(hb, back, sizeof *hb, cudaMemcpyDeviceToHost, s));
        TRY(cudaStreamSynchronize(s));
        f->wmax = 1.0;
        f->unit_w = d_w == nullptr;
        if (d_w) memcpy(&f->wmax, &hb->wbits, sizeof hb->wbits);
        // Pixel tables: one u32 per HEALPix pixel between the first and last
        // sample of each ring and one more, when they fit in max(2^24, 4n)
        // entries (HCG_RING_TABLE_MAX overrides; 0 keeps the binary searches).
        uint64_t cap = std::max<uint64_t>(1ull << 24, 4 * n);
        if (const char *v = getenv("HCG_RING_TABLE_MAX")) cap = strtoull(v, nullptr, 10);
        const bool tables = f->hpx.order <= kQuickOrder && hb->total > 0 && hb->total <= cap &&
                            dalloc(&f->d_ptab, hb->total * sizeof(uint32_t), s, ctx->pool) == cudaSuccess;
        k_ring_windows<<<rblocks, 256, 0, s>>>(f->hpx, f->firstring, f->usedrings, f->d_rings, tables, f->d_rwin);
        if (tables) {
            k_ring_ptab<<<nblk, 256, 0, s>>>(f->hpx, n, f->firstring, f->d_rings, f->d_keys, f->d_ptab);
        } else {
            cudaGetLastError();
            k_ring_no_tables<<<rblocks, 256, 0, s>>>(f->d_rings, f->usedrings);
        }
        TRY(cudaGetLastError());
        f->ptab_entries = f->d_ptab ? hb->total : 0;
    }
fail:
    if (!keep) {
        if (k0) cudaFreeAsync(k0, s);
        if (v0) cudaFreeAsync(v0, s);
    }
#undef TRY
    return e;
}

// Spectra from host memory, uploaded in chunks of kUploadChunk bytes through
// two staging buffers: the copy of chunk k + 1 (copy stream) overlaps the
// scatter of chunk k into sorted order (context stream). Copies wait for the
// work queued on the context stream before the call, and every later use of
// the spectra is ordered after the last scatter on the context stream.
cudaError_t upload_spectra(hcg_context *ctx, hcg_field *f, const float *h_in, uint32_t nchan, int layout) {
    cudaStream_t s = ctx->stream, cs = ctx->copy_stream;
    const uint32_t cstride = (nchan + 3) & ~3u;
    if (f->d_spec && f->cstride != cstride) {
        cudaFreeAsync(f->d_spec, s);
        f->d_spec = nullptr;
    }
    cudaError_t e = cudaSuccess;
    if (!f->d_spec) e = dalloc(&f->d_spec, spec_bytes(f->n, cstride), s, ctx->pool);
    if (e != cudaSuccess) return e;
    f->nchan = nchan;
    f->cstride = cstride;
    f->amax_set = false;
    const uint64_t n = f->n;
    // chunk geometry: whole input rows (sample-major) or whole planes (channel-major)
    const uint64_t unit = layout == HCG_LAYOUT_SAMPLE_MAJOR ? (uint64_t)nchan * 4 : n * 4;
    const uint64_t units = layout == HCG_LAYOUT_SAMPLE_MAJOR ? n : nchan;
    const uint64_t per = std::max<uint64_t>(1, kUploadChunk / unit);
    float *stage[2];
    for (int b = 0; b < 2; ++b) {
        stage[b] = (float *)ctx->scratch.get(19 + b, std::min(per, units) * unit, s, e);
        if (e != cudaSuccess) return e;
    }
    if ((e = cudaEventRecord(ctx->evu[4], s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(cs, ctx->evu[4], 0)) != cudaSuccess) return e;
    uint64_t k = 0;
    for (uint64_t u0 = 0; u0 < units; u0 += per, ++k) {
        const uint64_t cnt = std::min(per, units - u0);
        const int b = (int)(k & 1);
        if (k >= 2 && (e = cudaStreamWaitEvent(cs, ctx->evu[2 + b], 0)) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync(stage[b], h_in + u0 * (unit / 4), cnt * unit, cudaMemcpyHostToDevice, cs)) !=
            cudaSuccess)
            return e;
        if ((e = cudaEventRecord(ctx->evu[b], cs)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(s, ctx->evu[b], 0)) != cudaSuccess) return e;
        if (layout == HCG_LAYOUT_SAMPLE_MAJOR) {
            const uint32_t tpr = row_threads(cstride);
            k_scatter_rows<<<(unsigned)((cnt * tpr + 255) / 256), 256, 0, s>>>(u0, cnt, nchan, cstride, tpr, f->d_inv,
                                                                               stage[b], f->d_spec);
        } else {
            const uint32_t c0 = (uint32_t)u0, c1 = (uint32_t)(u0 + cnt);
            const uint32_t cend = c1 == nchan ? cstride : c1;  // the last chunk writes the padding
            dim3 grid((unsigned)((n + 31) / 32), (cend - c0 + 31) / 32);
            k_scatter_cols<<<grid, dim3(32, 8), 0, s>>>(n, c0, c1, cend, cstride, f->d_inv, stage[b], f->d_spec);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaEventRecord(ctx->evu[2 + b], s)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// `nb` channel planes (host floats [nb][n] at h_planes) into f's sorted
// spectra, in chunks of whole planes through the two staging buffers: copies
// on cs, scatters on us. A chunk's copy waits until the scatter that last read
// its staging buffer is done (ev_free), the scatter for its copy (ev_copied);
// `chunks` counts the chunks of every call that shares the staging buffers.
cudaError_t upload_plane_block(hcg_context *ctx, hcg_field *f, const float *h_planes, uint32_t nb, cudaStream_t cs,
                               cudaStream_t us, float *const stage[2], uint64_t stage_bytes,
                               cudaEvent_t ev_copied[2], cudaEvent_t ev_free[2], uint64_t &chunks) {
    const uint32_t cstride = (nb + 3) & ~3u;
    const uint64_t n = f->n;
    cudaError_t e = cudaSuccess;
    if (f->d_spec && f->cstride != cstride) {
        cudaFreeAsync(f->d_spec, us);
        f->d_spec = nullptr;
    }
    if (!f->d_spec && (e = dalloc(&f->d_spec, spec_bytes(n, cstride), us, ctx->pool)) != cudaSuccess) return e;
    f->nchan = nb;
    f->cstride = cstride;
    f->amax_set = false;
    if (n == 0) return cudaSuccess;
    const uint64_t per = std::max<uint64_t>(1, stage_bytes / (n * 4));
    for (uint64_t u0 = 0; u0 < nb; u0 += per, ++chunks) {
        const uint64_t cnt = std::min<uint64_t>(per, nb - u0);
        const int b = (int)(chunks & 1);
        if (chunks >= 2 && (e = cudaStreamWaitEvent(cs, ev_free[b], 0)) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync(stage[b], h_planes + u0 * n, cnt * n * 4, cudaMemcpyHostToDevice, cs)) != cudaSuccess)
            return e;
        if ((e = cudaEventRecord(ev_copied[b], cs)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(us, ev_copied[b], 0)) != cudaSuccess) return e;
        const uint32_t c0 = (uint32_t)u0, c1 = (uint32_t)(u0 + cnt);
        const uint32_t cend = c1 == nb ? cstride : c1;  // the last chunk writes the padding
        dim3 grid((unsigned)((n + 31) / 32), (cend - c0 + 31) / 32);
        k_scatter_cols<<<grid, dim3(32, 8), 0, us>>>(n, c0, c1, cend, cstride, f->d_inv, stage[b], f->d_spec);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaEventRecord(ev_free[b], us)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t permute_spectra(hcg_context *ctx, hcg_field *f, const float *d_in, uint32_t nchan, int layout) {
    cudaStream_t s = ctx->stream;
    uint32_t cstride = (nchan + 3) & ~3u;
    if (f->d_spec && f->cstride != cstride) {
        cudaFreeAsync(f->d_spec, s);
        f->d_spec = nullptr;
    }
    cudaError_t e = cudaSuccess;
    // The split of the previous spectra goes after the new ones have their place:
    // freed before, its memory would hold them, and the next split (larger) would
    // have to be mapped anew (1.8 against 1.8 to 32 ms for 1,253,838 samples x 3
    // channels, field after field).
    if (!f->d_spec) e = dalloc(&f->d_spec, spec_bytes(f->n, cstride), s, ctx->pool);
    if (e != cudaSuccess && f->d_xhi) {  // unless both do not fit
        cudaGetLastError();
        free_split(f, s);
        e = dalloc(&f->d_spec, spec_bytes(f->n, cstride), s, ctx->pool);
    }
    free_split(f, s);
    if (e != cudaSuccess) return e;
    f->nchan = nchan;
    f->cstride = cstride;
    f->amax_set = false;
    if (layout == HCG_LAYOUT_SAMPLE_MAJOR) {
        const SpecMax mx(f->d_spec, f->n, cstride);
        if (nchan > 1)
            e = cudaMemsetAsync(mx.amax, 0, cstride * sizeof(float) + 2 * sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
        // Two to eight blocks an SM, by 160 KB of spectra a block (the blocks of a
        // channel take turns at its maximum), up to 1024 rows. 200,000 samples, a
        // call with eight an SM / by this rule / without maxima: 2 channels 32.5 /
        // 25 / 30 us, 64 channels 51 / 41 / 45, 128 channels 65 / 58 / 55; 500,000 x
        // 256 channels 193 / 193 / 166 (a pass of its own for the maxima: 90).
        const uint32_t tpr = row_threads(cstride), cblk = (cstride + 127) / 128;
        const uint64_t blocks = std::max<uint64_t>(
            148 * 2, std::min<uint64_t>(148 * 8, f->n * cstride * sizeof(float) / 160000));
        const uint32_t rows =
            (uint32_t)std::max<uint64_t>(256 / tpr, std::min<uint64_t>(1024, f->n * cblk / blocks));
        k_permute_rows<<<dim3((unsigned)((f->n + rows - 1) / rows), cblk), 256, 0, s>>>(
            f->n, nchan, cstride, tpr, rows, f->d_perm, d_in, f->d_spec, mx.amax, mx.bad);
        f->amax_set = nchan > 1;
    } else {
        dim3 grid((unsigned)((f->n + 31) / 32), (cstride + 31) / 32);
        k_permute_cols<<<grid, dim3(32, 8), 0, s>>>(f->n, nchan, cstride, f->d_perm, d_in, f->d_spec);
    }
    return cudaGetLastError();
}

}  // namespace hcg

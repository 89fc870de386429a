// Per-item device functions of the gridding kernels, shared by the
// single-job launches (hcg_grid.cu) and the batch engine (hcg_batch.cu), so
// both execute the same arithmetic. The method is described in hcg_grid.cu.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>

#include "hcg_internal.h"
#include "hcg_sm100.cuh"

namespace hcg {
namespace {

__device__ __forceinline__ uint32_t lower_bound_u64(const uint64_t *__restrict__ a, uint32_t lo, uint32_t hi,
                                                    uint64_t key) {
    while (lo < hi) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(a + mid) < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}
__device__ __forceinline__ uint32_t upper_bound_u64(const uint64_t *__restrict__ a, uint32_t lo, uint32_t hi,
                                                    uint64_t key) {
    while (lo < hi) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(a + mid) <= key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void prep_item(HpxParams h, uint64_t firstring, uint64_t usedrings, double disc,
                                          const double *__restrict__ X, const double *__restrict__ Y,
                                          PixPrep *__restrict__ out, DevStats *stats, uint64_t p) {
    PixPrep P;
    double x = X[p], y = Y[p];
    P.l1 = dmul(x, kDeg2Rad);
    P.b1 = dmul(y, kDeg2Rad);
    P.cb1 = cos(P.b1);
    P.icb1 = __double2float_ru(1.0 / P.cb1);
    if (!isfinite(x) || !isfinite(y)) {
        P.ur = 0; P.nr = 0; P.polar = 0;
        for (int e = 0; e < 2; ++e) P.tt[e] = 0.0;
        // a blank pixel accepts no pair, also where coarsening gives it its run's
        // windows: its haversine is infinite
        P.h = PixHalf{0.0, 0.0, __longlong_as_double(0x7ff0000000000000ll), 0.0};
        out[p] = P;
        return;
    }
    // gridding.cu:306-323
    double disc_theta = dsub(kHalfPi, P.b1);
    double disc_phi = P.l1;
    double utheta = dsub(disc_theta, disc);
    if (dmul(utheta, kRad2Deg) < 0) utheta = 0;
    int hard1, hard2;
    uint64_t uring = pix2ring(h, ang2pix_quick(h, utheta, disc_phi, hard1));
    if (uring < firstring) uring = firstring;
    utheta = dadd(disc_theta, disc);
    uint64_t dring = pix2ring(h, ang2pix_quick(h, utheta, disc_phi, hard2));
    if (dring >= firstring + usedrings) dring = firstring + usedrings - 1;
    if (hard1 | hard2) atomicAdd(&stats->hard_roundings, 1ULL);
    P.ur = (int)(uring - firstring);
    P.nr = (dring >= uring) ? (int)(dring - uring + 1) : 0;
    double dt = dmul(disc_theta, kRad2Deg);
    P.polar = (dt <= kNorthB || dt >= kSouthB);
    P.tt[0] = fmodulo(dmul(dsub(disc_phi, disc), kInvHalfPi), 4.0);
    P.tt[1] = fmodulo(dmul(dadd(disc_phi, disc), kInvHalfPi), 4.0);
    sincos(P.l1 * 0.5, &P.h.sl, &P.h.cl);
    const double rc = sqrt(fmax(P.cb1, 0.0));
    P.h.sl *= rc;
    P.h.cl *= rc;
    sincos(P.b1 * 0.5, &P.h.sb, &P.h.cb);
    // A pixel past a pole (|lat| > 90, cos(lat) < 0) has no such operands: its
    // haversines are NaN, and pair_band takes each of its pairs by the full formula
    if (P.cb1 < 0.0) P.h.sl = P.h.cl = __longlong_as_double(0x7ff8000000000000ll);
    out[p] = P;
}

// loc2pix(z_ring, phi_edge) from its ring half and phi half.
__device__ __forceinline__ uint64_t edge_pix(const HpxParams &h, const RingRec &R, const PixPrep &P, int e) {
    const double tt = P.tt[e];
    if (R.eq) {
        uint64_t nl4 = 4 * h.nside;
        const double temp1 = dmul(u2d(h.nside), dadd(0.5, tt));
        uint64_t jp = d2u(dsub(temp1, R.t2));
        uint64_t jm = d2u(dadd(temp1, R.t2));
        uint64_t ir = h.nside + 1 + jp - jm;
        uint64_t kshift = 1 - (ir & 1);
        uint64_t t1 = jp + jm + kshift + 1 + nl4 + nl4 - h.nside;
        uint64_t ip = (h.order > 0) ? ((t1 >> 1) & (nl4 - 1)) : ((t1 >> 1) % nl4);
        return h.ncap + (ir - 1) * nl4 + ip;
    }
    const double tp = dsub(tt, u2d(d2u(tt)));
    uint64_t jp = d2u(dmul(tp, R.t2));
    uint64_t jm = d2u(dmul(dsub(1.0, tp), R.t2));
    uint64_t ir = jp + jm + 1;
    uint64_t ip = d2u(dmul(tt, u2d(ir)));
    return R.zpos ? 2 * ir * (ir - 1) + ip : h.npix - 2 * ir * (ir + 1) + ip;
}

// Samples [lo, hi) of ring R whose pixels lie in [lpix, rpix].
__device__ __forceinline__ void pixel_window(const RingRec &R, uint64_t lpix, uint64_t rpix,
                                             const uint64_t *__restrict__ keys, const uint32_t *__restrict__ ptab,
                                             uint32_t &lo, uint32_t &hi) {
    if (R.span) {
        // the ring's pixel table gives the same bounds as the searches below
        const int64_t q0 = (int64_t)(lpix - R.startpix) - (int64_t)R.pmin;
        lo = q0 <= 0 ? R.lut_lo : (q0 >= (int64_t)R.span ? R.lut_hi : __ldg(ptab + R.tbl + q0));
        const int64_t q1 = (int64_t)(rpix - R.startpix) - (int64_t)R.pmin + 1;  // first pixel > rpix
        const uint32_t h1 = q1 <= 0 ? R.lut_lo : (q1 >= (int64_t)R.span ? R.lut_hi : __ldg(ptab + R.tbl + q1));
        hi = h1 > lo ? h1 : lo;
        return;
    }
    lo = lower_bound_u64(keys, R.lut_lo, R.lut_hi, lpix);
    hi = upper_bound_u64(keys, lo, R.lut_hi, rpix);
}

// Candidate interval [lo, hi) of one ring for one pixel
// (gridding.cu:329-367). Returns false where the reference would spin.
__device__ __forceinline__ bool ring_window(const HpxParams &h, const RingRec &R, const PixPrep &P,
                                            const uint64_t *__restrict__ keys, const uint32_t *__restrict__ ptab,
                                            uint32_t &lo, uint32_t &hi) {
    lo = hi = 0;
    uint64_t lpix = P.polar ? R.startpix : edge_pix(h, R, P, 0);
    if (!(lpix >= R.startpix && lpix < R.startpix + R.npr)) return false;
    uint64_t rpix = P.polar ? R.startpix + R.npr - 1 : edge_pix(h, R, P, 1);
    if (!(rpix >= R.startpix && rpix < R.startpix + R.npr)) return false;
    if (R.lut_lo == 0) return true;  // first used ring: the reference's search returns "none"
    pixel_window(R, lpix, rpix, keys, ptab, lo, hi);
    return true;
}

// helpers.cu:128-130 (degrees), with cos(b1), cos(b2) precomputed.
__device__ __forceinline__ double dist_deg(double l1, double b1, double cb1, double l2, double b2, double cb2) {
    double sb = sin((b1 - b2) * 0.5);
    double sl = sin((l1 - l2) * 0.5);
    return 2.0 * asin(sqrt(sb * sb + cb1 * cb2 * (sl * sl))) * kRad2Deg;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Four consecutive channels c..c+3 of pixel p into the cube: [pixel][channel]
// with row stride `ostride`, or [channel][pixel] (plane stride npix) when
// ostride is 0.
__device__ __forceinline__ void store_cube4(float *__restrict__ out, uint32_t ostride, uint64_t npix, uint64_t p,
                                            uint32_t c, uint32_t nchan, const float v[4]) {
    if (ostride) {
        float *o = out + p * ostride;
        if (c + 3 < nchan && (ostride & 3) == 0) {
            *reinterpret_cast<float4 *>(o + c) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            for (int j = 0; j < 4; ++j)
                if (c + j < nchan) o[c + j] = v[j];
        }
    } else {
        for (int j = 0; j < 4; ++j)
            if (c + j < nchan) out[(uint64_t)(c + j) * npix + p] = v[j];
    }
}

}  // namespace

// Geometry arguments of the gathering kernels (shared by several translation units).
struct GridArgs {
    HpxParams h;
    const RingRec *rings;
    const PixPrep *prep;
    const uint64_t *keys;
    const double *l2, *b2, *cb2, *w;
    double sphere_radius, p0;
    DevStats *stats;
    const double2 *half;  // sorted samples' pair operands (hcg_field::d_half)
    const uint32_t *ptab; // per-ring pixel tables (RingRec::tbl), or null
    double hlo, hhi;      // haversine thresholds bracketing sphere_radius (see grid_args)
    int series;           // d^2 from the arcsine-squared series (small sphere_radius)
    double hpolar;        // haversine bound of every accepted pair (chord windows)
    float x2c[3];         // -4 R2D^2 p0 log2(e) times 1, 1/3, 8/45: the FP32 Gaussian's exponent by powers of h
    int series32;         // series && GAUSS1D: accepted pairs below the band take gauss_series_f32
    uint32_t ktype;       // HCG_GAUSS1D, HCG_GAUSS2D or HCG_TAPERED_SINC
    int ktaper;           // TAPERED_SINC with HCG_TAPER_FIX
    double kp1, kp2;      // second and third kernel parameters (p0 is the first)
    const RingWin *rwin;  // the rings' window records
    uint64_t firstring;
    float hpolar32;       // >= hpolar
    int unit_w;           // every sample weight is 1
    float hlo32, hhi32;   // <= hlo, >= hhi: the brackets an FP32 haversine decides
    double e2c[5];        // -4 R2D^2 p0 log2(e) times 1, 1/3, 8/45, 4/35, 128/1575: GAUSS1D's base-2 exponent by powers of h
    int exp2ok;           // series, GAUSS1D, and no accepted pair's weight is below 2^-1000 (exp2_small)
    double g2scale;       // -log2(e) / (2 (sigma_maj sigma_min)^2): GAUSS2D's base-2 exponent per d^2 and ellipse term
    int g2ok;             // series, GAUSS2D, and no accepted pair's weight is below 2^-1000 (exp2_small)
    int w32ok;            // the same for 2^-120: no accepted pair's FP32 weight is zero
    uint64_t n;           // samples
    double spa, cpa;      // GAUSS2D: sine and cosine of the position angle
    double tsx, tsr, tse; // TAPERED_SINC: the sinc's argument over pi per degree, 1 / (pi tsx), the taper's base-2 exponent per d^2
    int tsok;             // series, TAPERED_SINC, and the taper stays within 2^-1000 and 2^1000 (exp2_small)
};

namespace {

// Host: GridArgs of a field. The cutoff d < r (d = 2 asin(sqrt(h)) in degrees,
// helpers.cu:128-130) is decided from the haversine h alone when h is outside
// [h* (1 - 1e-9), h* (1 + 1e-9)], h* = sin^2(r / 2): the device's h and d carry
// relative errors below 1e-12 there, so the decision is the one the full
// formula takes. Inside the band the full formula decides.
inline GridArgs grid_args(const hcg_field *f, const PixPrep *prep, DevStats *stats) {
    GridArgs a{f->hpx, f->d_rings, prep, f->d_keys, f->d_l2, f->d_b2, f->d_cb2, f->d_w, f->sphere_radius,
               f->kparam0, stats, f->d_half, f->d_ptab, 0.0, 0.0, 0};
    const double s = std::sin(f->sphere_radius * kDeg2Rad * 0.5);
    const double hstar = s * s;
    a.hlo = hstar * (1.0 - 1e-9);
    a.hhi = hstar * (1.0 + 1e-9);
    a.series = hstar < 1e-3;
    a.hpolar = hstar * (1.0 + 1e-6);
    a.ktype = f->kernel_type;
    a.series32 = a.series && f->kernel_type == HCG_GAUSS1D;
    a.ktaper = f->taper_fix;
    a.kp1 = f->kparams[1];
    a.kp2 = f->kparams[2];
    a.rwin = f->d_rwin;
    a.firstring = f->firstring;
    a.hpolar32 = (float)(hstar * (1.0 + 2e-6));
    a.unit_w = f->unit_w;
    const double e2scale = -4.0 * kRad2Deg * kRad2Deg * f->kparam0 * 1.4426950408889634;
    const double series[5] = {1.0, 1.0 / 3.0, 8.0 / 45.0, 4.0 / 35.0, 128.0 / 1575.0};
    for (int i = 0; i < 5; ++i) a.e2c[i] = e2scale * series[i];
    for (int i = 0; i < 3; ++i) a.x2c[i] = (float)a.e2c[i];
    a.w32ok = a.series32 && e2scale <= 0.0 && e2scale * hstar * 1.01 > -120.0;
    a.exp2ok = a.series32 && e2scale <= 0.0 && e2scale * hstar * 1.01 > -1000.0;
    // d < sphere_radius and the ellipse term is at most the larger sigma squared
    const double s0 = f->kparam0 * f->kparam0, s1 = f->kparams[1] * f->kparams[1];
    a.g2scale = -0.5 * 1.4426950408889634 / (s0 * s1);
    a.g2ok = f->kernel_type == HCG_GAUSS2D && a.series &&
             -a.g2scale * f->sphere_radius * f->sphere_radius * std::max(s0, s1) * 1.01 < 1000.0;
    a.tsx = 1.0 / std::fabs(f->kparam0 * f->kparams[2]);
    a.tsr = 1.0 / (kPi * a.tsx);
    const double tp = kPi / (f->kparam0 * f->kparams[1]);
    a.tse = (f->taper_fix ? -1.4426950408889634 : 1.4426950408889634) * tp * tp;
    a.tsok = f->kernel_type == HCG_TAPERED_SINC && a.series && a.tsx > 1e-100 && a.tsx < 1e100 &&
             std::fabs(a.tse) * f->sphere_radius * f->sphere_radius * 1.01 < 1000.0;
    a.hlo32 = (float)(a.hlo * (1.0 - 2e-7));
    a.hhi32 = (float)(a.hhi * (1.0 + 2e-7));
    a.n = f->n;
    a.spa = std::sin(f->kparams[2]);
    a.cpa = std::cos(f->kparams[2]);
    return a;
}

// Candidate interval of the multi-channel path: the reference's window
// (gridding.cu:329-367; whole rings within 20 deg of a pole, 340-354)
// intersected with the pixels whose centres can hold a sample of the ring
// within the radius. An accepted pair has hav(d) < hpolar, and hav(d) =
// hav(db) + cos b_p cos b_s hav(dphi) with |db| >= the distance of b_p from
// the ring's latitude range and cos b_s >= the ring's smallest cos(lat), which
// bounds |dphi|; a sample lies within R.dphi of its pixel centre. The accepted
// pairs are the reference window's; only candidates beyond the radius are
// left out. Windows whose phi range wraps keep the reference's. `ref_len` is
// the reference window's length (its candidate count).
__device__ __forceinline__ bool ring_window_mc(const GridArgs &a, const RingRec &R, const PixPrep &P, uint32_t &lo,
                                               uint32_t &hi, uint32_t &ref_len) {
    ref_len = 0;
    if (!ring_window(a.h, R, P, a.keys, a.ptab, lo, hi)) return false;
    ref_len = hi > lo ? hi - lo : 0;
    if (R.lut_lo == 0 || hi <= lo || !(P.cb1 >= 0.0)) return true;  // past a pole the bound does not hold
    // hav(db) >= y^2 (1 - y^2 / 3) with y = db / 2 (sin y >= y - y^3 / 6)
    const double y = 0.5 * fmax(0.0, fmax(R.bmin - P.b1, P.b1 - R.bmax));
    const double hb = y < 1.0 ? y * y * (1.0 - y * y * (1.0 / 3.0)) : 0.0;
    if (!(hb < a.hpolar)) {  // no sample of the ring within the radius
        hi = lo;
        return true;
    }
    const double H = (a.hpolar - hb) / (R.cbmin * P.cb1);
    if (!(H < 0.25)) return true;
    // |dphi| <= 2 asin(sqrt(H)) <= 2 sqrt(H / (1 - H)) (asin x = atan(x / sqrt(1 - x^2)) <= x / sqrt(1 - x^2))
    const double W = 2.0 * sqrt(H / (1.0 - H)) * (1.0 + 1e-9) + R.dphi + 1e-9;
    const double dp = 2.0 * kPi / (double)R.npr;
    const double lp = P.l1 - 2.0 * kPi * floor(P.l1 / (2.0 * kPi));
    const double jl = floor((lp - W - R.phi0) / dp), jh = ceil((lp + W - R.phi0) / dp);
    if (!(jl >= 0.0 && jh < (double)R.npr && jh - jl + 1.0 < (double)R.npr)) return true;
    uint32_t clo, chi;
    pixel_window(R, R.startpix + (uint64_t)jl, R.startpix + (uint64_t)jh, a.keys, a.ptab, clo, chi);
    lo = max(lo, clo);
    hi = max(lo, min(hi, chi));
    return true;
}

// Out of line: the loops around it keep nothing for it.
struct RingWindow {
    uint32_t lo, hi, ref_len;
    bool ok;
};
__device__ __noinline__ RingWindow ring_window_call(const GridArgs &a, const PixPrep &P, int k) {
    RingWindow w;
    w.ok = ring_window_mc(a, a.rings[k], P, w.lo, w.hi, w.ref_len);
    return w;
}
__device__ __forceinline__ bool ring_window_general(const GridArgs &a, const PixPrep &P, int k, uint32_t &lo,
                                                    uint32_t &hi, uint32_t &ref_len) {
    const RingWindow w = ring_window_call(a, P, k);
    lo = w.lo;
    hi = w.hi;
    ref_len = w.ref_len;
    return w.ok;
}

// The pixels of a 2x2 group as the window arithmetic takes them: per pixel the
// edges' longitudes and ring range (empty for pixels outside the map or
// without samples), and the group's extent for the chord's bound.
struct GroupGeo {
    double tt[4][2];
    int ur[4], ue[4];  // rings [ur, ue)
    unsigned polar;    // bit q: whole-ring windows
    double lmin, lmax, bmin, bmax;  // longitudes in [0, 2 pi)
    float icb;         // >= 1 / cos(lat) of every pixel; inf: no chord bound
    int r0, r1;        // union of the ring ranges, [r0, r1]
};

template <typename GET>  // get(q): the PixPrep of pixel q, or null
__device__ __forceinline__ GroupGeo group_geo(GET get) {
    GroupGeo G;
    G.polar = 0;
    G.lmin = G.bmin = 1e300;
    G.lmax = G.bmax = -1e300;
    G.icb = 0.f;
    G.r0 = 1 << 30;
    G.r1 = -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const PixPrep *P = get(q);
        G.tt[q][0] = G.tt[q][1] = 0.0;
        G.ur[q] = 1;
        G.ue[q] = 0;
        if (!P || P->nr <= 0) continue;
        G.tt[q][0] = P->tt[0];
        G.tt[q][1] = P->tt[1];
        G.ur[q] = P->ur;
        G.ue[q] = P->ur + P->nr;
        G.r0 = min(G.r0, G.ur[q]);
        G.r1 = max(G.r1, G.ue[q] - 1);
        if (P->polar) G.polar |= 1u << q;
        const double lp = P->l1 - 2.0 * kPi * floor(P->l1 * (0.5 / kPi));
        G.lmin = fmin(G.lmin, lp);
        G.lmax = fmax(G.lmax, lp);
        // past a pole: no bound, in latitude neither; a blank pixel (NaN) accepts
        // nothing and leaves the others theirs
        const bool past = P->icb1 < 0.f;
        G.bmin = fmin(G.bmin, past ? -1e300 : P->b1);
        G.bmax = fmax(G.bmax, past ? 1e300 : P->b1);
        G.icb = past ? __int_as_float(0x7f800000) : fmaxf(G.icb, P->icb1);
    }
    if (G.lmax - G.lmin > kPi) G.icb = __int_as_float(0x7f800000);  // the group straddles phi = 0
    return G;
}

// The windows of a group's four pixels in the field's ring k in the general
// form, for stray edges.
__device__ __forceinline__ void group_windows_general(const GridArgs &a, int k, const GroupGeo &G, uint64_t pix0,
                                                      uint32_t nx, uint32_t lo[4], uint32_t hi[4], uint32_t &ref,
                                                      uint32_t &skips) {
    for (int q = 0; q < 4; ++q) {
        lo[q] = hi[q] = 0;
        if (k < G.ur[q] || k >= G.ue[q]) continue;
        uint32_t rl;
        if (ring_window_general(a, a.prep[pix0 + (q & 1) + (uint64_t)(q >> 1) * nx], k, lo[q], hi[q], rl)) {
            ref += rl;
        } else {
            lo[q] = 1;
            hi[q] = 0;
            ++skips;
        }
    }
}

// First sample of a ring ([first, last), pixels from `start` on) at or after each of
// N ring-local pixels: N binary searches in step, so that their loads are in flight
// together.
template <int N>
__device__ __forceinline__ void lower_bounds(const uint64_t *__restrict__ keys, uint32_t first, uint32_t last,
                                             uint32_t start, const uint32_t (&pix)[N], uint32_t (&at)[N]) {
    // ring-local pixels are at most 2^31: the keys' low words decide
    const uint32_t *key = reinterpret_cast<const uint32_t *>(keys);
#pragma unroll
    for (int i = 0; i < N; ++i) at[i] = first;
    uint32_t n = last - first;
    for (; n > 1; n -= n / 2) {
        uint32_t v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = __ldg(key + 2 * (uint64_t)(at[i] + n / 2 - 1)) - start;
#pragma unroll
        for (int i = 0; i < N; ++i) at[i] += v[i] < pix[i] ? n / 2 : 0;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) at[i] += n && __ldg(key + 2 * (uint64_t)at[i]) - start < pix[i] ? 1 : 0;
}

// The windows of a group's four pixels in the field's ring k from its 64-byte
// record: the reference window of each pixel (ring_window's integers, from the
// same rounded operations on ring-local 32-bit pixel numbers; an edge that
// rounds into another ring takes the general form), intersected with one chord
// bound for the group. The bound is FP32 rounded outwards, from the group's
// extent: it only leaves out candidates beyond the radius of every pixel, so it
// needs no more, and whole pixels inside it are kept without a pixel of margin.
// lo > hi marks a ring the reference would spin on; `ref` adds the reference
// windows' lengths, `skips` such rings. What bounds it: instruction issue; a
// general window takes about 600 instructions (four FP64 divisions, a root,
// 64-bit pixel numbers, a 104-byte record), a group's four here about 300.
// TABLE: the first sample at or after a pixel from the ring's pixel table, else
// (fields too sparse for tables, or with rings that span the circle, or nside above
// 2^26) by the group's ten binary searches in step. 2,000,000 samples on 1200 x 1200 pixels, 10 a beam,
// a pass with one channel / 16 channels on the FP32 engine: 2.78 / 5.66 ms; 5.66 /
// 8.73 with a general window for each pixel in turn, 4.56 / 6.03 with one a thread.
template <bool TABLE>
__device__ __forceinline__ void group_windows(const GridArgs &a, const RingWin &R, int k, const GroupGeo &G,
                                              uint64_t pix0, uint32_t nx, uint32_t lo[4], uint32_t hi[4],
                                              uint32_t &ref, uint32_t &skips) {
    using I = typename std::conditional<TABLE, int, long long>::type;  // tables: nside <= 2^26 (kQuickOrder)
    auto trunc_u = [](double x) { return TABLE ? (I)__double2uint_rz(x) : (I)__double2ull_rz(x); };
    const I ns = (I)a.h.nside, ring = (I)(a.firstring + (uint64_t)k);
    const double nsd = (double)ns;
    const bool eq = (R.tbl & kRingEq) != 0;
    const I i4 = eq ? 4 * ns : 4 * min(ring, (I)(4 * ns - ring));  // pixels of the ring
    const I span = (I)R.span, pmin = (I)R.pmin;
    const uint32_t *t = a.ptab + (TABLE ? R.tbl & kRingTbl : 0);
    auto first_of = [&](I pix) { return __ldg(t + max((I)0, min((I)(pix - pmin), span))); };  // first sample at or after pix
    uint32_t clo = 0, chi = 0xffffffffu;
    I cl = 0, ch = i4;  // !TABLE: the chord's first pixel and the one after its last
    if (span) {
        const float y = 0.5f * (float)fmax(0.0, fmax(R.bmin - G.bmax, G.bmin - R.bmax));
        const float hb = y < 1.f ? y * y * (1.f - y * y * (1.f / 3.f)) * (1.f - 1e-6f) : 0.f;
        const float H = (a.hpolar32 - hb) * R.icb * G.icb * (1.f + 1e-6f);
        if (!(hb < a.hpolar32)) {  // no sample of the ring within the radius
            chi = 0;
        } else if (H >= 0.f && H < 0.25f) {
            // |dphi| <= 2 asin(sqrt(H)) <= 2 sqrt(H / (1 - H)), and a sample lies within dphi of its pixel centre
            const float W = 2.f * sqrtf(__fdividef(H, 1.f - H)) * (1.f + 4e-6f) + R.dphi;
            const double w = (double)W * R.inv_dp + 1e-4, s = (R.tbl & kRingHalf) ? 0.5 : 0.0;
            const double xl = G.lmin * R.inv_dp - s - w, xh = G.lmax * R.inv_dp - s + w;
            const I jl = TABLE ? (I)__double2int_ru(xl) : (I)__double2ll_ru(xl);
            const I jh = TABLE ? (I)__double2int_rd(xh) : (I)__double2ll_rd(xh);
            if (jl >= 0 && jh < i4 && jh - jl + 1 < i4) {  // else: wraps, the reference windows stay
                if (TABLE) {
                    clo = first_of(jl);
                    chi = first_of(jh + 1);
                } else {
                    cl = jl;
                    ch = jh + 1;
                }
            }
        }
    }
    // straight-line code over the four pixels: the lookups of all of them are
    // in flight together
    I e0[4], e1[4];
    bool stray = false;
    if (eq) {
        const I c = ((ring - ns) & 1) + 1 + 7 * ns, want = ring - 2 * ns;
        auto edge = [&](double tt, bool &same) {
            const double t1 = dmul(nsd, dadd(0.5, tt));
            const I jp = trunc_u(dsub(t1, R.t2)), jm = trunc_u(dadd(t1, R.t2));
            same = same && jp - jm == want;
            return ((jp + jm + c) >> 1) & (i4 - 1);
        };
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            bool same = true;
            e0[q] = edge(G.tt[q][0], same);
            e1[q] = edge(G.tt[q][1], same);
            stray = stray || (!same && k >= G.ur[q] && k < G.ue[q] && !(G.polar >> q & 1u));
        }
    } else {
        auto edge = [&](double tt, bool &same) {
            const double tp = dsub(tt, floor(tt));
            const I ir = trunc_u(dmul(tp, R.t2)) + trunc_u(dmul(dsub(1.0, tp), R.t2)) + 1;
            const I ip = trunc_u(dmul(tt, (double)ir));
            same = same && 4 * ir == i4 && ip < i4;
            return ip;
        };
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            bool same = true;
            e0[q] = edge(G.tt[q][0], same);
            e1[q] = edge(G.tt[q][1], same);
            stray = stray || (!same && k >= G.ur[q] && k < G.ue[q] && !(G.polar >> q & 1u));
        }
    }
    if (stray) {  // an edge rounded into another ring
        group_windows_general(a, k, G, pix0, nx, lo, hi, ref, skips);
        return;
    }
    uint32_t rl[4] = {0, 0, 0, 0}, rh[4] = {0, 0, 0, 0};
    if (!TABLE && span) {
        uint32_t pix[10], at[10];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool whole = G.polar >> q & 1u;
            pix[q] = whole ? 0u : (uint32_t)e0[q];
            pix[4 + q] = whole ? (uint32_t)i4 : (uint32_t)(e1[q] + 1);
        }
        pix[8] = (uint32_t)cl;
        pix[9] = (uint32_t)max(ch, (I)0);
        lower_bounds(a.keys, R.lut_lo, R.lut_hi, (uint32_t)R.tbl, pix, at);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            rl[q] = at[q];
            rh[q] = at[4 + q];
        }
        clo = at[8];
        chi = min(chi, at[9]);
    } else if (span) {  // else no samples, or the first used ring (the reference's search returns "none")
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool whole = G.polar >> q & 1u;
            rl[q] = first_of(whole ? 0 : e0[q]);
            rh[q] = first_of(whole ? i4 : e1[q] + 1);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const bool act = k >= G.ur[q] && k < G.ue[q];
        const uint32_t h = max(rl[q], rh[q]);
        ref += act ? h - rl[q] : 0u;
        lo[q] = act ? max(rl[q], clo) : 0u;
        hi[q] = act ? max(lo[q], min(h, chi)) : 0u;
    }
}

// The form for the field, or TABLES: the table's (the call of the others costs a
// kernel registers: 4,000,000 samples on 1200 x 1200 pixels, single channel, 1982
// against 1967 us). The searches are out of line.
struct GroupWin {
    uint32_t lo[4], hi[4], ref, skips;
};
__device__ __noinline__ GroupWin group_windows_search(const GridArgs &a, GroupGeo G, int k, uint64_t pix0,
                                                      uint32_t nx) {
    GroupWin w;
    w.ref = w.skips = 0;
    group_windows<false>(a, a.rwin[k], k, G, pix0, nx, w.lo, w.hi, w.ref, w.skips);
    return w;
}
template <bool TABLES>
__device__ __forceinline__ void group_windows_any(const GridArgs &a, int k, const GroupGeo &G, uint64_t pix0,
                                                  uint32_t nx, uint32_t lo[4], uint32_t hi[4], uint32_t &ref,
                                                  uint32_t &skips) {
    if (TABLES || a.ptab) {
        group_windows<true>(a, a.rwin[k], k, G, pix0, nx, lo, hi, ref, skips);
    } else {
        const GroupWin w = group_windows_search(a, G, k, pix0, nx);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            lo[q] = w.lo[q];
            hi[q] = w.hi[q];
        }
        ref += w.ref;
        skips += w.skips;
    }
}

// exp(-x) for the FP32 weights of the multi-channel path, x >= 0 from FP64:
// 2^(-x log2 e) with the exponent rounded once to FP32 and the hardware
// base-2 exponential (ex2.approx.ftz.f32, relative error about 2^-22). For
// x <= 4.5 (d <= 3 sigma) the result is within 5e-7 of exp(-x), relative.
__device__ __forceinline__ float gauss_f32(double x) {
    const float t = (float)(-x * 1.4426950408889634);  // log2(e)
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t));
    return r;
}

// The same for an accepted pair whose cutoff is decided, from its haversine h <
// 1e-3 rounded to FP32: the arcsine-squared series h (1 + h / 3 + 8 h^2 / 45)
// (the next term is 2e-10 of it) with the scale folded into its coefficients.
// The exponent's relative error stays below 3e-7, the weight's below 1.6e-6 at
// d = 3 sigma.
__device__ __forceinline__ float gauss_series_f32(float hf, const float (&c)[3]) {
    const float t = hf * (c[0] + hf * (c[1] + hf * c[2]));
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t));
    return r;
}

// Half-angle differences of a pair and its haversine: sb = sin((b1 - b2) / 2),
// sl = sin((l1 - l2) / 2) sqrt(cos b1 cos b2) and h = sb^2 + sl^2, expanded from
// the positions' operands (PixHalf; `sl2`, `sb2` are the sample's).
struct PairHav {
    double sb, sl, h;
};
__device__ __forceinline__ PairHav pair_hav(const PixHalf &q, const double2 &sl2, const double2 &sb2) {
    PairHav v;
    v.sb = q.sb * sb2.y - q.cb * sb2.x;
    v.sl = q.sl * sl2.y - q.cl * sl2.x;
    v.h = v.sb * v.sb + v.sl * v.sl;
    return v;
}

// The arcsine-squared series of pair_d2.
__device__ __forceinline__ double series_d2(double h) {
    const double t = h * (1.0 + h * (1.0 / 3.0 + h * (8.0 / 45.0 + h * (4.0 / 35.0 + h * (128.0 / 1575.0)))));
    return 4.0 * t * (kRad2Deg * kRad2Deg);
}

// d^2 (degrees^2) of an accepted pair from its haversine: asin^2(x) =
// sum_n (2x)^(2n) / (2 n^2 C(2n, n)) at x = sqrt(h), five terms (used when
// h* < 1e-3, truncation below 1e-16 relative), else asin itself.
__device__ __forceinline__ double pair_d2(const GridArgs &a, double h) {
    if (a.series) return series_d2(h);
    const double d = 2.0 * asin(sqrt(h)) * kRad2Deg;
    return d * d;
}

// GAUSS1D's base-2 exponent of a pair from its haversine (five terms, pair_d2).
__device__ __forceinline__ double exponent2(const GridArgs &a, double h) {
    return h * (a.e2c[0] + h * (a.e2c[1] + h * (a.e2c[2] + h * (a.e2c[3] + h * a.e2c[4]))));
}

// 2^t for -1000 < t <= 0: the nearest integer by adding and subtracting
// 1.5 * 2^52, 2^f on |f| <= 1/2 by its interpolant of degree 11 in the Chebyshev
// points (4e-18 of it, 2e-17 with the coefficients rounded), and the integer into
// the exponent. The range is known, so nothing is tested; within 2 ulp.
__device__ __forceinline__ double exp2_small(double t) {
    const double big = 6755399441055744.0, k = t + big, f = t - (k - big);
    double p = 4.4558179083360645e-10;
    p = fma(p, f, 7.074194297288521e-09);
    p = fma(p, f, 1.0178057087733941e-07);
    p = fma(p, f, 1.3215432535912375e-06);
    p = fma(p, f, 1.5252733841556773e-05);
    p = fma(p, f, 0.00015403530463724353);
    p = fma(p, f, 0.001333355814640647);
    p = fma(p, f, 0.009618129107587256);
    p = fma(p, f, 0.055504108664821625);
    p = fma(p, f, 0.24022650695910158);
    p = fma(p, f, 0.6931471805599453);
    p = fma(p, f, 1.0);
    return __hiloint2double(__double2hiint(p) + (__double2loint(k) << 20), __double2loint(p));
}

__device__ __forceinline__ double ellipse_xy(const GridArgs &a, double x, double y, double &n2) {
    const double ys = y * a.cpa - x * a.spa, xc = x * a.cpa + y * a.spa;
    n2 = x * x + y * y;
    return (a.p0 * a.p0) * (ys * ys) + (a.kp1 * a.kp1) * (xc * xc);
}

// GAUSS2D's ellipse term of a pair, as a quotient: (sigma_maj sin)^2 +
// (sigma_min cos)^2 of (bearing - PA), times n2, which is returned beside it
// (kernel_other derives the bearing's tangent y / x).
__device__ __forceinline__ double ellipse(const GridArgs &a, const PixHalf &q, double cb1, const PairHav &v,
                                          const double2 &sl2, const double2 &sb2, double &n2) {
    const double cl = q.cl * sl2.y + q.sl * sl2.x;  // cos((l1 - l2) / 2) sqrt(cos b1 cos b2)
    const double cb = q.cb * sb2.y + q.sb * sb2.x;  // cos((b1 - b2) / 2)
    const double y = -2.0 * (v.sl * cl);
    const double x = 2.0 * (2.0 * (q.sb * q.cb) * (v.sl * v.sl) - cb1 * v.sb * cb);
    return ellipse_xy(a, x, y, n2);
}

// 1 / x, x >= 1e-300: the hardware's approximation (20 bits) and three
// Newton-Raphson steps r += r (1 - x r), each of which doubles the bits: within
// 2 ulp, and without the branch of a division, so that four of them interleave.
__device__ __forceinline__ double reciprocal(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#pragma unroll
    for (int i = 0; i < 3; ++i) r = fma(r, fma(-x, r, 1.0), r);
    return r;
}

// GAUSS2D from its ellipse term.
__device__ __forceinline__ double gauss2d(const GridArgs &a, double num, double n2, double d2) {
    const double ell = n2 > 0.0 ? num / n2 : 0.0;
    const double pp = a.p0 * a.kp1;
    return exp(-0.5 * d2 * ell / (pp * pp));
}

// The grid kernels other than GAUSS1D (gridding.cu:242-256), FP64, for an
// accepted pair with squared distance d2: GAUSS2D (sigma_maj, sigma_min, PA)
// at the great-circle bearing of the sample seen from the pixel
// (helpers.cu:133-137), TAPERED_SINC (sigma, a, b) with sinc(x) = 1 for
// |x| < 1e-10 (gridding.cu:229-235) and the taper exp(+(arg/a)^2) of the
// reference, or exp(-(arg/a)^2) with HCG_TAPER_FIX. The bearing's tangent
// y / x has y = cos b2 sin dl and x = cos b1 sin b2 - sin b1 cos b2 cos dl =
// sin(b2 - b1) + 2 sin b1 cos b2 sin^2(dl / 2); both, times cos b1, follow from
// the half-angle products, and only sin^2 and cos^2 of (bearing - PA) are
// wanted, so neither the arc tangent nor any sine or cosine is evaluated (the
// weight pass of 150,001 samples on 251 x 203 pixels took 355 us with them).
__device__ __forceinline__ double kernel_other(const GridArgs &a, const PixHalf &q, double cb1, const PairHav &v,
                                               const double2 &sl2, const double2 &sb2, double d2) {
    const double p0 = a.p0, p1 = a.kp1, p2 = a.kp2;
    if (a.ktype == HCG_GAUSS2D) {
        double n2;
        const double num = ellipse(a, q, cb1, v, sl2, sb2, n2);
        return gauss2d(a, num, n2, d2);
    }
    const double arg = kPi * sqrt(d2) / p0;
    const double x = arg / p2;
    const double s = fabs(x) < 1.e-10 ? 1. : sin(x) / x;
    const double t = (arg / p1) * (arg / p1);
    return s * exp(a.ktaper ? -t : t);
}

// Weight of an accepted pair with squared distance d2 (degrees^2). GEN: the
// field's kernel may be other than GAUSS1D. F32: multi-channel entries hold
// FP32 weights, so the Gaussian is evaluated in FP32 (gauss_f32).
template <bool F32, bool GEN>
__device__ __forceinline__ double kernel_at(const GridArgs &a, const PixHalf &q, double cb1, const PairHav &v,
                                            const double2 &sl2, const double2 &sb2, double win, double d2) {
    if (GEN && a.ktype != HCG_GAUSS1D) {
        const double k = kernel_other(a, q, cb1, v, sl2, sb2, d2);
        return win * (F32 ? (double)(float)k : k);
    }
    return win * (F32 ? (double)gauss_f32(d2 * a.p0) : exp(-d2 * a.p0));
}

// A pair near the cutoff (rare): inside the band [hlo, hhi] the reference's
// full formula decides, and for pixels past a pole (NaN haversine) it decides
// every pair. Out of line, by value and from memory again, so that the
// loop around it keeps nothing for it.
template <bool F32, bool GEN>
__device__ __noinline__ double pair_band(const GridArgs &a, const PixPrep *P, uint32_t idx) {
    const PixPrep Q = *P;
    const double2 sl2 = __ldg(a.half + idx), sb2 = __ldg(a.half + a.n + idx);
    const double win = __ldg(a.w + idx);
    const PairHav v = pair_hav(Q.h, sl2, sb2);
    if (v.h > a.hhi) return 0.0;
    if (v.h < a.hlo) {
        if (F32 && !GEN && a.series32) return win * (double)gauss_series_f32((float)v.h, a.x2c);
        return kernel_at<F32, GEN>(a, Q.h, Q.cb1, v, sl2, sb2, win, pair_d2(a, v.h));
    }
    const double l2 = __ldg(a.l2 + idx), b2 = __ldg(a.b2 + idx), cb2 = __ldg(a.cb2 + idx);
    const double d = dist_deg(Q.l1, Q.b1, Q.cb1, l2, b2, cb2);
    if (!(d < a.sphere_radius)) return 0.0;
    if (GEN && a.ktype == HCG_GAUSS2D) {  // the bearing from the positions as well
        double n2;
        const double num = ellipse_xy(a, Q.cb1 * sin(b2) - sin(Q.b1) * cb2 * cos(l2 - Q.l1), cb2 * sin(l2 - Q.l1), n2);
        const double k = gauss2d(a, num, n2, d * d);
        return win * (F32 ? (double)(float)k : k);
    }
    return kernel_at<F32, GEN>(a, Q.h, Q.cb1, v, sl2, sb2, win, d * d);
}

// Weights of sample idx for the four pixels of a group (0 outside
// sphere_radius, decided from the haversine). `in`: the sample is in the
// pixel's window. `wf` is the weight rounded to FP32 (F32 only), `nz`: it is
// not zero. Straight-line code: the four pixels' chains interleave, and a pair
// that is not accepted costs a select, not a branch. MODE kPairUnit: GAUSS1D
// with unit-weight samples (F32: the FP32 Gaussian of the series; else
// exp2_small), where the haversine rounded to FP32 decides all but the pairs
// within 2e-7 of the cutoff, relative. kPairEllipse, kPairSinc: GAUSS2D and
// TAPERED_SINC on small radii and with weights in range; kPairSlow: those kernels
// beyond, TAPERED_SINC's accepted pairs one by one out of line (pair_band; in line
// for all four pixels, accepted or not, a single-channel map of 200 x 120 pixels
// under a beam of 3.3 degrees took 2.85 ms, 1.96 ms so).
enum { kPairGeneral = 0, kPairUnit = 1, kPairEllipse = 2, kPairSinc = 3, kPairSlow = 4 };
template <bool F32, int MODE>
__device__ __forceinline__ void pair_weights(const GridArgs &a, const PixPrep *P, uint32_t nx, const PixHalf q[4],
                                             const double cb1[4], const double2 &sl2, const double2 &sb2, double win,
                                             uint32_t idx, const bool in[4], double w[4], float wf[4], bool nz[4]) {
    constexpr bool GEN = MODE >= kPairEllipse;
    PairHav v[4];
    bool acc[4];
    unsigned band = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = pair_hav(q[i], sl2, sb2);
    if (MODE == kPairUnit) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float hf = (float)v[i].h;
            acc[i] = in[i] && hf < a.hlo32;
            if (in[i] && !acc[i] && !(hf > a.hhi32)) band |= 1u << i;
        }
        if (F32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                wf[i] = acc[i] ? gauss_series_f32((float)v[i].h, a.x2c) : 0.f;
                w[i] = (double)wf[i];
                nz[i] = acc[i];
            }
        } else {
            double t[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = exponent2(a, v[i].h);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w[i] = exp2_small(t[i]);  // of a pair beyond the cutoff: not used
                nz[i] = acc[i];
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[i] = in[i] && v[i].h < a.hlo;
            if (in[i] && !acc[i] && !(v[i].h > a.hhi)) band |= 1u << i;
        }
        if (F32 && !GEN && a.series32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float gs = gauss_series_f32((float)v[i].h, a.x2c);
                w[i] = acc[i] ? win * (double)gs : 0.0;
            }
        } else if (MODE == kPairSlow && a.ktype == HCG_GAUSS2D) {
            double d2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d2[i] = pair_d2(a, acc[i] ? v[i].h : 0.0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                double n2;
                const double num = ellipse(a, q[i], cb1[i], v[i], sl2, sb2, n2), k = gauss2d(a, num, n2, d2[i]);
                w[i] = acc[i] ? win * (F32 ? (double)(float)k : k) : 0.0;
            }
        } else if (MODE == kPairSlow) {
            for (int i = 0; i < 4; ++i) {
                if (acc[i]) band |= 1u << i;
                w[i] = 0.0;
            }
        } else if (MODE == kPairEllipse) {
            // GAUSS2D, its weights in range: the four pixels' chains side by side
            // (through kernel_other, a division and a call of exp a pixel in turn,
            // the weight pass of 150,001 samples on 251 x 203 pixels took 148 us;
            // 80 us so)
            double t[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double h = v[i].h;
                double n2;
                const double num = ellipse(a, q[i], cb1[i], v[i], sl2, sb2, n2);
                const double ell = n2 > 1e-300 ? num * reciprocal(n2) : 0.0;
                t[i] = series_d2(h) * a.g2scale * ell;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double k = exp2_small(t[i]);  // of a pair beyond the cutoff: not used
                w[i] = acc[i] ? win * (F32 ? (double)(float)k : k) : 0.0;
            }
        } else if (MODE == kPairSinc) {
            // TAPERED_SINC, its taper in range: sin(x) / x with x = pi y, and the
            // taper from d^2, so that a pair takes one root's reciprocal and no
            // division (256,456 samples on 85 x 75 pixels, one channel: 300 us; 908
            // with four divisions, a sine and an exponential through kernel_at)
            double y[4], ry[4], t[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double d2 = series_d2(v[i].h), r = rsqrt(d2);
                y[i] = d2 * r * a.tsx;
                ry[i] = r * a.tsr;
                t[i] = d2 * a.tse;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double sinc = y[i] * kPi >= 1e-10 ? sinpi(y[i]) * ry[i] : 1.0;
                const double k = sinc * exp2_small(t[i]);  // of a pair beyond the cutoff: not used
                w[i] = acc[i] ? win * (F32 ? (double)(float)k : k) : 0.0;
            }
        } else if (!F32 && a.exp2ok) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double k = exp2_small(exponent2(a, v[i].h));
                w[i] = acc[i] ? win * k : 0.0;
            }
        } else {
            double d2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d2[i] = pair_d2(a, acc[i] ? v[i].h : 0.0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double k = kernel_at<F32, false>(a, q[i], 0.0, v[i], sl2, sb2, win, d2[i]);
                w[i] = acc[i] ? k : 0.0;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            wf[i] = F32 ? (float)w[i] : 0.f;
            nz[i] = w[i] != 0.0;
        }
    }
    if (band) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (band >> i & 1u) {
                w[i] = pair_band<F32, GEN>(a, P + (i & 1) + (uint64_t)(i >> 1) * nx, idx);
                wf[i] = F32 ? (float)w[i] : 0.f;
                nz[i] = MODE == kPairUnit && F32 ? wf[i] != 0.f : w[i] != 0.0;
            }
        }
    }
}

// The windows of the field's rings are those of pixel tables.
inline bool table_windows(const GridArgs &a) { return a.ptab != nullptr; }
// The single-channel and the multi-channel pair mode of a field.
inline int pair_mode1(const hcg_field *f, const GridArgs &a) {
    if (f->kernel_type != HCG_GAUSS1D) return a.g2ok ? kPairEllipse : a.tsok ? kPairSinc : kPairSlow;
    return a.unit_w && a.exp2ok ? kPairUnit : kPairGeneral;
}
inline int pair_mode(const hcg_field *f, const GridArgs &a) {
    if (f->kernel_type != HCG_GAUSS1D) return a.g2ok ? kPairEllipse : a.tsok ? kPairSinc : kPairSlow;
    return a.unit_w && a.w32ok ? kPairUnit : kPairGeneral;
}

// Sums of four values over a warp's lanes: lanes 8q .. 8q + 7 return value q's
// (six exchanges instead of twenty).
__device__ __forceinline__ double warp_sum4(const double v[4]) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16, odd = lane & 8;
    double a0 = up ? v[2] : v[0], a1 = up ? v[3] : v[1];
    a0 += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
    a1 += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
    double s = odd ? a1 : a0;
    s += __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 8);
#pragma unroll
    for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// A warp's ring records: per ring with candidates (compacted, in ring order),
// the union's first candidate as the sample index of candidate 0 of the ring
// block, the slot shift, and the four pixels' windows as (first sample, length).
struct GroupRecords {
    uint4 ra[32], rb[32];
    uint2 rc[32];
};
// A warp's shared memory for one 2x2 group taken by itself: pixels and records.
constexpr int kGroupWarps = 4, kGroupThreads = 32 * kGroupWarps, kGroupCtas = 5;
struct GroupShared {
    PixPrep prep[4];
    PixHalf h[4];
    double cb1[4];
    GroupRecords rec;
};

// Pixels of group grp into the warp's shared memory (pixels outside the map
// hold no rings).
__device__ __forceinline__ void group_load(GroupShared &S, const PixPrep *__restrict__ prep, uint64_t pix0,
                                           uint32_t nx, bool xin, bool yin) {
    static_assert(sizeof(PixPrep) == 11 * sizeof(double), "eleven words a pixel");
    const int lane = threadIdx.x & 31, q = lane >> 3, i = lane & 7;
    const bool valid = (!(q & 1) || xin) && (!(q >> 1) || yin);
    const double *src = reinterpret_cast<const double *>(prep + pix0 + (q & 1) + (uint64_t)(q >> 1) * nx);
    double *dst = reinterpret_cast<double *>(&S.prep[q]);
    __syncwarp();
    dst[i] = valid ? __ldg(src + i) : 0.0;
    if (i < 3) dst[8 + i] = valid ? __ldg(src + 8 + i) : 0.0;
    __syncwarp();
    if (lane < 4) {
        S.h[lane] = S.prep[lane].h;
        S.cb1[lane] = S.prep[lane].cb1;
    }
    __syncwarp();
}

// One block of up to 32 rings (lane = ring) of a group: every union candidate,
// 32 at a time, tested against the four pixels; `body(x, slot, w, wf, nz)` gets
// the candidate's spectrum value (single channel: `data`, rows of `cstride`) and
// weights. Warp-collective. What bounds it: instruction issue (about 40 a pair)
// with the FP64 pipe next. The ring of a candidate is found from one reduction of
// the ring ends that fall into the round (a bit each) instead of a search by
// shuffles, its record read from shared memory instead of sixteen shuffles, and a
// candidate's geometry is loaded once for four pixels, a round ahead (4,000,000
// samples on 1200 x 1200 pixels: 1524 -> 1424 us single channel, 945 -> 898 us
// for the entries; copies through shared memory or ring ends kept as bits there
// cost as many instructions as they saved).
template <bool F32, int MODE, int PARTS = 1, typename BODY>
__device__ __forceinline__ void group_rounds(const GridArgs &a, const PixHalf *s_h, const double *s_cb1,
                                             GroupRecords &S, uint64_t pix0, uint32_t nx, const uint32_t lo[4],
                                             const uint32_t hi[4], uint32_t shift, const float *__restrict__ data,
                                             uint32_t cstride, BODY body, uint32_t part = 0) {
    const int lane = threadIdx.x & 31;
    uint32_t glo = 0xffffffffu, ghi = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (hi[q] > lo[q]) {
            glo = min(glo, lo[q]);
            ghi = max(ghi, hi[q]);
        }
    }
    const uint32_t len = glo < ghi ? ghi - glo : 0;
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const int c = __popc(__ballot_sync(0xffffffffu, len > 0) & ((1u << lane) - 1u));
    __syncwarp();  // the records of the previous ring block are no longer read
    if (len) {
        auto n = [&](int q) { return hi[q] > lo[q] ? hi[q] - lo[q] : 0u; };
        S.ra[c] = make_uint4(glo - (incl - len), shift, lo[0], n(0));
        S.rb[c] = make_uint4(lo[1], n(1), lo[2], n(2));
        S.rc[c] = make_uint2(lo[3], n(3));
    }
    __syncwarp();
    // the round's samples, fetched while the round before is worked on
    int r = 0;
    double2 nsl, nsb;
    float nx1 = 0.f;
    auto fetch = [&](uint32_t tb) {
        const unsigned ends = __reduce_or_sync(0xffffffffu, len && incl > tb && incl - tb < 32 ? 1u << (incl - tb) : 0u);
        const int c0 = __popc(__ballot_sync(0xffffffffu, len && incl <= tb));
        const bool act = tb + lane < total;
        r = act ? c0 + __popc(ends & (0xffffffffu >> (31 - lane))) : c0;
        // a lane past the last candidate repeats the round's first one, outside every window
        const uint32_t idx = S.ra[r].x + (act ? tb + lane : tb);
        nsl = __ldg(a.half + idx);
        nsb = __ldg(a.half + a.n + idx);
        if (!F32) nx1 = __ldg(data + (uint64_t)idx * cstride);
    };
    const uint32_t tb0 = PARTS > 1 ? 32 * part : 0;
    if (total > tb0) fetch(tb0);
    for (uint32_t tb = tb0; tb < total; tb += 32 * PARTS) {
        // the pixels' constants are read anew each round (the barrier keeps the
        // compiler from holding their 40 registers, which cost a third of the warps)
        __syncwarp();
        PixHalf ph[4];
        double cb1[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            ph[q] = s_h[q];
            cb1[q] = MODE == kPairEllipse || MODE == kPairSlow ? s_cb1[q] : 0.0;  // only the ellipse takes it
        }
        const bool act = tb + lane < total;
        const uint4 ra = S.ra[r], rb = S.rb[r];
        const uint2 rc = S.rc[r];
        const uint32_t idx = ra.x + (act ? tb + lane : tb);
        const double2 sl2 = nsl, sb2 = nsb;
        const float x = nx1;
        if (tb + 32 * PARTS < total) fetch(tb + 32 * PARTS);
        const double win = MODE == kPairUnit || a.unit_w ? 1.0 : __ldg(a.w + idx);
        const bool in[4] = {act && idx - ra.z < ra.w, act && idx - rb.x < rb.y, act && idx - rb.z < rb.w,
                            act && idx - rc.x < rc.y};
        double w[4];
        float wf[4];
        bool nz[4];
        pair_weights<F32, MODE>(a, a.prep + pix0, nx, ph, cb1, sl2, sb2, win, idx, in, w, wf, nz);
        body(x, idx + ra.y, w, wf, nz);
    }
}

// Windows of this lane's ring k of a group computed from the pixels in the
// warp's shared memory.
template <bool TABLES>
__device__ __forceinline__ void group_lane_windows(const GridArgs &a, const GroupGeo &G, int k, uint64_t pix0,
                                                   uint32_t nx, uint32_t lo[4], uint32_t hi[4], uint32_t &ref,
                                                   uint32_t &skips) {
    if (k > G.r1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) lo[q] = hi[q] = 0;
    } else {
        group_windows_any<TABLES>(a, k, G, pix0, nx, lo, hi, ref, skips);
    }
}

// Pair counts a warp's groups add up (the same in every lane; flushed by its
// kernel).
struct PairCounts {
    unsigned long long cand = 0, within = 0, skips = 0;
    // warp-collective: the lanes' counts of one item
    __device__ __forceinline__ void add(uint32_t c, uint32_t w, uint32_t s) {
        cand += __reduce_add_sync(0xffffffffu, c);
        within += __reduce_add_sync(0xffffffffu, w);
        skips += __reduce_add_sync(0xffffffffu, s);
    }
};
// The block's counts to the context's statistics: one atomic per block (one
// per pixel or group on one address was a bound of its own). Block-collective.
__device__ __forceinline__ void flush_counts(const PairCounts &c, DevStats *stats) {
    __shared__ unsigned long long s_c[3];
    if (threadIdx.x < 3) s_c[threadIdx.x] = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        if (c.cand) atomicAdd(&s_c[0], c.cand);
        if (c.within) atomicAdd(&s_c[1], c.within);
        if (c.skips) atomicAdd(&s_c[2], c.skips);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_c[0]) atomicAdd(&stats->pairs_candidate, s_c[0]);
        if (s_c[1]) atomicAdd(&stats->pairs_within, s_c[1]);
        if (s_c[2]) atomicAdd(&stats->ring_skips, s_c[2]);
    }
}

// Single channel: one warp per 2x2 group of pixels, FP64 throughout: the
// windows (a ring per lane, four pixels each), every union candidate against
// the four pixels, normalise. Warp-collective. kPairSlow: the block's warps share
// one group, every kGroupWarps-th round of candidates each (a pair's evaluation
// is long, so that few pixels leave most of the GPU idle, and the windows formed
// by each warp cost little beside it); block-collective.
template <int MODE>
constexpr int kGrid1Parts = MODE == kPairSlow ? kGroupWarps : 1;
template <int MODE, bool TABLES>
__device__ __forceinline__ void grid1_item(const GridArgs &a, uint32_t nx, uint32_t ny,
                                           const float *__restrict__ data, uint32_t cstride, float *__restrict__ out,
                                           float *__restrict__ wout, uint64_t grp, GroupShared &S, PairCounts &pc) {
    constexpr int PARTS = kGrid1Parts<MODE>;
    const int lane = threadIdx.x & 31, part = PARTS > 1 ? threadIdx.x >> 5 : 0;
    const uint32_t gx = (nx + 1) / 2, gyi = (uint32_t)(grp / gx), gxi = (uint32_t)(grp % gx);
    const bool xin = 2 * gxi + 1 < nx, yin = 2 * gyi + 1 < ny;
    const uint64_t pix0 = (uint64_t)(2 * gyi) * nx + 2 * gxi;
    group_load(S, a.prep, pix0, nx, xin, yin);
    double acc[4] = {0.0, 0.0, 0.0, 0.0}, ws[4] = {0.0, 0.0, 0.0, 0.0};
    uint32_t ref = 0, within = 0, skips = 0;
    for (int rb = 0, nr = 1; rb < nr; rb += 32) {
        uint32_t lo[4], hi[4];
        {  // the group's extent is not kept across the pair tests (registers)
            const GroupGeo G = group_geo([&](int q) { return &S.prep[q]; });
            nr = G.r1 - G.r0 + 1;
            group_lane_windows<TABLES>(a, G, G.r0 + rb + lane, pix0, nx, lo, hi, ref, skips);
        }
        group_rounds<false, MODE, PARTS>(a, S.h, S.cb1, S.rec, pix0, nx, lo, hi, 0u, data, cstride,
                                  [&](float v, uint32_t, const double w[4], const float[4], const bool nz[4]) {
            const double x = (double)v;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (nz[q]) {
                    acc[q] += x * w[q];
                    ws[q] += w[q];
                    ++within;
                }
            }
        }, part);
    }
    pc.add(part == 0 ? ref : 0, within, part == 0 ? skips : 0);
    double A = warp_sum4(acc), W = warp_sum4(ws);
    const int q = lane >> 3;
    if (PARTS > 1) {
        __shared__ double s_sum[PARTS][8];
        if ((lane & 7) == 0) {
            s_sum[part][q] = A;
            s_sum[part][4 + q] = W;
        }
        __syncthreads();
        if (part != 0) return;
        A = W = 0.0;
        for (int p = 0; p < PARTS; ++p) {
            A += s_sum[p][q];
            W += s_sum[p][4 + q];
        }
    }
    if ((lane & 7) == 0 && (!(q & 1) || xin) && (!(q >> 1) || yin)) {
        const uint64_t p = pix0 + (q & 1) + (uint64_t)(q >> 1) * nx;
        out[p] = (float)(A / W);
        if (wout) wout[p] = (float)W;
    }
}

}  // namespace

// Launch arguments shared by the kernels of several translation units.
namespace {

// FP16 / BF16 halves of the tensor-core weight operand (fmt 0: FP16, 1: BF16).
__device__ __forceinline__ uint16_t tc_to16(float v, uint32_t fmt) {
    return fmt ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

__device__ __forceinline__ float tc_from16(uint16_t b, uint32_t fmt) {
    return fmt ? __bfloat162float(__ushort_as_bfloat16(b)) : __half2float(__ushort_as_half(b));
}

// hi/lo split of two weights at once (paired conversions): `hi` and `lo` hold
// the 16-bit values of a (low half) and b (high half), the same values as
// tc_to16 of each and of its remainder.
__device__ __forceinline__ void tc_split2(float a, float b, uint32_t fmt, uint32_t &hi, uint32_t &lo) {
    if (fmt) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        const float2 f = __bfloat1622float2(h);
        const __nv_bfloat162 l = __floats2bfloat162_rn(a - f.x, b - f.y);
        hi = *reinterpret_cast<const uint32_t *>(&h);
        lo = *reinterpret_cast<const uint32_t *>(&l);
    } else {
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
        hi = *reinterpret_cast<const uint32_t *>(&h);
        lo = *reinterpret_cast<const uint32_t *>(&l);
    }
}

}  // namespace

struct GroupArgs {
    uint32_t nx, ny, gx;
    uint64_t ngroups;
    uint64_t g0, g1;             // groups handled by this launch
    unsigned long long ebase;    // entry offset of group g0 in the entry buffer
    // entries for the tensor-core builders: the four weights times wscale as
    // 16-bit hi/lo pairs {hi(w0, w1), lo(w0, w1), hi(w2, w3), lo(w2, w3)}
    // (fmt 0: FP16, 1: BF16) instead of four FP32 weights
    uint32_t pack = 0, fmt = 0;
    float wscale = 1.f;
};

// Tiles of kTileX x kTileY pixels (kTileX/2 x kTileY/2 groups) whose union of
// ring windows is staged in shared memory by the accumulation kernels. Per
// tile: first ring r0 of its ring span, the number nr of rings of the span
// that hold union candidates (0 = no samples), the union size U and, per such
// ring c (in ring order), the union interval start ulo[c] and its slot
// base[c] in the staged list; ring_idx maps ring r0 + j of the span to c.
// Pixels much larger than the kernel give long spans with few occupied rings.
constexpr int kTileX = 16, kTileY = 8, kTileMaxRings = 1024, kTileMaxSpan = 4096;
constexpr uint32_t kCapUnknown = 0xffffffffu;
constexpr int kTileGroups = (kTileX / 2) * (kTileY / 2);
// Rings of a tile's span whose per-group windows the tile pass keeps for the
// weight pass (wider spans: the weight pass computes its windows itself).
// A kept window is (lo, hi); lo > hi marks a ring the reference would spin on.
constexpr int kWinSpan = 64;
struct TileArgs {
    uint32_t ntx, nty;
    uint64_t t0;  // first tile of this launch
    int *r0, *nr;
    uint32_t *U, *ulo, *base;  // ulo: [tile][kTileMaxRings], base: [tile][kTileMaxRings + 1]
    uint16_t *ring_idx;        // [tile][kTileMaxSpan]: index c of ring r0 + j (0xffff: no candidates)
    uint32_t *cap;             // per 2x2 group: union candidate count (kCapUnknown: left to group_count_item)
    uint4 *win;                // [tile][kWinSpan][kTileGroups][2]: the group's 4 pixel windows per ring (or null)
    unsigned long long *overflow;  // tiles beyond the ring table (their groups are counted by group_count_item)
    uint32_t pad;  // ring runs take a multiple of `pad` slots (> 1: the tensor-core engine's 8-row boxes)
    unsigned long long *off;    // entry offset of each group, from the tile pass (or null: scanned later)
    unsigned long long *entries;  // with off: entries handed out so far
    unsigned long long *ustat;  // [0]: sum, [1]: largest of the tiles' staged slots U (or null)
};

// hcg_tc.cu: the tensor-core builders' entry format of a field with split
// spectra (GroupArgs::fmt and ::wscale).
void tc_entry_format(const hcg_field *f, uint32_t &fmt, float &wscale);
// hcg_tc.cu: tensor-core accumulation of `ntiles` tiles from T.t0, after
// k_group emitted the entries (slot mode, packed hi/lo weights) and the
// weight sums.
cudaError_t tc_accum(hcg_context *ctx, const hcg_field *f, const GroupArgs &g, const TileArgs &T, uint64_t ntiles,
                     const unsigned long long *off, const uint32_t *cnt, const uint32_t *e_slot, const float4 *e_w,
                     const double *wsum, float *out, uint32_t ostride, float *wout, unsigned long long umax,
                     std::string &why);
// hcg_tc.cu: tensor-core accumulation of `ntiles` tiles whose weights the
// kernel evaluates itself (dense tiles; no entries).
cudaError_t tc_weights(hcg_context *ctx, const hcg_field *f, const GridArgs &a, const GroupArgs &g,
                       const TileArgs &T, uint64_t ntiles, float *out, uint32_t ostride, float *wout,
                       std::string &why);

namespace {

// Union candidates of a 2x2 group (upper bound of its entries), for the groups
// the tile pass left uncounted. Warp-collective.
__device__ __forceinline__ void group_count_item(const GridArgs &a, const GroupArgs &g, uint32_t *__restrict__ cap,
                                                 uint64_t grp, GroupShared &S) {
    const int lane = threadIdx.x & 31;
    if (cap[grp] != kCapUnknown) return;  // counted by the tile pass
    const uint32_t gyi = (uint32_t)(grp / g.gx), gxi = (uint32_t)(grp % g.gx);
    const uint64_t pix0 = (uint64_t)(2 * gyi) * g.nx + 2 * gxi;
    group_load(S, a.prep, pix0, g.nx, 2 * gxi + 1 < g.nx, 2 * gyi + 1 < g.ny);
    const GroupGeo G = group_geo([&](int q) { return &S.prep[q]; });
    unsigned long long count = 0;
    for (int rb = G.r0; rb <= G.r1; rb += 32) {
        uint32_t lo[4], hi[4], ref = 0, skips = 0, glo = 0xffffffffu, ghi = 0;
        group_lane_windows<false>(a, G, rb + lane, pix0, g.nx, lo, hi, ref, skips);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (hi[q] > lo[q]) {
                glo = min(glo, lo[q]);
                ghi = max(ghi, hi[q]);
            }
        }
        if (glo < ghi) count += ghi - glo;
    }
    count = warp_sum_u64(count);
    if (lane == 0) cap[grp] = (uint32_t)count;
}

// Shared memory of a tile's weight pass: per 2x2 group the pixel constants of
// the pair test and the ring range, per ring of the tile's span the shift from
// sample index to slot, and each warp's ring records.
constexpr int kTileShifts = 128, kWeightWarps = 4, kWeightThreads = 32 * kWeightWarps, kWeightCtas = 5;
struct TileGroupShared {
    struct Px {
        PixHalf h[4];
        double cb1[4];
    } px[kTileGroups];
    int r0[kTileGroups], r1[kTileGroups];
    uint32_t shift[kTileShifts];
    GroupRecords rec[kWeightWarps];
};

// FP64 distance and cutoff of every union candidate of the tile's 2x2 groups
// for their 4 pixels, compacted to entries with any non-zero weight, and the
// FP64 weight sums. Block-collective (kWeightThreads, one a pixel): the tile's
// pixels and slot shifts are loaded once, then each warp takes eight groups in
// turn (or `parts` blocks share the tile, block `part` taking every parts-th
// four groups). With a tile
// table (`T.ulo` set) the entries hold the sample's slot in the tile's staged
// list instead of the sample index, and the windows are the ones the tile pass
// kept. What bounds it: the latency of the window and geometry loads at the
// warps that fit, then instruction issue. 500,000 samples, 512 x 500 pixels:
// 305 us with a warp per group, each finding its own tile, pixels and windows.
// PACK: 0 FP32 weights, 1 packed hi/lo pairs (GroupArgs::pack), 2 as g.pack says.
template <int MODE = kPairGeneral, int PACK = 2>
__device__ __forceinline__ void group_tile_item(const GridArgs &a, const GroupArgs &g,
                                                const unsigned long long *__restrict__ off,
                                                uint32_t *__restrict__ e_idx, float4 *__restrict__ e_w,
                                                uint32_t *__restrict__ cnt, double *__restrict__ wsum,
                                                const TileArgs &T, bool tiled, uint64_t tile, uint32_t part,
                                                uint32_t parts, TileGroupShared &S, PairCounts &pc) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tx0 = (uint32_t)(tile % T.ntx) * kTileX, ty0 = (uint32_t)(tile / T.ntx) * kTileY;
    __syncthreads();  // shared state of a previous item is no longer read
    static_assert(kWeightThreads == kTileX * kTileY, "a thread per pixel");
    const uint32_t px = tid % kTileX, py = tid / kTileX;
    const int pg = (py / 2) * (kTileX / 2) + px / 2, pq = (py & 1) * 2 + (px & 1);
    const bool pin = tx0 + px < g.nx && ty0 + py < g.ny;
    if (tid < kTileGroups) {
        S.r0[tid] = 1 << 30;
        S.r1[tid] = -1;
    }
    __syncthreads();
    {
        const PixPrep *src = a.prep + (uint64_t)(ty0 + py) * g.nx + tx0 + px;
        S.px[pg].h[pq] = pin ? src->h : PixHalf{0.0, 0.0, 0.0, 0.0};
        S.px[pg].cb1[pq] = pin ? src->cb1 : 0.0;
        if (pin && src->nr > 0) {
            atomicMin(&S.r0[pg], src->ur);
            atomicMax(&S.r1[pg], src->ur + src->nr - 1);
        }
    }
    // no ring table: a tile without samples, or one spanning too many rings
    const bool slots = tiled && T.nr[tile] > 0;
    const int tr0 = slots ? T.r0[tile] : 0;
    __syncthreads();
    if (slots) {
        const int span = __reduce_max_sync(0xffffffffu, S.r1[lane]) - tr0 + 1;
        for (int j = tid; j < min(span, kTileShifts); j += kWeightThreads) {
            const uint32_t c = T.ring_idx[tile * kTileMaxSpan + j];
            // rings without tile candidates have none for the groups either
            S.shift[j] = c < kTileMaxRings
                             ? T.base[tile * (kTileMaxRings + 1) + c] - T.ulo[tile * kTileMaxRings + c]
                             : 0u;
        }
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
    const uint4 *win = slots && T.win ? T.win + tile * (kWinSpan * kTileGroups * 2) : nullptr;
    // windows of ring (first ring of group gl + lane) kept by the tile pass
    auto kept = [&](int gl, int rb, uint4 &w0, uint4 &w1) {
        const int j = rb + lane - tr0;
        w0 = w1 = make_uint4(0, 0, 0, 0);
        if (win && rb + lane <= S.r1[gl] && j < kWinSpan) {
            w0 = __ldg(win + (j * kTileGroups + gl) * 2);
            w1 = __ldg(win + (j * kTileGroups + gl) * 2 + 1);
        }
    };
    const uint32_t gx0 = tx0 / 2, gy0 = ty0 / 2, gny = (g.ny + 1) / 2;
    uint32_t within = 0;
    for (int gl = part * kWeightWarps + warp; gl < kTileGroups; gl += kWeightWarps * parts) {
        const uint32_t gxi = gx0 + gl % (kTileX / 2), gyi = gy0 + gl / (kTileX / 2);
        if (gxi >= g.gx || gyi >= gny) continue;
        const uint64_t grp = (uint64_t)gyi * g.gx + gxi;
        const bool xin = 2 * gxi + 1 < g.nx, yin = 2 * gyi + 1 < g.ny;
        const uint64_t pix0 = (uint64_t)(2 * gyi) * g.nx + 2 * gxi;
        const int R0 = S.r0[gl], R1 = S.r1[gl];
        const unsigned long long first = off[grp] - g.ebase;
        uint32_t *const ei = e_idx + first;
        float4 *const ew = e_w + first;
        uint32_t n = 0;
        double ws[4] = {0.0, 0.0, 0.0, 0.0};
        for (int rb = R0; rb <= R1; rb += 32) {
            const int k = rb + lane, j = k - tr0;
            uint4 w0, w1;
            kept(gl, rb, w0, w1);
            uint32_t lo[4] = {w0.x, w0.z, w1.x, w1.z}, hi[4] = {w0.y, w0.w, w1.y, w1.w};
            uint32_t shift = 0;  // slot = idx + shift (mod 2^32) for this lane's ring
            if (k <= R1) {
                if (slots) {
                    if (j < kTileShifts) {
                        shift = S.shift[j];
                    } else {
                        const uint32_t c = T.ring_idx[tile * kTileMaxSpan + j];
                        if (c < kTileMaxRings)
                            shift = T.base[tile * (kTileMaxRings + 1) + c] - T.ulo[tile * kTileMaxRings + c];
                    }
                }
                if (!win || j >= kWinSpan) {
                    uint32_t ref = 0, skips = 0;
                    const GroupGeo G = group_geo([&](int q) -> const PixPrep * {
                        return (!(q & 1) || xin) && (!(q >> 1) || yin) ? a.prep + pix0 + (q & 1) + (uint64_t)(q >> 1) * g.nx
                                                                       : nullptr;
                    });
                    group_lane_windows<false>(a, G, k, pix0, g.nx, lo, hi, ref, skips);
                }
            }
            group_rounds<true, MODE>(
                a, S.px[gl].h, S.px[gl].cb1, S.rec[warp], pix0, g.nx, lo, hi, shift, nullptr, 0u,
                [&](float, uint32_t slot, const double w[4], const float wf[4], const bool nz[4]) {
                    bool any = false;
                    float e[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        e[q] = wf[q];
                        ws[q] += w[q];
                        any = any || nz[q];
                        within += nz[q];
                    }
                    if (PACK == 1 || (PACK == 2 && g.pack)) {
                        // the four slots carry {hi(w0, w1), lo(w0, w1), hi(w2, w3), lo(w2, w3)}
                        uint32_t h01, l01, h23, l23;
                        tc_split2(e[0] * g.wscale, e[1] * g.wscale, g.fmt, h01, l01);
                        tc_split2(e[2] * g.wscale, e[3] * g.wscale, g.fmt, h23, l23);
                        e[0] = __uint_as_float(h01);
                        e[1] = __uint_as_float(l01);
                        e[2] = __uint_as_float(h23);
                        e[3] = __uint_as_float(l23);
                    }
                    const unsigned ball = __ballot_sync(0xffffffffu, any);
                    if (any) {
                        const uint32_t at = n + __popc(ball & lt);
                        ei[at] = slot;
                        ew[at] = make_float4(e[0], e[1], e[2], e[3]);
                    }
                    n += __popc(ball);
                });
        }
        const double W = warp_sum4(ws);
        const int q = lane >> 3;
        if (lane == 0) cnt[grp] = n;
        if ((lane & 7) == 0 && (!(q & 1) || xin) && (!(q >> 1) || yin))
            wsum[pix0 + (q & 1) + (uint64_t)(q >> 1) * g.nx] = W;
    }
    pc.add(0, within, 0);
}

// Exclusive scan of n u32 counts into u64 offsets (out[n] = the total), in
// three passes over `parts` contiguous parts of the input, each swept by a
// block of kScanThreads threads in coalesced rows: the part sums, a scan of
// the part sums (one block), then the scan of each part from its base.
constexpr int kScanThreads = 1024;

__device__ __forceinline__ void scan_part(uint64_t n, uint32_t parts, uint32_t p, uint64_t &b, uint64_t &e) {
    const uint64_t per = (n + parts - 1) / parts;
    b = min(n, (uint64_t)p * per);
    e = min(n, b + per);
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and sets `total`. Every thread of the block calls it.
__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long v, unsigned long long &total) {
    __shared__ unsigned long long s_warp[kScanThreads / 32];
    __shared__ unsigned long long s_total;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();  // the shared values of a previous call are no longer read
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        const unsigned long long x = lane < nw ? s_warp[lane] : 0ULL;
        unsigned long long xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long t = __shfl_up_sync(0xffffffffu, xi, o);
            if (lane >= o) xi += t;
        }
        if (lane < nw) s_warp[lane] = xi - x;  // exclusive over the warps
        if (lane == 31) s_total = xi;
    }
    __syncthreads();
    total = s_total;
    return s_warp[w] + incl - v;
}

__device__ __forceinline__ void scan_sums_item(const uint32_t *__restrict__ in, uint64_t n, uint32_t parts,
                                               unsigned long long *__restrict__ psum, uint32_t p) {
    uint64_t b, e;
    scan_part(n, parts, p, b, e);
    unsigned long long v = 0;
    for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) v += in[i];
    unsigned long long tot;
    block_exclusive_scan(v, tot);
    if (threadIdx.x == 0) psum[p] = tot;
}

// One block: psum[0..parts) -> exclusive prefix sums, psum[parts] = total.
__device__ __forceinline__ void scan_psum_item(unsigned long long *__restrict__ psum, uint32_t parts) {
    unsigned long long run = 0;
    for (uint32_t c = 0; c < parts; c += blockDim.x) {
        const uint32_t i = c + threadIdx.x;
        const unsigned long long v = i < parts ? psum[i] : 0ULL;
        unsigned long long tot;
        const unsigned long long ex = block_exclusive_scan(v, tot);
        if (i < parts) psum[i] = run + ex;
        run += tot;
    }
    if (threadIdx.x == 0) psum[parts] = run;
}

__device__ __forceinline__ void scan_apply_item(const uint32_t *__restrict__ in, uint64_t n, uint32_t parts,
                                                const unsigned long long *__restrict__ psum,
                                                unsigned long long *__restrict__ out, uint32_t p) {
    uint64_t b, e;
    scan_part(n, parts, p, b, e);
    unsigned long long run = psum[p];
    for (uint64_t c = b; c < e; c += blockDim.x) {
        const uint64_t i = c + threadIdx.x;
        const unsigned long long v = i < e ? in[i] : 0ULL;
        unsigned long long tot;
        const unsigned long long ex = block_exclusive_scan(v, tot);
        if (i < e) out[i] = run + ex;
        run += tot;
    }
    if (p == parts - 1 && threadIdx.x == 0) out[n] = psum[parts];
}

// FP32 channel accumulation of a group's entries; lane owns 4 channels per
// 128-channel pass. Output [pixel][channel] with row stride `ostride`.
// Warp-collective: every lane passes the same group.
__device__ __forceinline__ void group_accum_item(const GroupArgs &g, const unsigned long long *__restrict__ off,
                                                 const uint32_t *__restrict__ cnt, const uint32_t *__restrict__ e_idx,
                                                 const float4 *__restrict__ e_w, const double *__restrict__ wsum,
                                                 const float *__restrict__ spec, uint32_t nchan, uint32_t cstride,
                                                 float *__restrict__ out, uint32_t ostride,
                                                 float *__restrict__ wout, uint64_t grp) {
    int lane = threadIdx.x & 31;
    uint32_t gyi = (uint32_t)(grp / g.gx), gxi = (uint32_t)(grp % g.gx);
    uint64_t pix[4];
    bool valid[4];
    float inv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t xx = 2 * gxi + (q & 1), yy = 2 * gyi + (q >> 1);
        valid[q] = xx < g.nx && yy < g.ny;
        pix[q] = (uint64_t)yy * g.nx + xx;
        double w = valid[q] ? wsum[pix[q]] : 1.0;
        inv[q] = (float)(1.0 / w);
        if (valid[q] && wout && lane == 0) wout[pix[q]] = (float)w;
    }
    const unsigned long long e0 = off[grp] - g.ebase;
    const uint32_t ne = cnt[grp];
    for (uint32_t c0 = 0; c0 < nchan; c0 += 128) {
        uint32_t c = c0 + 4 * lane;
        float4 acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < cstride) {
            const float *sp = spec + c;
            uint32_t e = 0;
            for (; e + 4 <= ne; e += 4) {
                uint32_t id[4];
                float4 w[4], s[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    id[u] = __ldg(e_idx + e0 + e + u);
                    w[u] = __ldg(e_w + e0 + e + u);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] = __ldg(reinterpret_cast<const float4 *>(sp + (uint64_t)id[u] * cstride));
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float wv[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[q].x = fmaf(wv[q], s[u].x, acc[q].x);
                        acc[q].y = fmaf(wv[q], s[u].y, acc[q].y);
                        acc[q].z = fmaf(wv[q], s[u].z, acc[q].z);
                        acc[q].w = fmaf(wv[q], s[u].w, acc[q].w);
                    }
                }
            }
            for (; e < ne; ++e) {
                uint32_t id = __ldg(e_idx + e0 + e);
                float4 w = __ldg(e_w + e0 + e);
                float4 s = __ldg(reinterpret_cast<const float4 *>(sp + (uint64_t)id * cstride));
                const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[q].x = fmaf(wv[q], s.x, acc[q].x);
                    acc[q].y = fmaf(wv[q], s.y, acc[q].y);
                    acc[q].z = fmaf(wv[q], s.z, acc[q].z);
                    acc[q].w = fmaf(wv[q], s.w, acc[q].w);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!valid[q]) continue;
            const float v[4] = {acc[q].x * inv[q], acc[q].y * inv[q], acc[q].z * inv[q], acc[q].w * inv[q]};
            store_cube4(out, ostride, (uint64_t)g.nx * g.ny, pix[q], c, nchan, v);
        }
    }
}

// Union of the ring windows of all pixels of one tile, per ring, and the
// slot each ring's union starts at in the tile's staged list.
// Block-collective (W warps): a warp
// takes every W-th ring of the tile's span and each lane one 2x2 group, so a
// ring's record is one broadcast load, the chord's bound is formed once for
// four pixels, and the tile's union of a ring is one warp reduction. What bounds
// it: issue of the windows' arithmetic, then the latency of their table
// lookups. 4M samples, 1200 x 1200 pixels: 1034 us with a general window per
// thread and shared-memory atomics per group.
// W: four warps a tile where the tiles fill the GPU (96 registers, 20 warps an
// SM), eight where they do not and the latency of one tile is what counts.
constexpr int kRingCtas = 5;
template <int W, bool TABLES>
__device__ __forceinline__ void tile_rings_item(const GridArgs &a, const GroupArgs &g, const TileArgs &T,
                                                uint64_t tile) {
    __shared__ uint32_t s_lo[kTileMaxSpan], s_hi[kTileMaxSpan];
    __shared__ uint32_t s_cnt[kTileGroups];
    __shared__ unsigned long long s_cand, s_skips;
    __shared__ int s_r0, s_r1;
    const uint32_t tx0 = (uint32_t)(tile % T.ntx) * kTileX, ty0 = (uint32_t)(tile / T.ntx) * kTileY;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t xx = tx0 + 2 * (lane % (kTileX / 2)), yy = ty0 + 2 * (lane / (kTileX / 2));
    const uint64_t pix0 = (uint64_t)yy * g.nx + xx;
    static_assert(kTileGroups == 32, "a lane per group");
    const GroupGeo G = group_geo([&](int q) -> const PixPrep * {
        return xx + (q & 1) < g.nx && yy + (q >> 1) < g.ny ? a.prep + pix0 + (q & 1) + (uint64_t)(q >> 1) * g.nx
                                                            : nullptr;
    });
    __syncthreads();  // shared state of a previous item is no longer read
    if (tid < kTileGroups) s_cnt[tid] = 0;
    if (warp == 0) {
        const int lo = __reduce_min_sync(0xffffffffu, G.r0), hi = __reduce_max_sync(0xffffffffu, G.r1);
        if (lane == 0) {
            s_r0 = lo;
            s_r1 = hi;
            s_cand = s_skips = 0;
        }
    }
    __syncthreads();
    const int r0 = s_r0, nrt = s_r1 - s_r0 + 1;
    // candidate counts of the tile's 2x2 groups (the entries k_group may emit)
    auto write_caps = [&](bool known) {
        if (!T.cap || tid >= kTileGroups) return;
        const uint32_t gxi = (uint32_t)(tile % T.ntx) * (kTileX / 2) + tid % (kTileX / 2);
        const uint32_t gyi = (uint32_t)(tile / T.ntx) * (kTileY / 2) + tid / (kTileX / 2);
        const uint64_t grp = (uint64_t)gyi * g.gx + gxi;
        const bool in = gxi < g.gx && grp < g.ngroups;
        if (in) T.cap[grp] = known ? s_cnt[tid] : kCapUnknown;
        if (T.off && known) {
            // the tile's place among the entries, in the order the tiles come:
            // one atomic a tile instead of a scan of all groups (four launches)
            uint32_t incl = in ? s_cnt[tid] : 0u;
            const uint32_t mine_n = incl;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            unsigned long long first = 0;
            if (lane == 31) first = atomicAdd(T.entries, (unsigned long long)incl);
            first = __shfl_sync(0xffffffffu, first, 31);
            if (in) T.off[grp] = first + incl - mine_n;
        }
    };
    // a span beyond the table keeps no windows and no unions; its groups are
    // counted later, its candidate statistic is taken here all the same
    const bool known = nrt <= kTileMaxSpan;
    unsigned long long cand = 0;
    uint32_t skips = 0, mine = 0;  // mine: the group's union candidates
    for (int j = warp; j < nrt; j += W) {
        const int k = r0 + j;
        uint32_t lo[4], hi[4], ref = 0;
        group_windows_any<TABLES>(a, k, G, pix0, g.nx, lo, hi, ref, skips);
        cand += ref;
        if (!known) continue;
        if (T.win && j < kWinSpan) {
            uint4 *w = T.win + ((tile * kWinSpan + j) * kTileGroups + lane) * 2;
            w[0] = make_uint4(lo[0], hi[0], lo[1], hi[1]);
            w[1] = make_uint4(lo[2], hi[2], lo[3], hi[3]);
        }
        uint32_t glo = 0xffffffffu, ghi = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (hi[q] > lo[q]) {
                glo = min(glo, lo[q]);
                ghi = max(ghi, hi[q]);
            }
        }
        if (glo < ghi) mine += ghi - glo;
        glo = __reduce_min_sync(0xffffffffu, glo);
        ghi = __reduce_max_sync(0xffffffffu, ghi);
        if (lane == 0) {
            s_lo[j] = glo;
            s_hi[j] = ghi;
        }
    }
    // the candidate statistic: the reference windows' lengths (the pairs the
    // reference visits) of every (pixel, ring) of the tile, and the rings the
    // reference would spin on
    if (mine) atomicAdd(&s_cnt[lane], mine);
    cand = warp_sum_u64(cand);
    skips = __reduce_add_sync(0xffffffffu, skips);
    if (lane == 0 && cand) atomicAdd(&s_cand, cand);
    if (lane == 0 && skips) atomicAdd(&s_skips, (unsigned long long)skips);
    __syncthreads();
    if (tid == 0 && s_cand) atomicAdd(&a.stats->pairs_candidate, s_cand);
    if (tid == 0 && s_skips) atomicAdd(&a.stats->ring_skips, s_skips);
    write_caps(nrt <= 0 || known);  // no samples: nothing to count
    if (nrt <= 0 || !known) {
        if (tid == 0) {
            T.r0[tile] = 0;
            T.nr[tile] = 0;
            T.U[tile] = 0;
            if (!known) atomicAdd(T.overflow, 1ULL);
        }
        return;
    }
    if (tid < 32) {  // one warp: compaction of the occupied rings and prefix sums of their lengths
        uint32_t run = 0, count = 0;
        for (int jb = 0; jb < nrt; jb += 32) {
            const int j = jb + tid;
            const bool occ = j < nrt && s_lo[j] < s_hi[j];
            uint32_t len = occ ? s_hi[j] - s_lo[j] : 0;
            if (T.pad > 1) len = (len + T.pad - 1) / T.pad * T.pad;
            uint32_t incl = len;
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            const unsigned ball = __ballot_sync(0xffffffffu, occ);
            const uint32_t c = count + __popc(ball & ((1u << tid) - 1u));
            if (j < nrt) T.ring_idx[tile * kTileMaxSpan + j] = (occ && c < kTileMaxRings) ? (uint16_t)c : 0xffff;
            if (occ && c < kTileMaxRings) {
                T.ulo[tile * kTileMaxRings + c] = s_lo[j];
                T.base[tile * (kTileMaxRings + 1) + c] = run + incl - len;
            }
            run += __shfl_sync(0xffffffffu, incl, 31);
            count += __popc(ball);
        }
        if (tid == 0) {
            if (count > kTileMaxRings) {  // more occupied rings than the table holds
                T.r0[tile] = 0;
                T.nr[tile] = 0;
                T.U[tile] = 0;
                atomicAdd(T.overflow, 1ULL);
            } else {
                T.base[tile * (kTileMaxRings + 1) + count] = run;
                T.r0[tile] = r0;
                T.nr[tile] = (int)count;
                T.U[tile] = run;
                if (T.ustat) {
                    atomicAdd(T.ustat, (unsigned long long)run);
                    atomicMax(T.ustat + 1, (unsigned long long)run);
                }
            }
        }
    }
}

// Shared-memory reads by 32-bit address.
__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds4u(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds1(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// 16-byte asynchronous global -> shared copy (zero-filled when !valid).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// One arrival on `bar` once all of this thread's earlier cp.async copies have
// landed (the barrier's count includes it).
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(sm100::smem_u32(bar)) : "memory");
}
constexpr uint64_t kTileWaitNs = 1000000000ull;  // bound of the FP32 staging ring's barrier waits
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Channel sums of one tile for one slice of kAccumSlice channels. The tile's
// union of candidate spectra (its slots) is staged in shared memory in chunks
// of kAccumRows rows through a ring of kAccumBufs buffers: every thread copies
// its share of a chunk with cp.async and arrives on the chunk's `full` barrier
// when its copies land; each warp arrives on the buffer's `empty` barrier when
// it has summed the chunk, and the chunk kAccumBufs - 2 ahead is staged into a
// buffer only once every warp is done with that buffer's previous chunk.
//
// A warp sums two 2x2 groups, one after the other within a chunk, a lane owning
// four channels: an entry is the same for the whole warp, so nothing diverges.
// A chunk is a band of declination, and a group has entries in about half of
// the chunks; its warp's second group lies two group rows below the first, so
// that most warps have work in most chunks (a warp with two groups of one row
// waited through the other half). Each group's entries come in batches of 32,
// one a lane: the next batch is loaded into registers while the present one is
// summed from shared memory. Channel planes leave through a shared-memory
// transpose, as 64-byte runs (stores from the sums' layout write 4 bytes of
// every 32-byte sector). What bounds it: issue and shared-memory latency at 16
// warps an SM; an entry is six shared-memory wavefronts for 128 channels (four of
// spectra, two of entry) and 26 instructions, 16 of them multiply-adds. Packed
// FP32 pairs (fma.rn.f32x2) gained nothing: they take one of the two FMA pipes.
// 1M samples x 512 channels, 600 x 600 pixels: 3.09 ms (3.70 ms with half a warp
// a group, each thread reading every entry from L2).
//
// Block-collective (kTileThreads; kAccumBufs * kAccumRows * kAccumSlice floats
// of dynamic shared memory). A barrier wait that runs out (1 s) is counted in
// `timeouts` and the item winds down.
constexpr int kAccumBufs = 3, kAccumRows = 128, kAccumSlice = 128, kAccumWarps = 16;
constexpr int kTileThreads = 32 * kAccumWarps;
constexpr int kAccumSmem = kAccumBufs * kAccumRows * kAccumSlice * (int)sizeof(float);
constexpr int kAccumPitch = kTileX * kTileY + 1;  // the transpose's rows (channels) of pixels
static_assert(kTileGroups == 2 * kAccumWarps && kAccumSlice == 128, "two groups a warp, four channels a lane");
static_assert(kAccumSlice * kAccumPitch * (int)sizeof(float) <= kAccumSmem, "the transpose fits the staging ring");
__device__ __forceinline__ void tile_accum_item(const GroupArgs &g, const TileArgs &T,
                                                const unsigned long long *__restrict__ off,
                                                const uint32_t *__restrict__ cnt,
                                                const uint32_t *__restrict__ e_slot,
                                                const float4 *__restrict__ e_w, const double *__restrict__ wsum,
                                                const float *__restrict__ spec, uint32_t nchan, uint32_t cstride,
                                                float *__restrict__ out, uint32_t ostride,
                                                float *__restrict__ wout, uint64_t tile, uint32_t c0,
                                                unsigned long long *timeouts) {
    constexpr int NB = kAccumBufs, CH = kAccumRows;
    static_assert(NB >= 3, "the chunk NB - 2 ahead is staged while one is summed");
    extern __shared__ float4 s_spec[];  // [NB][CH][kAccumSlice / 4]
    __shared__ uint32_t s_ulo[kTileMaxRings], s_base[kTileMaxRings + 1];
    __shared__ float4 s_ew[kTileGroups][32];    // the groups' current batches of entries: weights
    __shared__ __align__(16) uint32_t s_er[kTileGroups][32];  // and slot * row bytes (mod 2^32)
    __shared__ uint64_t s_full[NB], s_empty[NB];
    __shared__ volatile int s_abort;
    __syncthreads();  // shared state of a previous item is no longer read
    const int tid = threadIdx.x;
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const int nrt = T.nr[tile];
    const uint32_t U = T.U[tile];
    for (int j = tid; j < nrt; j += kTileThreads) s_ulo[j] = T.ulo[tile * kTileMaxRings + j];
    for (int j = tid; j <= nrt; j += kTileThreads) s_base[j] = T.base[tile * (kTileMaxRings + 1) + j];
    if (tid == 0) {
        for (int b = 0; b < NB; ++b) {
            sm100::mbar_init(&s_full[b], kTileThreads);
            sm100::mbar_init(&s_empty[b], kAccumWarps);
        }
        s_abort = 0;
        sm100::mbar_fence_init();
    }
    // the warp's groups: rows (0, 2) or (1, 3) of the tile's four group rows
    const uint32_t gxl = warp & 7, gyl = warp >> 3;
    const uint32_t gxi = (uint32_t)(tile % T.ntx) * (kTileX / 2) + gxl;
    const uint32_t gy0 = (uint32_t)(tile / T.ntx) * (kTileY / 2) + gyl;
    constexpr uint32_t kRowBytes = kAccumSlice * 4;
    struct Batch {
        uint64_t e, end;   // next entry to load
        float4 w;          // the next batch's entry of this lane
        uint32_t next;     // and its slot (0xffffffff: none)
        uint32_t slot;     // the present batch's slot of this lane
        uint32_t pos;      // entries of it summed
    } B[2];
    auto load_batch = [&](Batch &b) {
        const bool in = b.e + lane < b.end;
        b.next = in ? __ldg(e_slot + b.e + lane) : 0xffffffffu;
        if (in) b.w = __ldg(e_w + b.e + lane);
        b.e += 32;
    };
    auto next_batch = [&](Batch &b, uint32_t gl) {  // false: the group's entries are all summed
        b.slot = b.next;
        b.pos = 0;
        if (__shfl_sync(0xffffffffu, b.next, 0) == 0xffffffffu) return false;
        __syncwarp();  // the previous batch is no longer read
        s_ew[gl][lane] = b.w;
        s_er[gl][lane] = b.next * kRowBytes;
        load_batch(b);
        __syncwarp();
        return true;
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint64_t grp = (uint64_t)(gy0 + 2 * i) * g.gx + gxi;
        const bool in = gxi < g.gx && grp < g.ngroups;
        B[i].e = in ? off[grp] - g.ebase : 0;
        B[i].end = in ? B[i].e + cnt[grp] : 0;
        B[i].w = make_float4(0.f, 0.f, 0.f, 0.f);
        load_batch(B[i]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) next_batch(B[i], 2 * warp + i);
    float4 acc[2][4];  // [group][pixel of the group]
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][k] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // stage rows [cs, min(U, cs + CH)) into buffer b: each warp takes kRows
    // consecutive rows, its lane r finds row r's sample (the ring j with
    // base[j] <= slot < base[j+1]) once, and the warp's 16-byte copies take
    // their row's sample from that lane; the thread's arrival on full[b]
    // completes when its copies have landed
    constexpr uint32_t kRows = CH / kAccumWarps, kParts = kAccumSlice / 4;
    static_assert(CH % kAccumWarps == 0 && kRows <= 32 && kParts == 32, "a row per copy of a warp");
    const uint32_t pc = c0 + 4 * lane;  // this lane's channels
    const bool pok = pc < cstride;
    const float *src0 = spec + (pok ? pc : 0);
    auto stage = [&](uint32_t cs, int b) {
        const uint32_t ce = min(U, cs + CH), r0 = cs + warp * kRows;
        const uint32_t nr = r0 < ce ? min(kRows, ce - r0) : 0;
        uint32_t idx = 0;
        if (lane < nr) {
            const uint32_t slot = r0 + lane;
            int lo = 0, hi = nrt;
            while (hi - lo > 1) {
                int mid = (lo + hi) >> 1;
                if (s_base[mid] <= slot) lo = mid; else hi = mid;
            }
            idx = s_ulo[lo] + (slot - s_base[lo]);
        }
        float4 *dst = s_spec + ((size_t)b * CH + (r0 - cs)) * kParts + lane;
        for (uint32_t r = 0; r < nr; ++r) {
            const uint32_t ri = __shfl_sync(0xffffffffu, idx, r);
            cp_async16(dst + r * kParts, src0 + (uint64_t)ri * cstride, pok);
        }
        cp_async_arrive(&s_full[b]);
    };
    const uint32_t nchunks = (U + CH - 1) / CH;
    for (uint32_t k = 0; k < NB - 2 && k < nchunks; ++k) stage(k * CH, (int)k);
    for (uint32_t k = 0; k < nchunks; ++k) {
        const uint32_t cs = k * CH, ce = min(U, cs + CH);
        const int b = (int)(k % NB);
        // the chunk NB - 2 ahead, into the buffer of chunk k - 2 once every warp is done with it
        const uint32_t kn = k + NB - 2;
        if (kn < nchunks) {
            const int bn = (int)(kn % NB);
            if (kn >= (uint32_t)NB && !s_abort &&
                !sm100::mbar_wait(&s_empty[bn], ((kn / NB) - 1) & 1, kTileWaitNs)) {
                atomicAdd(timeouts, 1ULL);
                s_abort = 1;
            }
            stage(kn * CH, bn);
        }
        if (!s_abort && !sm100::mbar_wait(&s_full[b], (k / NB) & 1, kTileWaitNs)) {
            atomicAdd(timeouts, 1ULL);
            s_abort = 1;
        }
        if (__any_sync(0xffffffffu, s_abort)) break;
        // shared address of this lane's channels of slot 0 (mod 2^32)
        const uint32_t at0 = sm100::smem_u32(s_spec + (size_t)b * CH * kParts + lane) - cs * kRowBytes;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t gl = 2 * warp + i;
            Batch &t = B[i];
            const uint32_t ew = sm100::smem_u32(&s_ew[gl][0]), er = sm100::smem_u32(&s_er[gl][0]);
            auto fma_entry = [&](const float4 &w, const float4 &x) {
                const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    acc[i][kk].x = fmaf(wv[kk], x.x, acc[i][kk].x);
                    acc[i][kk].y = fmaf(wv[kk], x.y, acc[i][kk].y);
                    acc[i][kk].z = fmaf(wv[kk], x.z, acc[i][kk].z);
                    acc[i][kk].w = fmaf(wv[kk], x.w, acc[i][kk].w);
                }
            };
            for (;;) {
                // entries [pos, lim) of the batch belong to this chunk: slots rise
                // along a group's entries, so they are the lanes below its end
                const uint32_t lim = __popc(__ballot_sync(0xffffffffu, t.slot < ce));
                uint32_t pos = t.pos;
                for (; pos < lim && (pos & 3); ++pos) fma_entry(lds4(ew + 16 * pos), lds4(at0 + lds1(er + 4 * pos)));
                for (; pos + 4 <= lim; pos += 4) {  // four rows' offsets in one read
                    const uint4 r = lds4u(er + 4 * pos);
                    const float4 x0 = lds4(at0 + r.x), x1 = lds4(at0 + r.y), x2 = lds4(at0 + r.z), x3 = lds4(at0 + r.w);
                    fma_entry(lds4(ew + 16 * pos), x0);
                    fma_entry(lds4(ew + 16 * pos + 16), x1);
                    fma_entry(lds4(ew + 16 * pos + 32), x2);
                    fma_entry(lds4(ew + 16 * pos + 48), x3);
                }
                for (; pos < lim; ++pos) fma_entry(lds4(ew + 16 * pos), lds4(at0 + lds1(er + 4 * pos)));
                t.pos = pos;
                if (lim < 32 || !next_batch(t, gl)) break;
            }
        }
        __syncwarp();
        if (lane == 0) sm100::mbar_arrive(&s_empty[b]);  // this warp is done with buffer b
    }
    cp_async_wait_all();  // no copy into the ring outlives the item
    const uint64_t npix = (uint64_t)g.nx * g.ny;
    float *s_t = reinterpret_cast<float *>(s_spec);  // [channel (4 * lane + j at j * 32 + lane)][pixel of the tile]
    // lane 4 i + k has pixel k of group i: weight sum and reciprocal
    float inv_l = 0.f;
    {
        const uint32_t i = (lane >> 2) & 1, k = lane & 3;
        const uint32_t xx = 2 * gxi + (k & 1), yy = 2 * (gy0 + 2 * i) + (k >> 1);
        if (lane < 8 && xx < g.nx && yy < g.ny) {
            const uint64_t p = (uint64_t)yy * g.nx + xx;
            const double ws = wsum[p];
            inv_l = (float)(1.0 / ws);
            if (wout && c0 == 0) wout[p] = (float)ws;
        }
    }
    if (!ostride) __syncthreads();                   // every warp is done with the ring
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t xx = 2 * gxi + (k & 1), yy = 2 * (gy0 + 2 * i) + (k >> 1);
            if (xx >= g.nx || yy >= g.ny) continue;
            const uint64_t p = (uint64_t)yy * g.nx + xx;
            const float inv = __shfl_sync(0xffffffffu, inv_l, 4 * i + k);  // the branch is the warp's
            const float4 A = acc[i][k];
            const float v[4] = {A.x * inv, A.y * inv, A.z * inv, A.w * inv};
            if (ostride) {
                store_cube4(out, ostride, npix, p, pc, nchan, v);
            } else {
                const uint32_t tp = (2 * (gyl + 2 * i) + (k >> 1)) * kTileX + 2 * gxl + (k & 1);
#pragma unroll
                for (int j = 0; j < 4; ++j) s_t[(j * 32 + lane) * kAccumPitch + tp] = v[j];
            }
        }
    }
    if (!ostride) {
        __syncthreads();
        const uint32_t tx0 = (uint32_t)(tile % T.ntx) * kTileX, ty0 = (uint32_t)(tile / T.ntx) * kTileY;
        const uint32_t xx = tx0 + lane % kTileX;
        for (uint32_t c = warp; c < kAccumSlice && c0 + c < nchan; c += kAccumWarps) {
            const float *row = s_t + ((c & 3) * 32 + (c >> 2)) * kAccumPitch;
            float *plane = out + (uint64_t)(c0 + c) * npix;
#pragma unroll
            for (uint32_t h = 0; h < kTileY / 2; ++h) {
                const uint32_t yy = ty0 + 2 * h + lane / kTileX;
                if (xx < g.nx && yy < g.ny) plane[(uint64_t)yy * g.nx + xx] = row[h * 32 + lane];
            }
        }
    }
}

}  // namespace
}  // namespace hcg

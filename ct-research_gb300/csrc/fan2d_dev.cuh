// fan2d_dev.cuh -- per-ray and per-pixel device code of the 2D fan / parallel
// operators, shared by the single-slice kernels (fan2d.cu) and the batched
// uneven-slice kernels (fan_batch.cu).
//
// Forward projection: the Siddon walk of siddon.cuh on a one-slice volume
// (n[2] = 1, no z crossings).
//  * fan (ProjectionFan_2D.cu:19-216): source (C_t - D sin b, C_s + D cos b),
//    ray through the point P on the line through the centre perpendicular to
//    the central ray: d = (P cos b + D sin b, P sin b - D cos b).
//  * parallel (ProjectionParallel_2D.cu:23-243): ray of offset t at angle th,
//    direction (-sin th, cos th) in (x, y) = (width, height) coordinates,
//    through (C_x + t cos th, C_y + t sin th).
// Backprojection: one pixel and a run of views per thread, the sum in a register.
//  * BP2_BACKPROJ (BackprojectionFan2D.cu:7-116): linear interpolation of R at
//    the pixel's detector position P/U times the reference's weight
//    2 * |T1S1 - End|: End is the far point 2*Rscan along the source->pixel
//    line and T1S1 its crossing with the pixel's low t edge (accepted when the
//    crossing's s lies in [0, s_high], as the reference tests) or else its low
//    s edge (t in [0, t_high]); pixel-views with neither add nothing.
//  * BP2_FBPFAN (FBPfan.cu:45-96): filtered R interpolated, times dbeta / U^2.
//  * BP2_FBPPAR (FBPparallel.cu:41-89): filtered R at t = x cos th + y sin th, times dth.
// Detector interpolation: index floor(|P - P0| / PInt), weights from the
// domain values (BackprojectionFan2D.cu:44-53).
#pragma once
#include <type_traits>

#include "ffloat.cuh"
#include "kernels.cuh"
#include "siddon.cuh"

namespace ct {

enum { BP2_BACKPROJ = 0, BP2_FBPFAN = 1, BP2_FBPPAR = 2 };

// Walk set-up of ray r = view * np + bin, computed; false for rays that miss the image.
__device__ __forceinline__ bool fan_ray_setup_compute(const FanGeom &g, long long r, RayWalk &w) {
    const int p = (int)(r % g.np), v = (int)(r / g.np);
    const double2 tr = g.trig_d[v];
    const double sb = tr.x, cb = tr.y;
    const double P = g.Pd[p];
    double src[3], d[3];
    const int n[3] = {g.nt, g.ns, 1};
    const double res[3] = {g.res[0], g.res[1], 1.0};
    if (g.parallel) {
        // x = width axis (t index), y = height axis (s index)
        src[0] = 0.5 * g.size[0] + P * cb + g.smax * sb;
        src[1] = 0.5 * g.size[1] + P * sb - g.smax * cb;
        d[0] = -sb;
        d[1] = cb;
    } else {
        src[0] = 0.5 * g.size[0] - g.D * sb;
        src[1] = 0.5 * g.size[1] + g.D * cb;
        d[0] = P * cb + g.D * sb;
        d[1] = P * sb - g.D * cb;
    }
    src[2] = 0.5;
    d[2] = 0.0;
    const double ires[3] = {g.ires[0], g.ires[1], 1.0}, ext[3] = {g.ext[0], g.ext[1], 1.0};
    return siddon_setup(src, d, n, res, ires, ext, w);
}

// Walk set-up of ray r: from the geometry's set-up table when it has one (the
// same values, stored once per plan), else computed.
__device__ __forceinline__ bool fan_ray_setup(const FanGeom &g, long long r, RayWalk &w) {
    if (!g.ray_tab) return fan_ray_setup_compute(g, r, w);
    const float4 *q = reinterpret_cast<const float4 *>(g.ray_tab + r);
    const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
    const int flags = __float_as_int(q2.z);
    const float inf = __int_as_float(0x7f800000);
    w.a0 = q0.x; w.a1 = q0.y; w.a2 = inf;
    w.n0 = q0.x; w.n1 = q0.y; w.n2 = inf;
    w.d0 = q0.z; w.d1 = q0.w; w.d2 = 0.0f;
    w.k0 = w.k1 = w.k2 = 0.0f;
    w.L = q1.x;
    w.scale = q1.y;
    w.idx = __float_as_int(q1.z);
    w.nseg = __float_as_int(q1.w);
    w.s0 = __float_as_int(q2.x);
    w.s1 = __float_as_int(q2.y);
    w.s2 = 0;
    w.grazing = (flags & 2) != 0;
    return (flags & 1) != 0;
}

// Lanes per ray of the forward projection: rays of a small sinogram are walked
// by kRayParts lanes each (a walk is one chain of ~1.5 n steps; at 90 x 256 rays
// the GPU holds 7 times as many threads), decided by the sinogram alone.
// 128^2, 90 views of 256 bins: 18.3 -> 12 us for the projection with the residual.
constexpr long long kSplitRays = 65536;
__host__ __device__ inline int fan_ray_lanes(const FanGeom &g) {
    return (long long)g.nb * g.np <= kSplitRays ? kRayParts : 1;
}

// Line integral of ray r = view * np + bin, by `lanes` consecutive lanes (each gets
// it; all lanes of the warp take part when lanes > 1); sets `grazing` for rays
// the FP64 re-walk must redo (ref_walk.cu).
__device__ __forceinline__ float fan_ray_value(const FanGeom &g, const float *__restrict__ img, long long r, int lanes,
                                               bool active, bool &grazing) {
    RayWalk w;
    float v = 0.0f;
    grazing = false;
    const unsigned nmax = (unsigned)(g.nt * g.ns - 1);
    if (active && fan_ray_setup(g, r, w)) {
        grazing = w.grazing;
        v = lanes > 1 ? ray_part_2d(w, img, nmax, threadIdx.x % kRayParts) : ray_integral_2d(w, img, nmax);
    }
    if (lanes > 1) {
#pragma unroll
        for (int d = 1; d < kRayParts; d <<= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, d));
    }
    return v;
}

// The reference's weight 2 |T1S1 - End| of one pixel-view in FP64
// (BackprojectionFan2D.cu:56-114), each operation rounded on its own as the
// reference's double arithmetic: End is the point 2 Rscan along the ray from
// the source through the detector point pd (angle atan(pd / Rscan)), T1S1 the
// line's crossing with the pixel's low t edge when its s lies in [0, s_high],
// else with its low s edge when its t lies in [0, t_high]; 0 when neither (the
// reference's thread returns).  Used where the FP32 tests lie within rounding
// distance of those bounds.
static __device__ __noinline__ float fan_chord_fp64(const FanGeom &g, int ti, int si, double sb, double cb, double pd) {
    const double R = g.D, ct = 0.5 * g.size[0], cs = 0.5 * g.size[1];
    const double src_t = __dsub_rn(ct, __dmul_rn(R, sb)), src_s = __dadd_rn(cs, __dmul_rn(R, cb));
    const double th = atan(__ddiv_rn(pd, R));
    const double smax = __dmul_rn(2.0, R);
    const double st = __dmul_rn(smax, sin(th)), cr = __dsub_rn(R, __dmul_rn(smax, cos(th)));
    const double end_t = __dsub_rn(__dadd_rn(ct, __dmul_rn(st, cb)), __dmul_rn(cr, sb));
    const double end_s = __dadd_rn(__dadd_rn(cs, __dmul_rn(st, sb)), __dmul_rn(cr, cb));
    const double dt = __dsub_rn(end_t, src_t), ds = __dsub_rn(end_s, src_s);
    double t2s = __ddiv_rn(ds, dt == 0.0 ? __dadd_rn(dt, 1e-15) : dt);
    double s2t = __ddiv_rn(dt, ds == 0.0 ? __dadd_rn(ds, 1e-15) : ds);
    t2s = fmin(fmax(t2s, -1e16), 1e16);
    s2t = fmin(fmax(s2t, -1e16), 1e16);
    const double tlo = __dmul_rn((double)ti, g.res[0]), thi = __dmul_rn((double)(ti + 1), g.res[0]);
    const double slo = __dmul_rn((double)si, g.res[1]), shi = __dmul_rn((double)(si + 1), g.res[1]);
    const double tlo_s = __dadd_rn(src_s, __dmul_rn(__dsub_rn(tlo, src_t), t2s));
    const double slo_t = __dadd_rn(src_t, __dmul_rn(__dsub_rn(slo, src_s), s2t));
    double T1, S1;
    if (tlo_s >= 0.0 && tlo_s <= shi) {
        T1 = tlo;
        S1 = tlo_s;
    } else if (slo_t >= 0.0 && slo_t <= thi) {
        T1 = slo_t;
        S1 = slo;
    } else {
        return 0.0f;
    }
    const double et = __dsub_rn(T1, end_t), es = __dsub_rn(S1, end_s);
    return (float)__dmul_rn(2.0, __dsqrt_rn(__dadd_rn(__dmul_rn(et, et), __dmul_rn(es, es))));
}

// a >= b and a < b for a float-float value and a float bound
__device__ __forceinline__ bool ff_ge(ff a, float b) { return a.hi > b || (a.hi == b && a.lo >= 0.0f); }
__device__ __forceinline__ bool ff_lt(ff a, float b) { return a.hi < b || (a.hi == b && a.lo < 0.0f); }

// The reference's detector coordinate P / U of pixel (ti, si) in one view in
// float-float (ffloat.cuh), for the pixel-views where the FP32 value lies near
// a decision boundary.  The pixel centre (ti + 1/2) res - size / 2 comes from
// the geometry's float-float constants (fan_geom_derive), so this runs no
// FP64.  One division, by a reciprocal and a float-float correction.
static __device__ __noinline__ ff fan_pd_ff(const FanGeom &g, int ti, int si, float sb, float cb, int wmode) {
    const ff it2 = ff_sub(ff_mul_f(ff{g.res_ff[0].x, g.res_ff[0].y}, (float)ti + 0.5f),
                          ff{g.hsize_ff[0].x, g.hsize_ff[0].y});
    const ff is2 = ff_sub(ff_mul_f(ff{g.res_ff[1].x, g.res_ff[1].y}, (float)si + 0.5f),
                          ff{g.hsize_ff[1].x, g.hsize_ff[1].y});
    const ff P2 = ff_add(ff_mul_f(it2, cb), ff_mul_f(is2, sb));
    if (wmode == BP2_FBPPAR) return P2;
    const ff R2 = {g.D_ff.x, g.D_ff.y};
    const ff den = ff_sub(R2, ff_sub(ff_mul_f(is2, cb), ff_mul_f(it2, sb)));   // Rscan - S
    const ff num = ff_mul(P2, R2);                                             // P / ((Rscan - S) / Rscan)
    const float r = __frcp_rn(den.hi);
    const float q1 = __fmul_rn(num.hi, r);
    const ff rem = ff_sub(num, ff_mul_f(den, q1));
    return ff_fast2sum(q1, __fmul_rn(rem.hi, r));
}

// Interpolated value of pixel (ti, si) in one view, times PInt, where the FP32
// detector coordinate lies near a bin or range boundary: the coordinate in
// float-float, the reference's range test, floor and weights
// |Pd - P[i]|, |P[i+1] - Pd| (BackprojectionFan2D.cu:44-53).
static __device__ __noinline__ float fan_value_near(const FanGeom &g, const float *__restrict__ Rv, int ti, int si,
                                                    float sb, float cb, int wmode) {
    const ff Pd2 = fan_pd_ff(g, ti, si, sb, cb, wmode);
    if (!(ff_ge(Pd2, g.minp) && ff_lt(Pd2, g.maxp))) return 0.0f;
    int p1 = ff_floor(ff_mul(ff_abs(ff_sub(Pd2, ff{g.p0, 0.0f})), ff{g.ipint_ff.x, g.ipint_ff.y}));
    p1 = min(max(p1, 0), g.np - 2);
    const float pa = __ldg(g.Pf + p1), pb = __ldg(g.Pf + p1 + 1);
    const float w1 = fabsf(__fadd_rn(__fsub_rn(Pd2.hi, pa), Pd2.lo));
    const float w0 = fabsf(__fsub_rn(__fsub_rn(pb, Pd2.hi), Pd2.lo));
    return __fmaf_rn(w0, __ldg(Rv + p1), __fmul_rn(w1, __ldg(Rv + p1 + 1)));
}

// 1 / x and 1 / sqrt(x) to 1-2 ulp
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The chord weight of a pixel-view over 2 in FP32, from d = centre - source =
// (dx, dy): the line crosses the pixel's low t edge (side_t) ht / dx of its
// length before the centre, the low s edge hs / dy, so |T1S1 - source| =
// |d| (1 - ht / dx), and End lies 2 Rscan from the source.
__device__ __forceinline__ float fan_chord(float dx, float dy, bool side_t, float ht, float hs, float R2s) {
    const float n2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
    const float n = __fmul_rn(n2, rsqrt_approx(n2));
    const float f = __fmaf_rn(side_t ? -ht : -hs, rcp_approx(side_t ? dx : dy), 1.0f);
    return fabsf(__fmaf_rn(-n, f, R2s));
}

// The low t edge is crossed -ht dy / dx from the centre in s, the low s edge
// -hs dx / dy in t.  The reference accepts the first for s in [0, s_high], i.e.
// for dy / dx in [-rlo, rhi], rlo = hs / ht and rhi = pcs / ht (pcs the centre's s
// from the image edge); where it does not, the second always holds.  a1 =
// dy + rlo dx and a2 = rhi dx - dy have the sign of dx where both bounds hold.
__device__ __forceinline__ bool fan_side_t(float dx, float a1, float a2) {
    return ((__float_as_int(a1) ^ __float_as_int(dx)) | (__float_as_int(a2) ^ __float_as_int(dx))) >= 0;
}

// The chord weight of a pixel-view over 2 near a bound of its side: the side from
// the unit direction (ex, ey) of the source -> detector point line.  The line
// passes through the pixel centre, so its crossing with the low t edge lies
// ds_t = -ht ey / ex from the centre in s, and with the low s edge dt_s = -hs ex / ey
// in t; the reference's tests s in [0, s_high] and t in [0, t_high] are decided on
// these small offsets, and within 1e-5 of a bound by the FP64 construction.
static __device__ __noinline__ float fan_chord_near(const FanGeom &g, int ti, int si, float sb, float cb) {
    const float it = (float)((ti + 0.5) * g.res[0] - 0.5 * g.size[0]);
    const float is = (float)((si + 0.5) * g.res[1] - 0.5 * g.size[1]);
    const float Rs = (float)g.D;
    const float tlo = (float)(ti * g.res[0]), slo = (float)(si * g.res[1]);
    const float ct = (float)(0.5 * g.size[0]), cs = (float)(0.5 * g.size[1]);
    const float pct = (float)((ti + 0.5) * g.res[0]), pcs = (float)((si + 0.5) * g.res[1]);
    const float ht = (float)(0.5 * g.res[0]), hs = (float)(0.5 * g.res[1]);
    const float P = __fmaf_rn(it, cb, __fmul_rn(is, sb)), S = __fmaf_rn(is, cb, -__fmul_rn(it, sb));
    const float Pd = __fdividef(__fmul_rn(P, Rs), __fsub_rn(Rs, S));
    const float ex0 = __fmaf_rn(Pd, cb, __fmul_rn(Rs, sb)), ey0 = __fmaf_rn(Pd, sb, __fmul_rn(-Rs, cb));
    const float inv = rsqrtf(__fmaf_rn(ex0, ex0, __fmul_rn(ey0, ey0)));
    const float ex = __fmul_rn(ex0, inv), ey = __fmul_rn(ey0, inv);
    const float st = __fmaf_rn(-Rs, sb, ct), ss = __fmaf_rn(Rs, cb, cs);
    const float iex = __fdividef(1.0f, ex);
    const float ds_t = __fmul_rn(__fmul_rn(-ht, ey), iex);
    const float c1 = pcs + ds_t, c2 = hs - ds_t;           // s_at >= 0, s_at <= s_high
    bool tie = fabsf(c1) < 1e-5f * (pcs + fabsf(ds_t)) || fabsf(c2) < 1e-5f * (hs + fabsf(ds_t));
    bool none = false;
    float a = __fmul_rn(__fsub_rn(tlo, st), iex);
    if (!(c1 >= 0.0f && c2 >= 0.0f)) {
        const float iey = __fdividef(1.0f, ey);
        const float dt_s = __fmul_rn(__fmul_rn(-hs, ex), iey);
        const float d1 = pct + dt_s, d2 = ht - dt_s;       // t_as >= 0, t_as <= t_high
        tie = tie || fabsf(d1) < 1e-5f * (pct + fabsf(dt_s)) || fabsf(d2) < 1e-5f * (ht + fabsf(dt_s));
        a = __fmul_rn(__fsub_rn(slo, ss), iey);
        none = !(d1 >= 0.0f && d2 >= 0.0f);
    }
    if (tie) {
        const ff pe = fan_pd_ff(g, ti, si, sb, cb, BP2_BACKPROJ);
        return 0.5f * fan_chord_fp64(g, ti, si, (double)sb, (double)cb, (double)pe.hi + (double)pe.lo);
    }
    return none ? 0.0f : fabsf(__fsub_rn(__fmul_rn(2.0f, Rs), a));
}

// One term of fan_warp_sum where an FP32 decision is not safe: the detector
// coordinate in float-float, and, with `tie`, the chord weight near a bound.
template <int WMODE>
__device__ __noinline__ float fan_view_exact(const FanGeom &g, const float *__restrict__ R, int ti, int si, int v,
                                             bool tie) {
    const float2 tr = g.trig_f[v];
    const float sb = tr.x, cb = tr.y;
    const float val = fan_value_near(g, R + (long long)v * g.np, ti, si, sb, cb, WMODE);
    const ff cs2 = ff_mul_f(ff{g.res_ff[1].x, g.res_ff[1].y}, (float)si + 0.5f);
    const float it = ff_sub(ff_mul_f(ff{g.res_ff[0].x, g.res_ff[0].y}, (float)ti + 0.5f),
                            ff{g.hsize_ff[0].x, g.hsize_ff[0].y}).hi;
    const float is = ff_sub(cs2, ff{g.hsize_ff[1].x, g.hsize_ff[1].y}).hi;
    const float Rs = g.D_ff.x;
    if (WMODE == BP2_BACKPROJ) {
        if (tie) return val * fan_chord_near(g, ti, si, sb, cb);
        const float ht = 0.5f * g.res_ff[0].x, hs = 0.5f * g.res_ff[1].x;
        const float dx = __fmaf_rn(Rs, sb, it), dy = __fmaf_rn(-Rs, cb, is);
        const float a1 = __fmaf_rn(__fdividef(hs, ht), dx, dy), a2 = __fmaf_rn(__fdividef(cs2.hi, ht), dx, -dy);
        return val * fan_chord(dx, dy, fan_side_t(dx, a1, a2), ht, hs, __fmul_rn(2.0f, Rs));
    }
    if (WMODE == BP2_FBPFAN) {
        const float lr = __fmul_rn(rcp_approx(__fsub_rn(Rs, __fmaf_rn(is, cb, -__fmul_rn(it, sb)))), Rs);
        return val * __fmul_rn(lr, lr);
    }
    return val;
}

// Views of fan_warp_sum whose gathers are in flight together: 4 measured 12.2 ms
// for a SIRT iteration of 64 uneven slices, 2 12.6 ms; one view at a time (each
// iteration waiting for its own gathers) 13.7 ms.
constexpr int kFanUnroll = 4;

// Sum of views [v0, v1) for the pixels of a warp, one per lane (ti, si), with
// the weighting WMODE and without the view-independent factor of fan_scale.
// All 32 lanes take part; a lane without a pixel passes some pixel and valid =
// false.  queue: 64 words of shared memory of the warp's own.
//
// The bin is the reference's floor(|Pd - P0| / PInt), PInt the spacing of the
// first two samples, with weights |Pd - P[i]| / PInt from the actual sample
// values: a discontinuous rule (float samples drift from the implied grid, by
// ~1e-3 mm over 1024 bins) that an FP32 Pd reproduces except near a bin or
// range boundary (FanGeom::near_q, about 1e-3 of the pixel-views).  Those, the
// detector's first and last bin and the chord weight's ties go to a queue, and
// the warp works off 32 of them at a time (fan_view_exact), one per lane: run
// where they occur, with one or two lanes active, they took 60% of the FBP's
// time and half of the chord weight's.
//
// Issue-bound: 51 instructions per pixel-view (FBP, the queue included) and about 60 (chord
// weight), 69% of the issue slots, against ~160 and 132 of the form this replaced, which divided in IEEE and
// built the unit direction of the line.  One approximate reciprocal of
// Rscan - S serves P / U and the FBP weight 1 / U^2 (the constants multiply the
// sum once, at the end); the floor is an addition rounded down.  Every rounding
// is written out and the order of the sum depends only on the pixels of the
// warp and the views, so the single-slice and the batched builds give
// identical results.
template <int WMODE>
__device__ __forceinline__ float fan_warp_sum(const FanGeom &g, const float *__restrict__ R, int ti, int si,
                                              bool valid, int v0, int v1, unsigned *queue) {
    // pixel centre relative to the rotation centre, and from the image corner
    const ff cs2 = ff_mul_f(ff{g.res_ff[1].x, g.res_ff[1].y}, (float)si + 0.5f);
    const float it = ff_sub(ff_mul_f(ff{g.res_ff[0].x, g.res_ff[0].y}, (float)ti + 0.5f),
                            ff{g.hsize_ff[0].x, g.hsize_ff[0].y}).hi;
    const float is = ff_sub(cs2, ff{g.hsize_ff[1].x, g.hsize_ff[1].y}).hi;
    const float ht = 0.5f * g.res_ff[0].x, hs = 0.5f * g.res_ff[1].x;
    const float Rs = g.D_ff.x;
    const float itR = WMODE == BP2_FBPPAR ? it : __fmul_rn(it, Rs), isR = WMODE == BP2_FBPPAR ? is : __fmul_rn(is, Rs);
    // quotient q = |Pd - P0| / PInt = Pd qs + qo
    const float qs = __fmul_rn(g.psgn, g.ipint_ff.x), qo = -__fmul_rn(g.p0, qs);
    const int np = g.np, lane = threadIdx.x & 31;
    const float near_q = g.near_q, near_f = 0.5f - near_q;
    // bins 1 .. inner take the FP32 path (the bound by np changes no value: with g.inner
    // alone the batch's backprojection spills more, 10.08 instead of 9.92 ms per iteration)
    const unsigned inner = (unsigned)max(min(np - 3, g.inner), 0);
    // Nearer than this to a bound of the chord's side, fan_chord_near decides: three
    // times the FP32 error of dx and dy (e0), and 2e-5 of the offset, since the float sin
    // and cos of a view leave the reference's line up to ~1e-5 mm off the pixel centre,
    // so that both of its tests may fail there
    const float rlo = __fdividef(hs, ht), rhi = __fdividef(cs2.hi, ht);
    const float e0 = 3e-7f * (Rs + g.hsize_ff[0].x + g.hsize_ff[1].x);
    const float e1 = 2.2e-5f * (Rs + g.hsize_ff[0].x + g.hsize_ff[1].x);
    const float tie_lo = fmaf(e0, 1.0f + rlo, e1), tie_hi = fmaf(e0, 1.0f + rhi, e1);
    const float R2s = __fmul_rn(2.0f, Rs);
    const float2 *__restrict__ trig = g.trig_f;
    const int first = np > 2 ? 1 : 0;                    // bin of p1 = 0 below
    const float *__restrict__ Pf = g.Pf + first;
    const float *__restrict__ Rv = R + first;
    float acc = 0.0f;
    int cnt = 0;      // queued terms of the warp
    auto flush = [&](int n) {
        const unsigned e = queue[lane];
        const int owner = e & 31;
        const int oti = __shfl_sync(0xffffffffu, ti, owner), osi = __shfl_sync(0xffffffffu, si, owner);
        const float x = lane < n ? fan_view_exact<WMODE>(g, R, oti, osi, v0 + (int)(e >> 6), (e >> 5) & 1) : 0.0f;
        for (int j = 0; j < n; ++j) {
            const int o = __shfl_sync(0xffffffffu, owner, j);
            const float xj = __shfl_sync(0xffffffffu, x, j);
            if (o == lane) acc = __fadd_rn(acc, xj);
        }
        cnt -= n;
        const unsigned rest = queue[32 + lane];
        __syncwarp();
        queue[lane] = rest;
        __syncwarp();
    };
    // U views from v: their gathers are in flight together, and one vote covers their
    // odd terms
    auto step = [&](auto uc, int v) {
        constexpr int U = decltype(uc)::value;
        float val[U], w[U];
        int p1[U];
        bool odd[U], tie[U], any = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float2 tr = __ldg(trig + v + u);
            const float sb = tr.x, cb = tr.y;
            float Pd = __fmaf_rn(itR, cb, __fmul_rn(isR, sb)), ir = 1.0f;
            if (WMODE != BP2_FBPPAR) {
                // P / U = P Rscan / (Rscan - S); the FBP's quotient corrected by its remainder
                const float den = __fsub_rn(Rs, __fmaf_rn(is, cb, -__fmul_rn(it, sb))), num = Pd;
                ir = rcp_approx(den);
                Pd = __fmul_rn(num, ir);
                if (WMODE == BP2_FBPFAN) Pd = __fmaf_rn(__fmaf_rn(-Pd, den, num), ir, Pd);
            }
            const float q = __fmaf_rn(Pd, qs, qo);
            const float tq = __fadd_rd(q, 8388608.0f);                           // 2^23 + floor(q)
            const float fc = __fsub_rn(q, __fsub_rn(tq, 8388607.5f));            // q - floor(q) - 1/2
            p1[u] = __float_as_int(tq) - 0x4b000001;                             // bin - 1
            odd[u] = fabsf(fc) > near_f || (unsigned)p1[u] >= inner;
            tie[u] = false;
            if (WMODE == BP2_BACKPROJ) {
                const float dx = __fmaf_rn(Rs, sb, it), dy = __fmaf_rn(-Rs, cb, is);
                const float a1 = __fmaf_rn(rlo, dx, dy), a2 = __fmaf_rn(rhi, dx, -dy);
                tie[u] = fabsf(a1) < tie_lo || fabsf(a2) < tie_hi;
                w[u] = fan_chord(dx, dy, fan_side_t(dx, a1, a2), ht, hs, R2s);
                odd[u] = odd[u] || tie[u];
            } else {
                const float lr = __fmul_rn(ir, Rs);                              // 1 / U
                w[u] = __fmul_rn(lr, lr);
            }
            const unsigned pc = min((unsigned)p1[u], inner);                     // for the reads only
            const float *__restrict__ r = Rv + ((long long)(v + u) * np + pc);
            const float w1 = fabsf(__fsub_rn(Pd, __ldg(Pf + pc))), w0 = fabsf(__fsub_rn(__ldg(Pf + pc + 1), Pd));
            val[u] = __fmaf_rn(w0, __ldg(r), __fmul_rn(w1, __ldg(r + 1)));
            any = any || odd[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (!odd[u]) acc = WMODE == BP2_FBPPAR ? __fadd_rn(acc, val[u]) : __fmaf_rn(val[u], w[u], acc);
        if (__any_sync(0xffffffffu, any)) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                // more than a bin off the detector: nothing to add (where q is no bin number, the
                // exact path decides)
                const bool off = near_q < 1.0f && (p1[u] < -2 || p1[u] >= np);
                const bool mine = odd[u] && valid && !off;
                const unsigned push = __ballot_sync(0xffffffffu, mine);
                if (mine)
                    queue[cnt + __popc(push & ((1u << lane) - 1u))] =
                        ((unsigned)(v + u - v0) << 6) | (tie[u] ? 32u : 0u) | (unsigned)lane;
                cnt += __popc(push);
                __syncwarp();
                if (cnt >= 32) flush(32);
            }
        }
    };
    int v = v0;
    for (; v + kFanUnroll <= v1; v += kFanUnroll) step(std::integral_constant<int, kFanUnroll>{}, v);
    for (; v < v1; ++v) step(std::integral_constant<int, 1>{}, v);
    if (cnt > 0) flush(cnt);
    return acc;
}

// The view-independent factor of fan_warp_sum's terms: 1 / PInt of the weights,
// and 2 (chord), dbeta or dtheta.
template <int WMODE>
__device__ __forceinline__ float fan_scale(const FanGeom &g) {
    const float ipint = 1.0f / g.pint;
    if (WMODE == BP2_BACKPROJ) return __fmul_rn(2.0f, ipint);
    return __fmul_rn(ipint, g.bint);
}

// Backprojection of the block's pixels pix0 .. pix0 + fan_bp_pixels(blockDim.x):
// a warp owns 32 consecutive pixels and one of kFanGroups equal runs of the
// views (several, one after the other, where the block has fewer warps), and
// the partial sums meet in shared memory, added in a fixed order, so that the
// result does not depend on the block size.  write(i, sum) stores pixel i.
//
// One thread per pixel over all views left a 256^2 slice with 3.4 warps per
// scheduler and a 128^2 one with fewer warps than schedulers: 227 us (360
// views) and 68 us (90 views).  The 512^2 / 720-view / 1024-bin FBP
// backprojection went from 759 to 320 us with this and fan_warp_sum, the
// batch's from 11.0 to 6.5 ms.
constexpr int kFanGroups = 8;
__host__ __device__ constexpr int fan_bp_pixels(int block) {
    return block / 32 >= kFanGroups ? 32 * (block / 32 / kFanGroups) : 32;
}

template <int WMODE, class Write>
__device__ __forceinline__ void fan_bp_block(const FanGeom &g, const float *__restrict__ R, int pix0, Write &&write) {
    __shared__ float part[kFanGroups][64];
    __shared__ unsigned queue[16][64];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int npix = g.nt * g.ns, nb = g.nb;
    const int tiles = nw >= kFanGroups ? nw / kFanGroups : 1;      // 32-pixel tiles of the block (at most 2)
    const int tile = nw >= kFanGroups ? wid / kFanGroups : 0;
    if (tile < tiles && pix0 + 32 * tile < npix) {
        const int i = pix0 + 32 * tile + lane, ic = min(i, npix - 1);
        const int ti = ic % g.nt, si = ic / g.nt;
        for (int k = nw >= kFanGroups ? wid % kFanGroups : wid; k < kFanGroups; k += nw) {
            const int v0 = (int)((long long)nb * k / kFanGroups), v1 = (int)((long long)nb * (k + 1) / kFanGroups);
            part[k][32 * tile + lane] = fan_warp_sum<WMODE>(g, R, ti, si, i < npix, v0, v1, queue[wid]);
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 32 * tiles; j += blockDim.x) {
        if (pix0 + j >= npix) break;
        float s[kFanGroups];
#pragma unroll
        for (int k = 0; k < kFanGroups; ++k) s[k] = part[k][j];
#pragma unroll
        for (int h = kFanGroups / 2; h > 0; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) s[k] = __fadd_rn(s[k], s[k + h]);
        write(pix0 + j, __fmul_rn(s[0], fan_scale<WMODE>(g)));
    }
}

// Sums of two per-thread FP32 terms over the block into out[0], out[1], for any
// blockDim.x that is a multiple of 32 and at most 1024: FP32 warp sums, FP64
// partials, one barrier and two atomics per block.
__device__ __forceinline__ void block_sum_pair(float a, float b, double *out) {
    __shared__ double part[2][32];
    a = warp_sum(a);
    b = warp_sum(b);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) {
        part[0][wid] = (double)a;
        part[1][wid] = (double)b;
    }
    __syncthreads();
    if (wid < 2 && wid < nw) {
        for (int j = wid; j < 2; j += nw) {
            const double w = warp_sum(lane < nw ? part[j][lane] : 0.0);
            if (lane == 0) atomicAdd(out + j, w);
        }
    }
}

}  // namespace ct

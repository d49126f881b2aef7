// fdkui.cu -- curved-detector (equiangular) short-scan FDK of ImplementUI.cu.
//
// The scanner pipeline of the reference (ImplementUI.cu:6-158): R is double,
// [view][xi][gamma] on an equiangular detector (gamma in radians, xi rows in
// mm at the source-to-detector distance Ds2d).
//  1. Taps per xi row (GFunction :6-22): the S-L kernel of the equiangular
//     detector, 2/(pi dG')^2 at the centre and
//     -2 n^2 / pi^2 / (4n^2 - 1) / sin^2(n dG') at offset n, dG' = dG * prop(xi)
//     with prop = Ds2d / sqrt(Ds2d^2 + xi^2).
//  2. Weight and filter (PreWeightFiltration :25-86): every sample times
//     (D / prop) cos(gamma prop) W, W the Parker weight of
//     (beta prop, b0 prop, gamma prop, fan prop); then the row convolved with
//     its taps, times dG'.
//  3. Backprojection (BackProjection :88-150): per voxel and view, the
//     bilinear sample at gamma = atan(t_rot / (D - s_rot)) and
//     xi = Ds2d tan(asin(z / |voxel - source|)), times dBeta / (dG dXi) / L2 / prop.
//
// GB300 design:
//  * Filter: one block per row.  The weights run in double exactly as the
//    reference orders them (the Parker branch tests decide between 0, a ramp
//    and 1, and at a symmetric detector's edge the reference's own rounding
//    yields NaN rows, reproduced).  The O(LG^2) convolution runs in FP32 on
//    float pairs with exact sums, not in GB300's 1/64-rate FP64; the row goes
//    out as float.
//  * Backprojection: a set-up kernel writes each column-view's record, and one
//    thread per (t, s) column and 16 z sums the views, 160-odd at a time.
//    The row coordinates sit in shared memory.  Per
//    column-view the offset of gamma from its detector sample is computed in
//    float-float (one division, by the tangent-difference identity) since its
//    bilinear weights are differences at the scale of dG ~ 1e-3 rad; the
//    xi position is linear in z (tan(asin(z/sqrt(L2))) = z / sqrt(L2 - z^2),
//    and L2 - z^2 is the in-plane distance), so the per-voxel work is FP32,
//    accumulated in float pairs and written once as double.
#include <cmath>
#include <mutex>
#include <vector>

#include "devbuf.cuh"
#include "ffloat.cuh"
#include "kernels.cuh"

namespace ct {

namespace {

constexpr double kPiUI = 3.141592653589793;

struct UIGeom {
    int lg, lb, lx;               // gammas, views, xi rows
    int nt, ns, nz;               // display: Size[0] x Size[1] x z_length
    double gint, xint, bint;
    double ming, maxg, minx, maxx;
    double g0, x0;
    double b0, fan, D, ds2d;
    double ct, cs, cz, rz;
    // float copies for the backprojection's loop (converted there from the doubles at
    // every use, they kept the FP64 pipe at 88%)
    float x0f, ixintf, minxf, maxxf;
    // and for its set-up: dBeta / (dG dXi), 1 / dG
    float ctf, csf, g0f, cw0f, gscf, ds2df;
    float2 D2;                    // D as a float pair
};

// ---------------------------------------------------------------------------
// filter
// ---------------------------------------------------------------------------
constexpr int kUIFilterBlock = 256;

__device__ __forceinline__ float2 split(double d) {
    const float h = (float)d;
    return make_float2(h, (float)(d - (double)h));
}

// One block per (view, xi) row, 4 consecutive outputs per thread.  Shared
// memory: the weighted row and the row's taps, split into float pairs.
//
// The sums of the pairs' products (a.x + a.y)(c.x + c.y) without a.y c.y run
// exactly in FP32: the row is scaled by a power of two to |w| < 1 and the taps to
// sum |G| <= 1, so every partial sum is within 1 of 0 and, started at 3, the
// running sum s stays in (2, 4), above any product.  Then t = s + a.x c.x
// rounded, t - s is exact, and one more FMA gives the error of t; the errors and
// the two cross products are summed in floats that go into a float pair every 64
// samples.  6 operations per tap (12 with the product's error and TwoSum), and a
// 16-byte load brings 4 taps: FP32-bound, 26.2 -> 14.5 ms at 800 x 80 rows of 936.
__device__ __forceinline__ float block_max(float v, float *part) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) v = fmaxf(v, part[i]);
    return v;
}

// Exponent e with 2^(e-1) <= v < 2^e, in the range of normal powers of two; 0 for 0
// and what is not finite.
__device__ __forceinline__ int scale_exp(float v) {
    return (v > 0.0f && v < __int_as_float(0x7f800000)) ? max(min(ilogbf(v) + 1, 126), -125) : 0;
}

// The cone-tilt proportion of row x (:44-46).
__device__ __forceinline__ double tilt(const UIGeom &g, double xv) {
    return __ddiv_rn(g.ds2d, sqrt(__dadd_rn(__dmul_rn(g.ds2d, g.ds2d), __dmul_rn(xv, xv))));
}

// cos(gamma prop) of every row and sample, which all views share
__global__ void __launch_bounds__(256)
fdkui_cos_kernel(const UIGeom g, const double *__restrict__ gama, const double *__restrict__ xi,
                 double *__restrict__ cosw) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= (long long)g.lx * g.lg) return;
    cosw[i] = cos(__dmul_rn(gama[i % g.lg], tilt(g, xi[i / g.lg])));
}

__global__ void __launch_bounds__(kUIFilterBlock)
fdkui_filter_kernel(const UIGeom g, const double *__restrict__ R, const double *__restrict__ beta,
                    const double *__restrict__ gama, const double *__restrict__ xi, const float2 *__restrict__ taps,
                    const double *__restrict__ cosw, float *__restrict__ rcov) {
    extern __shared__ float4 smu[];
    __shared__ float part[2][kUIFilterBlock / 32];
    const int lg = g.lg, lg4 = (lg + 3) & ~3, fs = 2 * lg - 1;
    const int pad = 4 + ((4 - ((lg + 3) & 3)) & 3);        // taps start at `pad`: lg - 1 + pad is a multiple of 4
    const int gl = (fs + pad + 8 + 3) & ~3;
    float *wh = reinterpret_cast<float *>(smu), *wl = wh + lg4, *Gh = wl + lg4, *Gl = Gh + gl;
    const int row = blockIdx.x;   // view * lx + x
    const int b = row / g.lx, x = row % g.lx;
    const double pr = tilt(g, xi[x]);
    const double bp = __dmul_rn(beta[b], pr), b0p = __dmul_rn(g.b0, pr), mgp = __dmul_rn(g.fan, pr);
    const double dp = __ddiv_rn(g.D, pr), gip = __dmul_rn(g.gint, pr);
    const double *in = R + (long long)row * lg;
    const float2 *tr = taps + (long long)x * fs;
    float gsum = 0.0f, wmax = 0.0f;
    for (int i = threadIdx.x; i < gl; i += blockDim.x) {
        const float2 t = (i >= pad && i < fs + pad) ? tr[i - pad] : make_float2(0.0f, 0.0f);
        Gh[i] = t.x;
        Gl[i] = t.y;
        gsum += fabsf(t.x);
    }
    for (int q = threadIdx.x; q < lg4; q += blockDim.x) {
        float2 v = make_float2(0.0f, 0.0f);
        if (q < lg) {
            const double gp = __dmul_rn(gama[q], pr);
            const double gp2 = __dmul_rn(2.0, gp);
            double W;
            // Parker weight, the reference's tests in its order (:54-61)
            if (bp >= b0p && bp < __dsub_rn(__dadd_rn(b0p, mgp), gp2)) {
                const double sn = sin(__ddiv_rn(__dmul_rn(kPiUI / 4, bp), __dsub_rn(__ddiv_rn(mgp, 2.0), gp)));
                W = __dmul_rn(sn, sn);
            } else if (bp >= __dsub_rn(__dadd_rn(b0p, mgp), gp2) && bp <= __dsub_rn(__dadd_rn(b0p, kPiUI), gp2)) {
                W = 1.0;
            } else if (bp > __dsub_rn(__dadd_rn(b0p, kPiUI), gp2) && bp <= __dadd_rn(__dadd_rn(b0p, kPiUI), mgp)) {
                const double sn = sin(__ddiv_rn(__dmul_rn(kPiUI / 4, __dsub_rn(__dadd_rn(kPiUI, mgp), bp)),
                                                __dadd_rn(__ddiv_rn(mgp, 2.0), gp)));
                W = __dmul_rn(sn, sn);
            } else {
                W = 0.0;
            }
            v = split(__dmul_rn(__dmul_rn(__dmul_rn(in[q], dp), cosw[(long long)x * lg + q]), W));
        }
        wh[q] = v.x;
        wl[q] = v.y;
        wmax = fmaxf(wmax, fabsf(v.x));
    }
    // the sum of the taps' sizes, rounded up
    gsum = warp_sum(gsum);
    if ((threadIdx.x & 31) == 0) part[1][threadIdx.x >> 5] = gsum;
    const int em = scale_exp(block_max(wmax, part[0]));
    gsum = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) gsum += part[1][i];
    const int eg = scale_exp(gsum * 1.0001f);
    const float ms = ldexpf(1.0f, -em), gs = ldexpf(1.0f, -eg);
    for (int q = threadIdx.x; q < lg4; q += blockDim.x) {
        wh[q] *= ms;
        wl[q] *= ms;
    }
    for (int i = threadIdx.x; i < gl; i += blockDim.x) {
        Gh[i] *= gs;
        Gl[i] *= gs;
    }
    __syncthreads();
    float *o = rcov + (long long)row * lg;
    const double unscale = ldexp(1.0, em + eg);
    for (int pb = 4 * threadIdx.x; pb < lg; pb += 4 * blockDim.x) {
        const float *gh = Gh + pad + (lg - 1) + pb, *gq = Gl + pad + (lg - 1) + pb;   // output pb + j, sample q: [j - q]
        float s[4] = {3.0f, 3.0f, 3.0f, 3.0f}, lh[4] = {0.0f, 0.0f, 0.0f, 0.0f}, ll[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float4 hx = *reinterpret_cast<const float4 *>(gh), hy = *reinterpret_cast<const float4 *>(gq);
        for (int q0 = 0; q0 < lg4; q0 += 64) {
            float e[4] = {0.0f, 0.0f, 0.0f, 0.0f}, c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const int q1 = min(q0 + 64, lg4);
#pragma unroll 2
            for (int q = q0; q < q1; q += 4) {
                const float4 lx = *reinterpret_cast<const float4 *>(gh - q - 4);
                const float4 ly = *reinterpret_cast<const float4 *>(gq - q - 4);
                const float4 ax = *reinterpret_cast<const float4 *>(wh + q), ay = *reinterpret_cast<const float4 *>(wl + q);
                const float tx[8] = {lx.x, lx.y, lx.z, lx.w, hx.x, hx.y, hx.z, hx.w};
                const float ty[8] = {ly.x, ly.y, ly.z, ly.w, hy.x, hy.y, hy.z, hy.w};
                const float mx[4] = {ax.x, ax.y, ax.z, ax.w}, my[4] = {ay.x, ay.y, ay.z, ay.w};
#pragma unroll
                for (int d = 0; d < 4; ++d)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float cx = tx[4 + i - d], cy = ty[4 + i - d];
                        const float t = __fmaf_rn(mx[d], cx, s[i]);
                        e[i] = __fadd_rn(e[i], __fmaf_rn(mx[d], cx, __fsub_rn(s[i], t)));
                        c[i] = __fmaf_rn(my[d], cx, __fmaf_rn(mx[d], cy, c[i]));
                        s[i] = t;
                    }
                hx = lx;
                hy = ly;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {       // (lh, ll) += e, += c
                    const float v = j ? c[i] : e[i];
                    const float t = __fadd_rn(lh[i], v), bb = __fsub_rn(t, lh[i]);
                    ll[i] = __fadd_rn(ll[i], __fadd_rn(__fsub_rn(lh[i], __fsub_rn(t, bb)), __fsub_rn(v, bb)));
                    lh[i] = t;
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (pb + i < lg)
                o[pb + i] = (float)__dmul_rn(gip, unscale * (((double)s[i] - 3.0) + ((double)lh[i] + (double)ll[i])));
    }
}

// ---------------------------------------------------------------------------
// backprojection
// ---------------------------------------------------------------------------
constexpr int kUIZ = 16;

// cos, sin of beta and the source position of a view, as float pairs
struct UIView {
    float2 cb, sb, st, ss;
};

// What depends on the (t, s) column and the view alone: detector cell (g1 < 0:
// off the detector) and weights, xi per unit z, dBeta/(dG dXi) sqrt(L2xy), L2xy.
struct __align__(8) UICol {
    float wg1, wg2, kx, cw, l2xy;
    int g1;
};

// The records of views [v0, v0 + nv), one thread per column and `per` views.
// Float-float (ffloat.cuh, ~2^-46) instead of FP64, which runs at 1/64 of the
// FP32 rate: 1.6 ms for 800 views of 512 x 512 columns against 8.5.  (Before it was a
// kernel of its own this ran once per 16 z of a column.)
__global__ void __launch_bounds__(128)
fdkui_setup_kernel(const UIGeom g, const UIView *__restrict__ views, const double *__restrict__ gama,
                   const float2 *__restrict__ tang, const float *__restrict__ dgam, UICol *__restrict__ rec, int v0,
                   int nv, int per) {
    const int t = blockIdx.x * 32 + threadIdx.x;
    const int s = blockIdx.y * 4 + threadIdx.y;
    if (t >= g.nt || s >= g.ns) return;
    const float it = ((float)t - 0.5f) - g.ctf, is = ((float)s - 0.5f) - g.csf;     // exact half integers
    const ff D2 = {g.D2.x, g.D2.y};
    const float g0f = g.g0f, cw0 = g.cw0f, gsc = g.gscf;
    const long long ncol = (long long)g.nt * g.ns;
    const int k0 = blockIdx.z * per, k1 = min(k0 + per, nv);
    for (int k = k0; k < k1; ++k) {
        const UIView vw = views[v0 + k];
        const ff cb = {vw.cb.x, vw.cb.y}, sb = {vw.sb.x, vw.sb.y};
        UICol c{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, -1};
        const ff dt = ff_add(ff_mul_f(cb, it), ff_mul_f(sb, is));
        const ff den = ff_sub(D2, ff_sub(ff_mul_f(cb, is), ff_mul_f(sb, it)));
        // gamma - G_k = atan(u) for a sample k
        auto offset = [&](int q) {
            const ff T = {tang[q].x, tang[q].y};
            const ff num = ff_sub(dt, ff_mul(T, den)), dn = ff_add(den, ff_mul(dt, T));
            const float u = ff_div_r(num, dn, __fdividef(1.0f, dn.hi)).hi;
            return u - u * u * u * (1.0f / 3.0f);
        };
        // gamma = atan(dt / den).  Its bilinear weights are differences at the
        // scale of dG, so the offset from a sample is computed from the
        // tangent-difference identity: gamma - G_k = atan(u),
        // u = (dt - T_k den) / (den + dt T_k), T_k = tan(G_k), |u| <~ dG, and
        // atan(u) = u - u^3/3 to 1e-16.  An FP32 atan picks the cell.
        const float gf = atanf(dt.hi / den.hi);
        int g1 = (int)floorf(fabsf(gf - g0f) * gsc);
        g1 = min(max(g1, 0), g.lg - 2);
        float dg = dgam[g1], del = offset(g1);
        // one step to the neighbouring cell if the estimate missed
        const float sg = dg >= 0.0f ? 1.0f : -1.0f;
        const int step = (sg * del < 0.0f && g1 > 0) ? -1 : ((sg * del > sg * dg && g1 < g.lg - 2) ? 1 : 0);
        if (step != 0) {
            g1 += step;
            dg = dgam[g1];
            del = offset(g1);
        }
        // inside an inner cell: on the detector
        bool on = g1 > 0 && g1 < g.lg - 2 && sg * del >= 0.0f && sg * del <= sg * dg;
        if (!on) {
            const double gm = gama[g1] + (double)del;
            on = gm >= g.ming && gm < g.maxg;
        }
        if (on) {
            const float ex = ff_sub(ff{it, 0.0f}, ff{vw.st.x, vw.st.y}).hi;
            const float es = ff_sub(ff{is, 0.0f}, ff{vw.ss.x, vw.ss.y}).hi;
            const float l2xy = fmaf(ex, ex, es * es);
            const float rxy = sqrtf(l2xy);
            c = UICol{fabsf(del), fabsf(dg - del), g.ds2df / rxy, cw0 * rxy, l2xy, g1};
        }
        rec[k * ncol + (long long)s * g.nt + t] = c;
    }
}

// Views [v0, v0 + nv) of columns with the records rec.  The sums of earlier
// views come from part (float pairs) unless `first`, and go back to it, or, with
// `last`, into the display.
// 8 blocks per SM (64 registers): 48.0 ms for filter and backprojection of 936 x 80 x
// 800 into 512 x 512 x 50, against 52.2 / 56.8 / 63.2 ms at 6 / 5 / 4.
__global__ void __launch_bounds__(128, 8)
fdkui_bp_kernel(const UIGeom g, const UICol *__restrict__ rec, const float *__restrict__ xif,
                const float *__restrict__ rcov, float2 *__restrict__ part, double *__restrict__ disp, int v0, int nv,
                bool first, bool last) {
    // detector-row coordinate pairs (xi[x], xi[x+1]) for the row weights
    extern __shared__ float2 xrow[];
    for (int x = threadIdx.x + 32 * threadIdx.y; x < g.lx - 1; x += 128) xrow[x] = make_float2(xif[x], xif[x + 1]);
    __syncthreads();
    const int t = blockIdx.x * 32 + threadIdx.x;
    const int s = blockIdx.y * 4 + threadIdx.y;
    const int z0 = blockIdx.z * kUIZ;
    if (t >= g.nt || s >= g.ns) return;
    const int nzc = min(kUIZ, g.nz - z0);
    const long long plane = (long long)g.ns * g.nt;
    const long long o0 = ((long long)z0 * g.ns + s) * g.nt + t;
    float izs[kUIZ];
    float acc_h[kUIZ], acc_l[kUIZ];
#pragma unroll
    for (int k = 0; k < kUIZ; ++k) {
        izs[k] = (float)((z0 + k - 0.5) * g.rz - g.cz);
        // held in its register: the compiler recomputed it in FP64 at every view
        asm volatile("" : "+f"(izs[k]));
        const float2 a = (!first && k < nzc) ? part[o0 + k * plane] : make_float2(0.0f, 0.0f);
        acc_h[k] = a.x;
        acc_l[k] = a.y;
    }
    const float x0 = g.x0f, ixint = g.ixintf, minx = g.minxf, maxx = g.maxxf;
    const float sx = (g.lx > 1 && xif[g.lx - 1] < xif[0]) ? -1.0f : 1.0f;
    const long long vstride = (long long)g.lx * g.lg;
    rec += (long long)s * g.nt + t;
    UICol cn = *rec;
    for (int v = 0; v < nv; ++v) {
        const UICol c = cn;
        if (v + 1 < nv) {          // the next view's record, ahead of this one's work
            rec += plane;
            cn = *rec;
        }
        if (c.g1 < 0) continue;
        const float wg1 = c.wg1, wg2 = c.wg2, kx = c.kx, cw = c.cw, l2xy = c.l2xy;
        const float *rv = rcov + (long long)(v0 + v) * vstride + c.g1;
#pragma unroll
        for (int k = 0; k < kUIZ; ++k) {
            const float iz = izs[k];
            const float X = kx * iz;
            if (k >= nzc || !(X >= minx && X < maxx)) continue;
            // floor by an addition rounded down: the floor and float-to-int instructions run
            // at the FP64 pipe's rate, and kept it at 86%
            const int x1 = min(__float_as_int(__fadd_rd(fabsf(X - x0) * ixint, 8388608.0f)) - 0x4b000000, g.lx - 2);
            const float2 xd = xrow[x1];
            const float wx1 = sx * (X - xd.x), wx2 = sx * (xd.y - X);
            const float *r1 = rv + x1 * g.lg, *r2 = r1 + g.lg;
            const float val = wx2 * fmaf(wg2, __ldg(r1), wg1 * __ldg(r1 + 1)) +
                              wx1 * fmaf(wg2, __ldg(r2), wg1 * __ldg(r2 + 1));
            const float l2 = fmaf(iz, iz, l2xy);
            const float r = rsqrtf(l2);
            const float term = val * (cw * r * r * r);      // / L2 / prop = sqrt(L2xy) / L2^1.5
            const float tt = acc_h[k] + term;
            const float bb = tt - acc_h[k];
            acc_l[k] += (acc_h[k] - (tt - bb)) + (term - bb);
            acc_h[k] = tt;
        }
    }
#pragma unroll
    for (int k = 0; k < kUIZ; ++k)
        if (k < nzc) {
            if (last) disp[o0 + k * plane] = (double)acc_h[k] + (double)acc_l[k];
            else part[o0 + k * plane] = make_float2(acc_h[k], acc_l[k]);
        }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
struct UIState {
    DevBuf beta, gama, tang, dgam, xi, xif, taps, views, rcov, R, disp, cosw, rec, part;
    // the end of the last call, which used the tables and workspaces, and its device
    cudaEvent_t used = nullptr;
    int dev = -1;
    void release() {
        if (used) {
            cudaEventSynchronize(used);
            cudaEventDestroy(used);
        }
        used = nullptr;
        dev = -1;
        for (DevBuf *b : {&beta, &gama, &tang, &dgam, &xi, &xif, &taps, &views, &rcov, &R, &disp, &cosw, &rec,
                          &part})
            b->release();
    }
    // Buffers of the current device.
    int begin() {
        int d = 0;
        CT_CUDA(cudaGetDevice(&d), "cudaGetDevice");
        if (dev != d) release();
        dev = d;
        if (!used) CT_CUDA(cudaEventCreateWithFlags(&used, cudaEventDisableTiming), "FDKUI: event");
        return CT_OK;
    }
    // The kernels of the last call have read the tables and left the workspaces, on whatever
    // stream it ran (the copies of the tables do not wait for a non-blocking one).
    int wait() {
        CT_CUDA(cudaEventSynchronize(used), "FDKUI: tables in use");
        return CT_OK;
    }
};
std::mutex g_ui_mutex;
UIState &ui_state() {
    static UIState st;
    return st;
}

// Equiangular S-L taps per xi row in double as GFunction computes them, as float pairs.
std::vector<float2> ui_taps(const UIGeom &g, const double *xi) {
    const int fs = 2 * g.lg - 1;
    std::vector<float2> out((size_t)g.lx * fs);
    for (int x = 0; x < g.lx; ++x) {
        const double gp = g.gint * (g.ds2d / std::sqrt(1.0 * g.ds2d * g.ds2d + 1.0 * xi[x] * xi[x]));
        float2 *row = out.data() + (size_t)x * fs;
        auto put = [&](int i, double v) {
            row[i].x = (float)v;
            row[i].y = (float)(v - (double)row[i].x);
        };
        put(g.lg - 1, 2.0 / (1.0 * (kPiUI * gp) * (kPiUI * gp)));
        for (int n = 1; n < g.lg; ++n) {
            const double sn = std::sin(n * gp);
            const double v = -2.0 * (1.0 * n * n) / (1.0 * kPiUI * kPiUI) / (4 * (1.0 * n * n) - 1) / (1.0 * sn * sn);
            put(g.lg - 1 - n, v);
            put(g.lg - 1 + n, v);
        }
    }
    return out;
}

int ui_make(UIGeom &g, const double *xi, const double *gama, const double *beta, double b0, double fan, double D,
            double ds2d, int lg, int lb, int lx, const int *size, int nz) {
    CT_REQUIRE(xi && gama && beta && size, "FDKUI: null argument");
    CT_REQUIRE(lg >= 2 && lb >= 2 && lx >= 2, "FDKUI: at least 2 gammas, views and xi rows");
    CT_REQUIRE(lg <= 4096, "FDKUI: at most 4096 gammas per row");
    CT_REQUIRE((long long)lb * lx < (1LL << 31), "FDKUI: too many rows");
    CT_REQUIRE(size[0] > 0 && size[1] > 0 && size[2] > 0 && nz > 0, "FDKUI: display sizes must be positive");
    CT_REQUIRE(size[1] <= 65535 * 4, "FDKUI: Size[1] too large");
    CT_REQUIRE(D > 0 && ds2d > 0, "FDKUI: distances must be positive");
    for (int i = 0; i < lg; ++i) CT_REQUIRE(std::isfinite(gama[i]), "FDKUI: non-finite Gamadomain");
    for (int i = 0; i < lx; ++i) CT_REQUIRE(std::isfinite(xi[i]), "FDKUI: non-finite Xigamadomain");
    for (int i = 0; i < lb; ++i) CT_REQUIRE(std::isfinite(beta[i]), "FDKUI: non-finite BetaScanRange");
    g = UIGeom{};
    g.lg = lg; g.lb = lb; g.lx = lx;
    g.nt = size[0]; g.ns = size[1]; g.nz = nz;
    g.gint = std::fabs(gama[1] - gama[0]);
    g.xint = std::fabs(xi[1] - xi[0]);
    g.bint = std::fabs(beta[1] - beta[0]);
    g.maxg = std::max(gama[0], gama[lg - 1]);
    g.ming = std::min(gama[0], gama[lg - 1]);
    g.maxx = std::max(xi[0], xi[lx - 1]);
    g.minx = std::min(xi[0], xi[lx - 1]);
    g.g0 = gama[0];
    g.x0 = xi[0];
    g.b0 = b0; g.fan = fan; g.D = D; g.ds2d = ds2d;
    // integer halves of the integer extents, as the reference divides them (:103-105)
    g.ct = size[0] / 2;
    g.cs = size[1] / 2;
    g.cz = size[2] / 2;
    g.rz = 1.0 * size[2] / nz;
    g.x0f = (float)g.x0;
    g.ixintf = (float)(1.0 / g.xint);
    g.minxf = (float)g.minx;
    g.maxxf = (float)g.maxx;
    g.ctf = (float)g.ct;
    g.csf = (float)g.cs;
    g.g0f = (float)g.g0;
    g.cw0f = (float)(g.bint / (g.gint * g.xint));
    g.gscf = (float)(1.0 / g.gint);
    g.ds2df = (float)g.ds2d;
    g.D2 = ff_split_host(g.D);
    CT_REQUIRE(g.gint > 0 && g.xint > 0, "FDKUI: domains must have a non-zero step");
    return CT_OK;
}

// The tables of the backprojection, and with `filter` the filter's taps (a sine per tap and row).
int ui_upload(UIState &S, const UIGeom &g, const double *xi, const double *gama, const double *beta, bool filter) {
    std::vector<float> xf(g.lx);
    for (int i = 0; i < g.lx; ++i) xf[i] = (float)xi[i];
    std::vector<UIView> vw(g.lb);
    for (int v = 0; v < g.lb; ++v) {
        const double b = beta[v];
        vw[v] = UIView{ff_split_host(std::cos(b)), ff_split_host(std::sin(b)), ff_split_host(g.D * std::cos(b + kPiUI / 2)),
                       ff_split_host(g.D * std::sin(b + kPiUI / 2))};
    }
    // per gamma sample: tan(G_k) and the cell width G_{k+1} - G_k
    std::vector<float2> tg(g.lg);
    std::vector<float> dg(g.lg, 0.0f);
    for (int k = 0; k < g.lg; ++k) {
        tg[k] = ff_split_host(std::tan(gama[k]));
        if (k + 1 < g.lg) dg[k] = (float)(gama[k + 1] - gama[k]);
    }
    const std::vector<float2> taps = filter ? ui_taps(g, xi) : std::vector<float2>();
    int s;
    if ((s = S.wait())) return s;
    if (filter && (s = upload(S.taps, taps.data(), taps.size()))) return s;
    if ((s = upload(S.tang, tg.data(), tg.size())) || (s = upload(S.dgam, dg.data(), dg.size()))) return s;
    if ((s = upload(S.beta, beta, (size_t)g.lb)) || (s = upload(S.gama, gama, (size_t)g.lg)) ||
        (s = upload(S.xi, xi, (size_t)g.lx)) || (s = upload(S.xif, xf.data(), xf.size())) ||
        (s = upload(S.views, vw.data(), vw.size())))
        return s;
    return CT_OK;
}

int ui_filter(UIState &S, const UIGeom &g, const double *d_R, float *d_rcov, cudaStream_t st) {
    const size_t smem = sizeof(float) * 2 * (size_t)(((g.lg + 3) & ~3) + ((2 * g.lg - 1 + 18) & ~3));
    if (smem > 48 * 1024)
        CT_CUDA(cudaFuncSetAttribute(fdkui_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                "fdkui filter smem attribute");
    if (int s = S.cosw.ensure(sizeof(double) * (size_t)g.lx * g.lg)) return s;
    fdkui_cos_kernel<<<(unsigned)(((long long)g.lx * g.lg + 255) / 256), 256, 0, st>>>(
        g, S.gama.as<double>(), S.xi.as<double>(), S.cosw.as<double>());
    CT_LAUNCH_CHECK("fdkui_cos_kernel");
    fdkui_filter_kernel<<<g.lb * g.lx, kUIFilterBlock, smem, st>>>(g, d_R, S.beta.as<double>(), S.gama.as<double>(),
                                                                   S.xi.as<double>(), S.taps.as<float2>(),
                                                                   S.cosw.as<double>(), d_rcov);
    CT_LAUNCH_CHECK("fdkui_filter_kernel");
    CT_CUDA(cudaEventRecord(S.used, st), "FDKUI: event");
    return CT_OK;
}

// Column-view records held at a time (170 views of 512 x 512 columns)
constexpr size_t kUIRecBytes = size_t(1) << 30;

int ui_bp(UIState &S, const UIGeom &g, const float *d_rcov, double *d_disp, cudaStream_t st) {
    dim3 grid((g.nt + 31) / 32, (g.ns + 3) / 4, (g.nz + kUIZ - 1) / kUIZ), block(32, 4);
    CT_REQUIRE(grid.z <= 65535, "FDKUI: z_length too large");
    const size_t smem = sizeof(float2) * (size_t)g.lx;
    CT_REQUIRE(smem <= 48 * 1024, "FDKUI: at most 6144 detector rows");
    const size_t ncol = (size_t)g.nt * g.ns;
    const int chunk = (int)std::max<size_t>(1, std::min<size_t>(g.lb, kUIRecBytes / (sizeof(UICol) * ncol)));
    const size_t need_rec = sizeof(UICol) * ncol * chunk, need_part = chunk < g.lb ? sizeof(float2) * ncol * g.nz : 0;
    int s;
    if ((s = S.rec.ensure(need_rec)) || (s = S.part.ensure(need_part))) return s;
    for (int v0 = 0; v0 < g.lb; v0 += chunk) {
        const int nv = std::min(chunk, g.lb - v0);
        int per = 8;
        while (per > 1 && ncol * ((nv + per - 1) / per) < 1024ull * sm_count()) per /= 2;
        per = std::max(per, (nv + 65534) / 65535);
        const dim3 sgrid(grid.x, grid.y, (nv + per - 1) / per);
        fdkui_setup_kernel<<<sgrid, block, 0, st>>>(g, S.views.as<UIView>(), S.gama.as<double>(), S.tang.as<float2>(),
                                                    S.dgam.as<float>(), S.rec.as<UICol>(), v0, nv, per);
        CT_LAUNCH_CHECK("fdkui_setup_kernel");
        fdkui_bp_kernel<<<grid, block, smem, st>>>(g, S.rec.as<UICol>(), S.xif.as<float>(), d_rcov,
                                                   S.part.as<float2>(), d_disp, v0, nv, v0 == 0, v0 + nv == g.lb);
        CT_LAUNCH_CHECK("fdkui_bp_kernel");
    }
    CT_CUDA(cudaEventRecord(S.used, st), "FDKUI: event");
    return CT_OK;
}

}  // namespace

// Free the device buffers the drop-in keeps between calls (ct_dropin_release).
void fdkui_release_cache() {
    std::lock_guard<std::mutex> lk(g_ui_mutex);
    ui_state().release();
}

}  // namespace ct

using namespace ct;

extern "C" {

int ct_fdkui_filter(const double *d_R, float *d_Rcov, const double *Xigamadomain, const double *Gamadomain,
                    const double *BetaScanRange, double betaStartAngle, double MaxGama, double Distance,
                    double Distance_s2d, int LGama, int LBeta, int LXigama, void *stream) {
    CT_REQUIRE(d_R && d_Rcov, "ct_fdkui_filter: null argument");
    const int one[3] = {1, 1, 1};
    UIGeom g;
    int s = ui_make(g, Xigamadomain, Gamadomain, BetaScanRange, betaStartAngle, MaxGama, Distance, Distance_s2d,
                    LGama, LBeta, LXigama, one, 1);
    if (s) return s;
    std::lock_guard<std::mutex> lk(g_ui_mutex);
    UIState &S = ui_state();
    if ((s = S.begin()) || (s = ui_upload(S, g, Xigamadomain, Gamadomain, BetaScanRange, true)))
        return s;
    return ui_filter(S, g, d_R, d_Rcov, as_stream(stream));
}

int ct_fdkui_bp(const float *d_Rcov, double *d_Display, const double *Xigamadomain, const double *Gamadomain,
                const double *BetaScanRange, double Distance, double Distance_s2d, int LGama, int LBeta,
                int LXigama, const int *Size, int z_length, void *stream) {
    CT_REQUIRE(d_Rcov && d_Display, "ct_fdkui_bp: null argument");
    UIGeom g;
    int s = ui_make(g, Xigamadomain, Gamadomain, BetaScanRange, 0.0, 0.0, Distance, Distance_s2d, LGama, LBeta,
                    LXigama, Size, z_length);
    if (s) return s;
    std::lock_guard<std::mutex> lk(g_ui_mutex);
    UIState &S = ui_state();
    if ((s = S.begin()) || (s = ui_upload(S, g, Xigamadomain, Gamadomain, BetaScanRange, false)))
        return s;
    return ui_bp(S, g, d_Rcov, d_Display, as_stream(stream));
}

int ct_FDKUI(double *Display, const double *R, const double *Xigamadomain, const double *Gamadomain,
             const double *BetaScanRange, double betaStartAngle, double MaxGama, double Distance,
             double Distance_s2d, int LGama, int LBeta, int LXigama, const int *Size, int z_length) {
    CT_REQUIRE(Display && R, "ct_FDKUI: null argument");
    UIGeom g;
    int s = ui_make(g, Xigamadomain, Gamadomain, BetaScanRange, betaStartAngle, MaxGama, Distance, Distance_s2d,
                    LGama, LBeta, LXigama, Size, z_length);
    if (s) return s;
    std::lock_guard<std::mutex> lk(g_ui_mutex);
    UIState &S = ui_state();
    const size_t nr = (size_t)LGama * LBeta * LXigama, nd = (size_t)Size[0] * Size[1] * z_length;
    if ((s = S.begin()) || (s = ui_upload(S, g, Xigamadomain, Gamadomain, BetaScanRange, true)) || (s = S.R.ensure(nr * sizeof(double))) ||
        (s = S.rcov.ensure(nr * sizeof(float))) || (s = S.disp.ensure(nd * sizeof(double))))
        return s;
    CT_CUDA(cudaMemcpy(S.R.ptr, R, nr * sizeof(double), cudaMemcpyHostToDevice), "H2D projections");
    if ((s = ui_filter(S, g, S.R.as<double>(), S.rcov.as<float>(), nullptr)) ||
        (s = ui_bp(S, g, S.rcov.as<float>(), S.disp.as<double>(), nullptr)))
        return s;
    CT_CUDA(cudaMemcpy(Display, S.disp.ptr, nd * sizeof(double), cudaMemcpyDeviceToHost), "D2H display");
    return CT_OK;
}

}  // extern "C"

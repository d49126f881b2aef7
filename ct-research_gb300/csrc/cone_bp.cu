// cone_bp.cu -- voxel-driven cone-beam backprojection for sm_103a.
//
// Two weightings of the same bilinear detector interpolation:
//  * CHORD (Backprojection3D.cu:8-291): each voxel-view adds
//      bilinear(R) * 2 * |entry - centre|, the chord of the source->voxel-centre
//      line through the voxel.  For a line through the centre the chord is
//      2 * min_a(h_a / |d_a|) * |d| (h = half voxel, d = centre - source),
//      which equals the reference's low-face construction.
//  * FDK (FDK.cu:50-126): bilinear(filtered R) * LR^2 * dbeta, where
//      LR = D / (D - dect_s); in STICKY mode a voxel whose projection leaves
//      the detector re-adds the last in-range value of its column, as the
//      reference does because it never resets Display_pBeta (:73, :100-123).
//
// Layout: each view's projection is first repacked into pairs,
//   Q[v][x][p] = (R[x][p], R[x][p+1]),
// so that one aligned 8-byte load gives a detector row's two taps.
//
// Interpolation follows the reference's discontinuous index rule exactly:
// column floor(|P - P0| / PInt) and row floor(|xi - xi0| / XigamaInt), with
// PInt and XigamaInt the spacing of the first two (float) samples and the
// weights |P - P[i]| / PInt, |xi - xi[j]| / XigamaInt from the actual sample
// values (Backprojection3D.cu:73-87).  Float samples drift from that implied
// grid (by ~1e-3 mm across a 512-row detector), so an index one off changes a
// weight by up to ~4e-3: the column coordinate is computed per column-view in
// float-float (ffloat.cuh), and the row quotient, affine in z, is stepped in
// 64-bit fixed point with a per-row table of the samples' own quotients.
//
// Two kernels.  What depends on the (t, s) column and the view alone (detector
// column and weights, row quotient and its step per z, the z range on the
// detector, the chord factor and its ties) is a 32-byte record that
// cone_bp_setup_kernel writes once per column-view; it used to be recomputed by
// each of the column's nz / 32 threads, 250 of 1030 instructions per thread and
// view.  cone_bp_kernel's threads own one column and ZC consecutive z; the view
// loop runs inside the thread with the ZC sums in registers, and each voxel is
// written once at the end (no atomics, deterministic).  The fused SIRT variant
// writes clamp(x + lambda * bp / (colsum + eps), lo, hi) instead of bp.
#include "cone_geom.cuh"
#include "ffloat.cuh"

namespace ct {

namespace {

constexpr int BP_BX = 32;          // t per block (one warp)
constexpr int BP_BY = 4;           // s per block
// z per thread (register accumulators) and the blocks per SM its registers aim at.
// 32 z share a column-view's record best: 45.2 ms at 512^3 / 360 views and 4 blocks
// (57 at 5, 50 at 6), 47.7 with 16 z and 8 blocks.  A thread sums its views one after
// the other, so a small scan, whose blocks do not fill the GPU several times over, takes
// fewer z per thread: more threads, and fewer of them off the fast path at the
// ends of a column.  us of a backprojection with 16 / 8 / 4 z: 150 x 140 x 110 and 120
// views (1225 blocks at 16 z) 839 / 519 / 610; 64 x 60 x 50 and 90 views (210 at
// 8 z) 434 / 196 / 78; of an FDK of 180 x 170 x 140 and 120 views (2322 at 16 z) 877 / 908
// with 16 / 8 z, of 80 x 70 x 50 and 200 views (378 at 8 z) 517 / 222 / 219.  The lines lie
// between these.  At 8 z, 4 / 5 / 6 / 8 blocks: SIRT3D of 151 x 133 x 97 in 3.33 / 3.37 /
// 3.42 / 3.48 ms (3.81 with 16 z).
constexpr int kZLong = 32, kZShort = 16, kZTiny = 8, kZLeast = 4;
constexpr int bp_min_blocks(int zc) { return zc == kZShort ? 8 : 4; }

int bp_zc(const ConeGeom &g) {
    const long long cols = (long long)((g.nt + BP_BX - 1) / BP_BX) * ((g.ns + BP_BY - 1) / BP_BY), sms = sm_count();
    if (cols * ((g.nz + kZLong - 1) / kZLong) >= 12 * sms) return kZLong;
    if (cols * ((g.nz + kZShort - 1) / kZShort) >= 12 * sms) return kZShort;
    return cols * ((g.nz + kZTiny - 1) / kZTiny) >= 3 * sms ? kZTiny : kZLeast;
}

// Pairs of n consecutive samples; the last sample of a row pairs with 0.
__global__ void __launch_bounds__(256)
pack_pairs_kernel(const float *__restrict__ R, float2 *__restrict__ Q, long long n, int np) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        Q[i] = make_float2(R[i], (int)(i % np) + 1 < np ? R[i + 1] : 0.0f);
}

// The sum of detector row x's two taps, q0 + x * stride bytes their pair (one
// multiply-add for the address).
__device__ __forceinline__ float row_sum(const float2 *q0, unsigned x, unsigned stride, float wa, float wb) {
    unsigned long long a;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(x), "r"(stride), "l"(q0));
    const float2 q = __ldg(reinterpret_cast<const float2 *>(a));
    return fmaf(wa, q.x, wb * q.y);
}

enum { W_CHORD = 0, W_FDK_ZERO = 1, W_FDK_STICKY = 2 };

// FP64 re-evaluation of the reference's detector-range tests for one column
// and view (Backprojection3D.cu:31-43 and :66-71, FDK.cu:80-100):
// P in [minP, maxP) and xi(z) in [minXigama, maxXigama).  Used only when the
// FP32 decision lies within rounding distance of a detector edge; it matters
// most for the sticky FDK value, which is taken at the last in-range z.
__device__ __noinline__ void range_fp64(const ConeGeom &g, int ti, int si, double sb, double cb, bool &pin,
                                        int &zlo, int &zhi) {
    const double it = (ti + 0.5) * g.res[0] - 0.5 * g.size[0];
    const double is = (si + 0.5) * g.res[1] - 0.5 * g.size[1];
    const double dect_t = it * cb + is * sb;
    const double dect_s = -it * sb + is * cb;
    const double lr = g.D / (g.D - dect_s);
    const double P = dect_t * lr;
    pin = (P >= (double)g.minp) && (P < (double)g.maxp);
    const double rz = g.res[2], cz = 0.5 * g.size[2];
    const double mnx = g.minx, mxx = g.maxx;
    int lo = min(max(zlo, 0), g.nz);
    while (lo > 0 && ((lo - 1 + 0.5) * rz - cz) * lr >= mnx) --lo;
    while (lo < g.nz && !(((lo + 0.5) * rz - cz) * lr >= mnx)) ++lo;
    int hi = min(max(zhi, -1), g.nz - 1);
    while (hi + 1 < g.nz && ((hi + 1 + 0.5) * rz - cz) * lr < mxx) ++hi;
    while (hi >= 0 && !(((hi + 0.5) * rz - cz) * lr < mxx)) --hi;
    zlo = lo;
    zhi = hi;
}

// The reference's chord construction for one voxel-view in FP64
// (Backprojection3D.cu:243-281): false when no low face of the voxel holds the
// entry point of the source->centre line, in which case the reference returns
// and the rest of the column gets nothing from this view.  Each operation is
// rounded separately (no FMA contraction), as the host build of that code is.
__device__ __noinline__ bool chord_entry_found(const ConeGeom &g, int ti, int si, int zi, double sb, double cb) {
    const double EPS = 1e-15;
    const double ct = g.size[0] / 2, cs = g.size[1] / 2, cz = g.size[2] / 2;
    const double rt = g.res[0], rs = g.res[1], rz = g.res[2];
    const double it = __dsub_rn(__dmul_rn(ti + 0.5, rt), ct);
    const double is = __dsub_rn(__dmul_rn(si + 0.5, rs), cs);
    const double iz = __dsub_rn(__dmul_rn(zi + 0.5, rz), cz);
    const double st = __dsub_rn(ct, __dmul_rn(g.D, sb)), ss = __dadd_rn(cs, __dmul_rn(g.D, cb)), sz = cz;
    const double et = __dadd_rn(it, ct), es = __dadd_rn(is, cs), ez = __dadd_rn(iz, cz);
    const double tlo = __dmul_rn((double)ti, rt), thi = __dmul_rn((double)(ti + 1), rt);
    const double slo = __dmul_rn((double)si, rs), shi = __dmul_rn((double)(si + 1), rs);
    const double zlo = __dmul_rn((double)zi, rz), zhi = __dmul_rn((double)(zi + 1), rz);
    const double dt = __dsub_rn(et, st), ds = __dsub_rn(es, ss), dz = __dsub_rn(ez, sz);
    const double dte = __dadd_rn(dt, EPS), dse = __dadd_rn(ds, EPS), dze = __dadd_rn(dz, EPS);
    auto hit = [](double a0, double off, double d1, double de) {   // a0 + off * d1 / de
        return __dadd_rn(a0, __ddiv_rn(__dmul_rn(off, d1), de));
    };
    const double tlo_s = hit(ss, __dsub_rn(tlo, st), ds, dte), tlo_z = hit(sz, __dsub_rn(tlo, st), dz, dte);
    if (tlo_s >= slo && tlo_s <= shi && tlo_z >= zlo && tlo_z <= zhi) return true;
    const double slo_t = hit(st, __dsub_rn(slo, ss), dt, dse), slo_z = hit(sz, __dsub_rn(slo, ss), dz, dse);
    if (slo_t >= tlo && slo_t <= thi && slo_z >= zlo && slo_z <= zhi) return true;
    const double zlo_t = hit(st, __dsub_rn(zlo, sz), dt, dze), zlo_s = hit(ss, __dsub_rn(zlo, sz), ds, dze);
    return zlo_t >= tlo && zlo_t <= thi && zlo_s >= slo && zlo_s <= shi;
}

// The in-plane parts of the reference's first two face tests, which do not
// depend on z (Backprojection3D.cu:262-270): the line from the source to the
// voxel centre crosses the low t face within the voxel's s bounds, or the low
// s face within its t bounds.  Same operations as chord_entry_found.
__device__ __noinline__ bool chord_side_found(const ConeGeom &g, int ti, int si, double sb, double cb) {
    const double EPS = 1e-15;
    const double ct = g.size[0] / 2, cs = g.size[1] / 2;
    const double rt = g.res[0], rs = g.res[1];
    const double it = __dsub_rn(__dmul_rn(ti + 0.5, rt), ct);
    const double is = __dsub_rn(__dmul_rn(si + 0.5, rs), cs);
    const double st = __dsub_rn(ct, __dmul_rn(g.D, sb)), ss = __dadd_rn(cs, __dmul_rn(g.D, cb));
    const double et = __dadd_rn(it, ct), es = __dadd_rn(is, cs);
    const double tlo = __dmul_rn((double)ti, rt), thi = __dmul_rn((double)(ti + 1), rt);
    const double slo = __dmul_rn((double)si, rs), shi = __dmul_rn((double)(si + 1), rs);
    const double dt = __dsub_rn(et, st), ds = __dsub_rn(es, ss);
    const double dte = __dadd_rn(dt, EPS), dse = __dadd_rn(ds, EPS);
    const double tlo_s = __dadd_rn(ss, __ddiv_rn(__dmul_rn(__dsub_rn(tlo, st), ds), dte));
    if (tlo_s >= slo && tlo_s <= shi) return true;
    const double slo_t = __dadd_rn(st, __ddiv_rn(__dmul_rn(__dsub_rn(slo, ss), dt), dse));
    return slo_t >= tlo && slo_t <= thi;
}

// Last z of a column that a view reaches when the source->centre line passes
// near a voxel edge (two faces' chord parameters tie within FP32 margins): the
// reference's FP64 face tests may then all fail at some z, and it returns,
// dropping that z and all above it for this view.  Called rarely (symmetric
// geometries); kept out of line so the hot loop keeps its registers.
__device__ __noinline__ int chord_end_z(const ConeGeom &g, int ti, int si, double sb, double cb, int zlo, int zhi,
                                        bool tie_ts, float ztie, float mmax, bool tz1, float zc1, bool tz2, float zc2) {
    const float rz = (float)g.res[2];
    const float hz = 0.5f * rz;
    const float x_base = (float)(0.5 * g.res[2] - 0.5 * g.size[2]);
    int zab = 0x7fffffff;
    // A face crossing lies |iz| * h_a / |d_a| off the voxel centre in z.  Where
    // that stays below hz (10% margin) at every z of the column, the z parts of
    // the t and s face tests pass everywhere and their z-independent in-plane
    // parts decide every z at once; near the diagonal views this replaces a
    // per-z FP64 replay of the whole column.
    const float izc = fmaxf(fabsf(fmaf((float)max(zlo, 0), rz, x_base)), fabsf(fmaf((float)min(zhi, g.nz - 1), rz, x_base)));
    if (tie_ts && izc * mmax < 0.9f * hz && chord_side_found(g, ti, si, sb, cb)) tie_ts = false;
    if (tie_ts) {
        // t/s faces limit the chord where |iz| <= ztie: check those z in order
        for (int z = max(zlo, 0); z <= min(zhi, g.nz - 1); ++z) {
            const float iz = fmaf((float)z, rz, x_base);
            if (fabsf(iz) > ztie * (1.0f + 1e-5f)) continue;
            if (!chord_entry_found(g, ti, si, z, sb, cb)) { zab = z; break; }
        }
    }
    const int r1 = (int)rintf(zc1), r2 = (int)rintf(zc2);
    if (tz1 && r1 >= zlo && r1 <= zhi && r1 < zab && !chord_entry_found(g, ti, si, r1, sb, cb)) zab = r1;
    if (tz2 && r2 >= zlo && r2 <= zhi && r2 < zab && !chord_entry_found(g, ti, si, r2, sb, cb)) zab = r2;
    return min(zhi, zab - 1);
}

// The record of a column-view, in two arrays [view][s][t]:
//  a = (wa, wb, p1, zr): the weights of detector columns p1 and p1 + 1 times the
//    chord factor 2 mts or the FDK weight; p1 < 0: nothing from this view; zr =
//    zlo | (zend + 1) << 16, the z that take the view relative to the set-up's
//    first slice, clamped to [0, 65535] (FDK sticky: zend the last z on the
//    detector, whose row all z above keep);
//  b = (r, dq): the row quotient at the set-up's first slice and its step per z,
//    fixed point with kRowFrac fraction bits: the step's rounding times the slices of a
//    set-up stays below 2^-25 rows (with 36 bits a column of 60000 slices was 3e-7 off
//    the reference, 1.2e-7 with these).  r has half of a unit of the loop's 32 fraction
//    bits added.
constexpr int kRowFrac = 40;
constexpr long long kRowHalf = 1LL << (kRowFrac - 33);
constexpr int kZSlab = 65504;      // slices a set-up covers (a multiple of the z tiles)
struct __align__(16) ColView {
    float wa, wb;
    int p1;
    unsigned zr;
};

__device__ __forceinline__ long long ff_fixed(ff a) {
    constexpr float one = (float)(1LL << kRowFrac);
    return __float2ll_rn(__fmul_rn(a.hi, one)) + __float2ll_rn(__fmul_rn(a.lo, one));
}

// Chord face parameters of a column-view, h / |d| along t and s: approximate
// reciprocals (a few ulp); the chord factor needs ~1e-7, and the tie tests have
// margins of 1e-5.
__device__ __forceinline__ void chord_faces(const ConeGeom &g, float it, float is, float sb, float cb, float &dt,
                                            float &ds, float &mt, float &ms) {
    dt = it + g.bp_Df * sb;
    ds = is - g.bp_Df * cb;
    mt = __fdividef(g.bp_ht, fabsf(dt));
    ms = __fdividef(g.bp_hs, fabsf(ds));
}

// Records of views [v0, v0 + nv) for slices zbase .. zbase + kZSlab - 1.  A thread
// takes one column and `per` views.
template <int WMODE>
__global__ void __launch_bounds__(128)
cone_bp_setup_kernel(const ConeGeom g, ColView *__restrict__ ta, longlong2 *__restrict__ tb, int v0, int nv, int per,
                     int zbase) {
    const int ti = blockIdx.x * 32 + threadIdx.x;
    const int si = blockIdx.y * 4 + threadIdx.y;
    if (ti >= g.nt || si >= g.ns) return;
    // voxel-centre coordinates relative to the rotation centre, exact to ~2^-48
    const ff it2 = ff_from((ti + 0.5) * g.res[0] - 0.5 * g.size[0]);
    const ff is2 = ff_from((si + 0.5) * g.res[1] - 0.5 * g.size[1]);
    const ff izb2 = ff_from((zbase + 0.5) * g.res[2] - 0.5 * g.size[2]);
    const ff D2 = {g.bp_D.x, g.bp_D.y};
    const ff ipint2 = {g.bp_ipint.x, g.bp_ipint.y};
    const ff xq2 = {g.bp_xq.x, g.bp_xq.y};   // row quotient per mm of xi
    const ff p02 = {g.p0, 0.0f};
    // the view-independent factors of the row quotient: (iz lr - xi0) xq = lr (iz xq) - xi0 xq
    const ff rzxq2 = {g.bp_rzxq.x, g.bp_rzxq.y}, izbxq2 = ff_mul(izb2, xq2), x0xq2 = {g.bp_x0xq.x, g.bp_x0xq.y};
    const float it = it2.hi, is = is2.hi;
    const float D = g.bp_Df;
    const float ipint = g.bp_ipintf;
    const float hz = g.bp_hz;
    const float czf = g.bp_czf;
    const float x_base = g.bp_xbase;      // iz at z = 0
    const float iz_vol = fabsf(x_base);   // largest |iz| of the volume
    const float irz = g.bp_irz, iD = g.bp_iD;
    const long long ncol = (long long)g.nt * g.ns;
    const int k0 = blockIdx.z * per, k1 = min(k0 + per, nv);
    long long o = k0 * ncol + (long long)si * g.nt + ti;
    for (int k = k0; k < k1; ++k, o += ncol) {
        const int v = v0 + k;
        const float2 tr = g.trigf[v];   // float (sin, cos): no FP64 conversion in the loop
        const float sb = tr.x, cb = tr.y;
        // detector coordinates of the column in float-float: the reference's
        // FP64 dect_t, dect_s, LengthRatio = D / (D - dect_s) and P = dect_t * LR
        // (Backprojection3D.cu:28-37)
        const ff dt2 = ff_add(ff_mul_f(it2, cb), ff_mul_f(is2, sb));
        const ff ds2 = ff_sub(ff_mul_f(is2, cb), ff_mul_f(it2, sb));
        const ff den2 = ff_sub(D2, ds2);
        const ff lr2 = ff_div_r(D2, den2, __fdividef(1.0f, den2.hi));
        const ff P2 = ff_mul(dt2, lr2);
        const float dect_s = ds2.hi, lr = lr2.hi, P = P2.hi;
        bool pin = P >= g.minp && P < g.maxp;
        // xi(z) = iz(z) * lr; detector rows in range for z in [zlo, zhi]
        // xi(z) >= minx  <=>  z >= (minx / lr - x_base) / rz, with 1/lr = (D - dect_s) / D
        const float ilr = (D - dect_s) * iD;
        const float zlo_f = fmaf(g.minx, ilr, -x_base) * irz, zhi_f = fmaf(g.maxx, ilr, -x_base) * irz;
        int zlo = (int)ceilf(zlo_f);             // first z with xi >= minx
        int zhi = (int)ceilf(zhi_f) - 1;         // last z with xi < maxx
        // FP32 rounding is ~3e-5 in z units: re-decide in FP64 near an edge
        const bool near_edge = fabsf(zlo_f - rintf(zlo_f)) < 2.5e-4f || fabsf(zhi_f - rintf(zhi_f)) < 2.5e-4f ||
                               fabsf(P - g.minp) < 2e-4f || fabsf(P - g.maxp) < 2e-4f;
        if (near_edge) range_fp64(g, ti, si, g.trig[v].x, g.trig[v].y, pin, zlo, zhi);
        ColView c{0.0f, 0.0f, -1, 0u};
        if (!pin || (WMODE == W_FDK_STICKY && zhi < zlo)) {   // off the detector for this view
            ta[o] = c;
            tb[o] = make_longlong2(0, 0);
            continue;
        }
        // detector column floor(|P - P0| / PInt) and weights |P - P[p1]| / PInt,
        // |P[p1+1] - P| / PInt from the domain values (Backprojection3D.cu:73-83)
        const int p1 = min(max(ff_floor(ff_mul(ff_abs(ff_sub(P2, p02)), ipint2)), 0), g.np - 2);
        const float pa = __ldg(g.P + p1), pb = __ldg(g.P + p1 + 1);
        const float wq1 = fabsf(__fadd_rn(__fsub_rn(P2.hi, pa), P2.lo)) * ipint;   // weight of column p1+1
        const float wq0 = fabsf(__fsub_rn(__fsub_rn(pb, P2.hi), P2.lo)) * ipint;   // weight of column p1
        // row quotient q(z) = |xi(z) - xi[0]| / XigamaInt, affine in z: floor and weights
        // follow the reference's FP64 values except within ~1e-8 of a row boundary
        long long dq = ff_fixed(ff_mul(rzxq2, lr2));
        long long r = ff_fixed(ff_sub(ff_mul(izbxq2, lr2), x0xq2)) + kRowHalf;

        int zend = zhi;           // last z that receives this view's value
        float c0 = lr * lr * g.bint;
        if (WMODE == W_CHORD) {
            float dt, ds, mt, ms;
            chord_faces(g, it, is, sb, cb, dt, ds, mt, ms);
            const float mts = fminf(mt, ms);
            // The source->centre line passes near a voxel edge when two faces'
            // parameters tie; only then can the reference's FP64 face tests all
            // fail and end the column.  Ties are found in FP32 with a wide margin
            // and decided in FP64 (chord_end_z).  A z face can tie only where
            // |iz| reaches hz / mts, i.e. when the volume is tall enough.
            const bool tie_ts = fabsf(mt - ms) <= 1e-5f * mts;
            bool tz1 = false, tz2 = false;
            float zc1 = 0.0f, zc2 = 0.0f;
            if (iz_vol * mts > 0.999f * hz) {
                const float ztie = __fdividef(hz, mts);   // |iz| where the z faces tie with mts
                zc1 = (czf + ztie) * irz - 0.5f;
                zc2 = (czf - ztie) * irz - 0.5f;
                tz1 = fabsf(zc1 - rintf(zc1)) < 1e-3f;
                tz2 = fabsf(zc2 - rintf(zc2)) < 1e-3f;
            }
            if (tie_ts || tz1 || tz2)
                zend = chord_end_z(g, ti, si, g.trig[v].x, g.trig[v].y, zlo, zhi, tie_ts, hz / mts, fmaxf(mt, ms), tz1, zc1, tz2,
                                   zc2);
            c0 = 2.0f * mts;
        }
        c.wa = wq0 * c0;
        c.wb = wq1 * c0;
        c.p1 = p1;
        if (WMODE == W_FDK_STICKY && zhi < zbase) {   // the whole slab keeps the row of zhi
            r += (long long)(zhi - zbase) * dq;
            dq = 0;
            zend = 0x7ffffff0;
        }
        const int a = min(max(zlo - zbase, 0), 65535), e = min(max(zend - zbase + 1, 0), 65535);
        c.zr = (unsigned)a | ((unsigned)e << 16);
        ta[o] = c;
        tb[o] = make_longlong2(r, dq);
    }
}

// Views [v0, v0 + nv) of the scan, whose pairs Q and records (ta, tb) hold
// (index 0 = view v0).  Each voxel's sum b = (sum over these views) + prev
// (when prev is given) is written to out, or with UPDATE folded into out = vol
// as clamp(vol + lambda * b / (colsum + eps), lo, hi).
//
// Per voxel-view of the fast path: the fixed-point step, one row-table load, one
// pair load (two where z advances a row or more), the row sum, the blend, the
// chord polynomial and the sum.
template <int WMODE, bool UPDATE, int BP_ZC>
__global__ void __launch_bounds__(BP_BX * BP_BY, bp_min_blocks(BP_ZC))
cone_bp_kernel(const ConeGeom g, const float2 *__restrict__ Q, const ColView *__restrict__ ta,
               const longlong2 *__restrict__ tb, int v0, int nv, const float *prev, float *out,
               const float *__restrict__ colsum, float eps, float lambda, float lo, float hi, int zt0, int zbase) {
    // the row table (x - q(xi[x]), q(xi[x+1]) - x) of ConeGeom::xtab
    extern __shared__ float2 xtab[];
    const int tid = threadIdx.x + BP_BX * threadIdx.y;
    for (int x = tid; x < g.nx - 1; x += BP_BX * BP_BY) xtab[x] = g.xtab[x];
    __syncthreads();

    const int ti = blockIdx.x * BP_BX + threadIdx.x;
    const int si = blockIdx.y * BP_BY + threadIdx.y;
    const int z0 = (zt0 + (int)blockIdx.z) * BP_ZC;
    if (ti >= g.nt || si >= g.ns) return;
    const int zr0 = z0 - zbase;        // relative to the set-up

    const float it = ff_from((ti + 0.5) * g.res[0] - 0.5 * g.size[0]).hi;
    const float is = ff_from((si + 0.5) * g.res[1] - 0.5 * g.size[1]).hi;
    const float rz = g.bp_rz, hz = g.bp_hz;
    const float iz0 = ff_from((z0 + 0.5) * g.res[2] - 0.5 * g.size[2]).hi;   // iz of this thread's first z
    // largest |iz| of the thread's z range: decides whether z faces can limit the chord
    const float izmax = fmaxf(fabsf(iz0), fabsf(fmaf((float)(BP_ZC - 1), rz, iz0)));
    const float izw = izmax / g.wmin;  // a column's weights sum to at least 2 mts wmin
    const long long vstride = (long long)g.nx * g.np;
    const long long ncol = (long long)g.nt * g.ns;
    const unsigned last = (unsigned)(g.nx - 2);
    constexpr unsigned all = 0xffffffffu >> (32 - BP_ZC);
    const float kc = 0.5f * (BP_ZC - 1);
    const float izc = fmaf(kc, rz, iz0);
    const float hspan = kc * rz, izq = fabsf(izc) + 0.25f * hspan;

    float acc[BP_ZC];
#pragma unroll
    for (int k = 0; k < BP_ZC; ++k) acc[k] = 0.0f;

    ta += (long long)si * g.nt + ti;
    tb += (long long)si * g.nt + ti;
    const float2 *Qview = Q;
    const unsigned row_bytes = 8u * (unsigned)g.np;
    // the records stream from DRAM once per z tile: the next view's are fetched
    // before this one's work
    float4 cn = __ldcs(reinterpret_cast<const float4 *>(ta));
    longlong2 rn = __ldcs(tb);
    for (int v = 0; v < nv; ++v, Qview += vstride) {
        const float4 c = cn;
        const longlong2 rb = rn;
        if (v + 1 < nv) {
            ta += ncol;
            tb += ncol;
            cn = __ldcs(reinterpret_cast<const float4 *>(ta));
            rn = __ldcs(tb);
        }
        const int p1 = __float_as_int(c.z);
        if (p1 < 0) continue;   // whole column off the detector for this view
        const float wa = c.x, wb = c.y;
        const unsigned zr = __float_as_uint(c.w);
        const int zlo = (int)(zr & 0xffffu), zend = (int)(zr >> 16) - 1;
        // 32 fraction bits from here, rounded (rb.x has the half): a quotient that is whole stays whole
        const long long dqf = (rb.y + kRowHalf) >> (kRowFrac - 32);
        long long r = (rb.x + zr0 * rb.y) >> (kRowFrac - 32);
        const float2 *Qv = Qview + p1, *Qn = Qv + g.np;     // rows x and x + 1
        // sticky FDK: z above zhi re-add the value at zhi (the row quotient stops there)
        const int kz = zend - zr0;
        if (WMODE == W_FDK_STICKY && kz < 0) r += (long long)kz * dqf;
        // z of this thread that take this view, as a bit mask over k
        const int klo = max(zlo - zr0, 0), khi = min(((WMODE == W_FDK_STICKY) ? 0x7fff : kz), BP_ZC - 1);
        const unsigned inmask = (klo > khi) ? 0u
                               : ((khi >= BP_ZC - 1 ? all : ((2u << khi) - 1)) & ~((1u << klo) - 1));
        // Fast path: every z of the thread takes the view from rows [0, nx - 2] (the ends of
        // the affine quotient decide), no z face limits the chord, and the chord length
        // |d| = sqrt(qq + iz^2) is the quadratic in k about the thread's middle z
        // (relative error below 1e-7, bounded by the third-order term
        // |iz| h^3 / (2 |d|^4) and the fourth, h^4 / (8 |d|^4), which alone is left in the
        // mid-plane; h the half span of the z).
        bool fast = inmask == all && (unsigned)(int)(r >> 32) <= last &&
                    (unsigned)(int)((r + (BP_ZC - 1) * dqf) >> 32) <= last &&
                    !(WMODE == W_FDK_STICKY && kz < BP_ZC - 1);
        float dt = 0.0f, ds = 0.0f, qq = 0.0f, lc = 0.0f, l1 = 0.0f, l2 = 0.0f;
        if (WMODE == W_CHORD) {
            const float2 tr = g.trigf[v0 + v];
            dt = it + g.bp_Df * tr.x;
            ds = is - g.bp_Df * tr.y;
            qq = fmaf(dt, dt, ds * ds);
            const float lc2 = fmaf(izc, izc, qq);
            const float ilc = rsqrtf(lc2);
            lc = lc2 * ilc;
            l1 = izc * rz * ilc;
            l2 = 0.5f * qq * rz * rz * ilc * ilc * ilc;
            const float hl = hspan * ilc;
            // |iz| mts < hz for every z, to 10% of margin
            fast = fast && 0.55f * izw * (wa + wb) < hz && izq * ilc * hl * hl * hl < 2e-7f;
        }
        if (fast) {
            auto add = [&](int k, unsigned x, unsigned f, float top, float bot) {
                const float fr = __uint2float_rn(f);                          // fraction * 2^32
                const float2 xt = xtab[x];
                const float w1 = fmaf(fr, 2.3283064365386963e-10f, xt.x);    // |w1|: weight of row x+1
                const float w0 = fmaf(fr, -2.3283064365386963e-10f, xt.y);   // |w0|: weight of row x
                const float val = fmaf(fabsf(w0), top, fabsf(w1) * bot);
                if (WMODE == W_CHORD) {
                    // chord 2 * min(h_a / |d_a|) * |d|, d = (dt, ds, iz)
                    const float dk = (float)k - kc;
                    acc[k] = fmaf(val, fmaf(dk, fmaf(dk, l2, l1), lc), acc[k]);
                } else {
                    acc[k] += val;
                }
            };
            unsigned x = (unsigned)(r >> 32), f = (unsigned)r;
            if ((dqf >> 32) == 0) {
                // less than a row per z: the upper row is the upper or the lower row of the z before
                const unsigned df = (unsigned)dqf;
                float top = row_sum(Qv, x, row_bytes, wa, wb), bot = row_sum(Qn, x, row_bytes, wa, wb);
#pragma unroll
                for (int k = 0; k < BP_ZC; ++k) {
                    if (k > 0) {
                        const unsigned xo = x;
                        asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, 0;" : "+r"(f), "+r"(x) : "r"(df));
                        top = x != xo ? bot : top;
                        bot = row_sum(Qn, x, row_bytes, wa, wb);
                    }
                    add(k, x, f, top, bot);
                }
            } else {
                long long rk = r;
#pragma unroll
                for (int k = 0; k < BP_ZC; ++k) {
                    if (k > 0) rk += dqf;
                    const unsigned xk = (unsigned)(rk >> 32);
                    add(k, xk, (unsigned)rk, row_sum(Qv, xk, row_bytes, wa, wb), row_sum(Qn, xk, row_bytes, wa, wb));
                }
            }
        } else {
            float mts = 0.0f;
            if (WMODE == W_CHORD) mts = fminf(__fdividef(g.bp_ht, fabsf(dt)), __fdividef(g.bp_hs, fabsf(ds)));
            long long rk = r;
#pragma unroll
            for (int k = 0; k < BP_ZC; ++k) {
                if (k > 0) rk += (WMODE == W_FDK_STICKY && k > kz) ? 0LL : dqf;
                // an index outside [0, nx-2] (z off the detector, or a negative
                // quotient wrapped by the unsigned compare) is clamped for the read only
                const int x1 = (int)min((unsigned)(int)(rk >> 32), last);
                const float fr = __uint2float_rn((unsigned)rk);
                const float2 xt = xtab[x1];
                const float w1 = fmaf(fr, 2.3283064365386963e-10f, xt.x);
                const float w0 = fmaf(fr, -2.3283064365386963e-10f, xt.y);
                const float val = fmaf(fabsf(w0), row_sum(Qv, x1, row_bytes, wa, wb),
                                       fabsf(w1) * row_sum(Qn, x1, row_bytes, wa, wb));
                float w = 1.0f;
                if (WMODE == W_CHORD) {
                    // a z face limits the chord by min(1, hz / (|iz| mts))
                    const float iz = fmaf((float)k, rz, iz0);
                    const float d2 = fmaf(iz, iz, qq);
                    w = fminf(1.0f, hz / (fabsf(iz) * mts)) * (d2 * rsqrtf(d2));
                }
                const bool in = (inmask >> k) & 1;
                acc[k] = in ? fmaf(val, w, acc[k]) : acc[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < BP_ZC; ++k) {
        const int z = z0 + k;
        if (z < g.nz) {
            const long long o = ((long long)z * g.ns + si) * g.nt + ti;
            const float b = prev ? acc[k] + prev[o] : acc[k];
            if (UPDATE) {
                const float x = out[o] + lambda * b / (colsum[o] + eps);
                out[o] = fminf(fmaxf(x, lo), hi);
            } else {
                out[o] = b;
            }
        }
    }
}

}  // namespace

size_t cone_bp_pairs_bytes(const ConeGeom &g, int nviews) { return sizeof(float2) * (size_t)nviews * g.nx * g.np; }

size_t cone_bp_table_bytes(const ConeGeom &g, int nviews) {
    return (sizeof(ColView) + sizeof(longlong2)) * (size_t)nviews * g.nt * g.ns;
}

int cone_bp_pack(const ConeGeom &g, const float *R, float2 *Q, int v0, int nv, cudaStream_t st) {
    const long long n = (long long)nv * g.nx * g.np;
    int blocks = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 16);
    pack_pairs_kernel<<<blocks, 256, 0, st>>>(R + (long long)v0 * g.nx * g.np, Q, n, g.np);
    CT_LAUNCH_CHECK("pack_pairs_kernel");
    return CT_OK;
}

int cone_bp_ztile(const ConeGeom &g) { return bp_zc(g); }

namespace {

// The records of views [v0, v0 + nv) from slice zbase into tab.
int setup_launch(const ConeGeom &gk, void *tab, int v0, int nv, int weighting, int zbase, cudaStream_t st) {
    const long long ncol = (long long)gk.nt * gk.ns;
    ColView *ta = static_cast<ColView *>(tab);
    longlong2 *tb = reinterpret_cast<longlong2 *>(ta + nv * ncol);
    // 8 views per thread, fewer where the columns alone leave the GPU idle
    int per = 8;
    while (per > 1 && ncol * ((nv + per - 1) / per) < 1024LL * sm_count()) per /= 2;
    const int nz = (nv + per - 1) / per;
    CT_REQUIRE(nz <= 65535, "cone_bp: too many views per chunk");
    const dim3 grid((gk.nt + 31) / 32, (gk.ns + 3) / 4, nz), block(32, 4);
    if (weighting == W_CHORD) cone_bp_setup_kernel<W_CHORD><<<grid, block, 0, st>>>(gk, ta, tb, v0, nv, per, zbase);
    else if (weighting == W_FDK_ZERO)
        cone_bp_setup_kernel<W_FDK_ZERO><<<grid, block, 0, st>>>(gk, ta, tb, v0, nv, per, zbase);
    else cone_bp_setup_kernel<W_FDK_STICKY><<<grid, block, 0, st>>>(gk, ta, tb, v0, nv, per, zbase);
    CT_LAUNCH_CHECK("cone_bp_setup_kernel");
    return CT_OK;
}

}  // namespace

// weighting: 0 chord, 1 FDK (off-detector adds 0), 2 FDK sticky
int cone_bp_launch(const ConeGeom &g, const float2 *Q, void *tab, bool tab_ready, int v0, int nv, const float *prev,
                   float *out, int weighting, const float *colsum, float eps, float lambda, float lo, float hi,
                   bool update, cudaStream_t st, int zt0, int nzt) {
    CT_REQUIRE(g.np >= 2 && g.nx >= 2, "cone_bp: detector needs at least 2x2 samples");
    CT_REQUIRE(v0 >= 0 && nv > 0 && v0 + nv <= g.nb, "cone_bp: view range out of bounds");
    const int zc = bp_zc(g);
    const int ntiles = (g.nz + zc - 1) / zc;
    if (nzt <= 0) nzt = ntiles - zt0;
    CT_REQUIRE(zt0 >= 0 && nzt > 0 && zt0 + nzt <= ntiles, "cone_bp: z tile range out of bounds");
    ConeGeom gk = g;   // with the set-up's constants
    cone_bp_consts(gk);
    dim3 block(BP_BX, BP_BY);
    const size_t smem = sizeof(float2) * (size_t)g.nx;
    CT_REQUIRE(smem <= 48 * 1024, "cone_bp: at most 6144 detector rows");
    const ColView *ta = static_cast<const ColView *>(tab);
    const longlong2 *tb = reinterpret_cast<const longlong2 *>(ta + nv * (long long)g.nt * g.ns);
    // slabs of at most kZSlab slices, each with its own records (one slab below 65505 slices)
    const int slab = kZSlab / zc;
    for (int t = zt0; t < zt0 + nzt;) {
        const int zb = t / slab * slab, n = std::min(zt0 + nzt, zb + slab) - t, zbase = zb * zc;
        if (!tab_ready || ntiles > slab)
            if (int s = setup_launch(gk, tab, v0, nv, weighting, zbase, st)) return s;
        const dim3 grid((g.nt + BP_BX - 1) / BP_BX, (g.ns + BP_BY - 1) / BP_BY, n);
#define CT_BP_RUN(W, U, Z)                                                                                        \
    cone_bp_kernel<W, U, Z><<<grid, block, smem, st>>>(gk, Q, ta, tb, v0, nv, prev, out, colsum, eps, lambda, lo, \
                                                       hi, t, zbase)
#define CT_BP_CASE(W, U)                            \
    if (zc == kZLong) CT_BP_RUN(W, U, kZLong); \
    else if (zc == kZShort) CT_BP_RUN(W, U, kZShort); \
    else if (zc == kZTiny) CT_BP_RUN(W, U, kZTiny); \
    else CT_BP_RUN(W, U, kZLeast)
        if (update) {
            if (weighting == W_CHORD) { CT_BP_CASE(W_CHORD, true); }
            else if (weighting == W_FDK_ZERO) { CT_BP_CASE(W_FDK_ZERO, true); }
            else { CT_BP_CASE(W_FDK_STICKY, true); }
        } else {
            if (weighting == W_CHORD) { CT_BP_CASE(W_CHORD, false); }
            else if (weighting == W_FDK_ZERO) { CT_BP_CASE(W_FDK_ZERO, false); }
            else { CT_BP_CASE(W_FDK_STICKY, false); }
        }
#undef CT_BP_RUN
#undef CT_BP_CASE
        CT_LAUNCH_CHECK("cone_bp_kernel");
        t += n;
    }
    return CT_OK;
}

}  // namespace ct

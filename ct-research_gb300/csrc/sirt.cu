// sirt.cu -- regulariser and reduction kernels of the SIRT(-TV) loops.
//
// TV step.  The reference has no SIRT+TV driver; its TV building block is
// the TV-flow update of tv.m (Exterior_toolbox/Code_ProLu_OptDenoise/tv.m:
// 30-44: I <- I + dt * curvature, epsilon-regularised gradient).  This file
// runs the same flow in 3D with forward differences and Neumann boundaries:
//   TV_eps(x) = sum_v sqrt(|D+ x|_v^2 + eps^2),  g = dTV_eps/dx,
//   g_v = -(dx_v + dy_v + dz_v)/n_v + dx_{v-ex}/n_{v-ex} + dy_{v-ey}/n_{v-ey} + dz_{v-ez}/n_{v-ez},
// and each sub-iteration moves x <- max(x - step * g / rms(g), lo), i.e. a
// normalised gradient step whose RMS size is `step` (ASD-POCS style).
// Two passes per sub-iteration: gradient + sum(g^2) (block reduction, one
// double atomic per block), then the update.
#include <type_traits>

#include "kernels.cuh"

namespace ct {

namespace {

// Gradient: a warp owns 30 columns in x (lanes 1 .. 30; lanes 0 and 31 carry the
// neighbours) times TV_RY rows in y and a run of planes.
constexpr int TV_WX = 30, TV_RY = 4, TV_WARPS = 4;

// 1 / sqrt(v); FTZ where v cannot be subnormal (the same result there).
template <bool FTZ>
__device__ __forceinline__ float tv_rsqrt(float v) {
    float r;
    if (FTZ) asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    else r = rsqrtf(v);
    return r;
}

// The gradient of one sub-step.  Every lane keeps its column's TV_RY rows and one
// on either side of three planes in registers (the plane after next is in
// flight), evaluates each voxel's forward differences and norm once, and takes
// the (i-1) terms from the lane before it by a shuffle, the (j-1) terms from the
// row before, the (k-1) terms from the plane before; only the row below the tile
// and the plane below the run are evaluated twice.  Tiles and planes clear of the
// volume's faces skip their tests.  Every rounding is written out (TV flows amplify
// a last bit).  No shared memory and no barrier: 52
// instructions per voxel against 146 of the form this replaced (a 32 x 8 tile of
// columns that met in shared memory, two barriers per plane); 256^3: 63 -> 38 us.
// One double atomic per block.
template <bool FTZ>
__global__ void __launch_bounds__(32 * TV_WARPS, 8)
tv_grad_kernel(const float *__restrict__ x, float *__restrict__ g, int nx, int ny, int nz, int kc, float eps2,
               double *__restrict__ sumsq) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = blockIdx.x * TV_WX - 1 + lane;
    const int j0 = (blockIdx.y * TV_WARPS + wid) * TV_RY;
    const int k0 = blockIdx.z * kc, k1 = min(k0 + kc, nz);
    const int plane = nx * ny;
    const bool out = lane >= 1 && lane <= TV_WX && i < nx;
    const bool xf = i + 1 < nx, xb = i > 0;
    const bool clear = blockIdx.x > 0 && (int)(blockIdx.x + 1) * TV_WX < nx && j0 > 0 && j0 + TV_RY < ny;
    float s[TV_RY];
#pragma unroll
    for (int r = 0; r < TV_RY; ++r) s[r] = 0.0f;
    if (j0 < ny) {
        // offsets of rows j0 - 1 .. j0 + TV_RY in a plane (clamped: what lies outside is never used)
        int o[TV_RY + 2];
        const int ic = min(max(i, 0), nx - 1);
#pragma unroll
        for (int r = 0; r < TV_RY + 2; ++r) o[r] = min(max(j0 - 1 + r, 0), ny - 1) * nx + ic;
        const int ks = max(k0 - 1, 0);           // the plane before the run, for its (k-1) terms
        float pa[TV_RY + 2], pb[TV_RY + 2], pc[TV_RY + 2], pz[TV_RY];
#pragma unroll
        for (int r = 0; r < TV_RY + 2; ++r) {
            pa[r] = __ldg(x + (ks * plane + o[r]));
            pb[r] = __ldg(x + (min(ks + 1, nz - 1) * plane + o[r]));
        }
#pragma unroll
        for (int r = 0; r < TV_RY; ++r) pz[r] = 0.0f;
        // plane k with its own values c and the next plane's n
        auto plane_terms = [&](auto inner, int k, const float (&c)[TV_RY + 2], const float (&n)[TV_RY + 2]) {
            constexpr bool IN = decltype(inner)::value;
            const bool zf = IN || k + 1 < nz, store = out && k >= k0;
            const int og = k * plane + j0 * nx + i;
            float pyb = 0.0f;
#pragma unroll
            for (int r = 0; r <= TV_RY; ++r) {   // row j0 - 1 + r
                const int j = j0 - 1 + r;
                const float v = c[r];
                const float vx = __shfl_down_sync(0xffffffffu, v, 1);
                const float dx = (IN || xf) ? vx - v : 0.0f;
                const float dy = (IN || j + 1 < ny) ? c[r + 1] - v : 0.0f;
                const float dz = zf ? n[r] - v : 0.0f;
                const float inv_n = tv_rsqrt<FTZ>(__fadd_rn(__fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy))), eps2));
                if (r > 0) {
                    const float pxb = __shfl_up_sync(0xffffffffu, __fmul_rn(dx, inv_n), 1);
                    const float S = -(dx + dy + dz);
                    float gv = __fmul_rn(S, inv_n);
                    if (IN || xb) gv = __fadd_rn(gv, pxb);
                    if (IN || j > 0) gv = __fadd_rn(gv, pyb);
                    if (IN || k > 0) gv = __fadd_rn(gv, pz[r - 1]);
                    pz[r - 1] = __fmul_rn(dz, inv_n);
                    if (store && (IN || j < ny)) {
                        g[og + (r - 1) * nx] = gv;
                        s[r - 1] = fmaf(gv, gv, s[r - 1]);
                    }
                }
                pyb = __fmul_rn(dy, inv_n);
            }
        };
        auto step = [&](int k, const float (&c)[TV_RY + 2], const float (&n)[TV_RY + 2], float (&p)[TV_RY + 2]) {
            const int kp = min(k + 2, nz - 1) * plane;
#pragma unroll
            for (int r = 0; r < TV_RY + 2; ++r) p[r] = __ldg(x + (kp + o[r]));
            if (clear && k > 0 && k + 1 < nz) plane_terms(std::true_type{}, k, c, n);
            else plane_terms(std::false_type{}, k, c, n);
        };
        for (int k = ks;;) {
            step(k, pa, pb, pc);
            if (++k >= k1) break;
            step(k, pb, pc, pa);
            if (++k >= k1) break;
            step(k, pc, pa, pb);
            if (++k >= k1) break;
        }
    }
    // FP32 sums of at most 32 planes per row, of the rows and of the warp, then FP64
#pragma unroll
    for (int r = 1; r < TV_RY; ++r) s[0] += s[r];
    block_sum_atomic_f<TV_WARPS>(s[0], sumsq);
}

void tv_grad_launch(dim3 grid, cudaStream_t st, float eps2, const float *x, float *g, int nx, int ny, int nz, int kc,
                    double *sumsq) {
    // the argument of the root is at least eps2: normal unless that is not
    if (eps2 >= 1.17549435e-38f) tv_grad_kernel<true><<<grid, 32 * TV_WARPS, 0, st>>>(x, g, nx, ny, nz, kc, eps2, sumsq);
    else tv_grad_kernel<false><<<grid, 32 * TV_WARPS, 0, st>>>(x, g, nx, ny, nz, kc, eps2, sumsq);
}

// x <- max(x - scale g, lo): 16 bytes per load where both pointers allow it.
__device__ __forceinline__ void tv_move(float *__restrict__ x, const float *__restrict__ g, long long n, float scale,
                                        float lo) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    const bool wide = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(g)) & 15) == 0;
    const long long n4 = wide ? n >> 2 : 0;
    float4 *x4 = reinterpret_cast<float4 *>(x);
    const float4 *g4 = reinterpret_cast<const float4 *>(g);
#pragma unroll 2
    for (long long i = t; i < n4; i += stride) {
        const float4 d = __ldg(g4 + i);
        float4 v = x4[i];
        v.x = fmaxf(fmaf(-scale, d.x, v.x), lo);
        v.y = fmaxf(fmaf(-scale, d.y, v.y), lo);
        v.z = fmaxf(fmaf(-scale, d.z, v.z), lo);
        v.w = fmaxf(fmaf(-scale, d.w, v.w), lo);
        x4[i] = v;
    }
    for (long long i = 4 * n4 + t; i < n; i += stride) x[i] = fmaxf(fmaf(-scale, g[i], x[i]), lo);
}

__global__ void __launch_bounds__(256)
tv_apply_kernel(float *__restrict__ x, const float *__restrict__ g, long long n, float step, float lo,
                const double *__restrict__ sumsq) {
    // one warp's FP64 root and division per block (in every warp they kept the FP64 pipe busy for half of the pass)
    __shared__ float scale;
    __shared__ bool moves;
    if (threadIdx.x < 32) {
        const double ss = *sumsq;
        moves = ss > 0.0;
        scale = (float)(step * sqrt((double)n / ss));
    }
    __syncthreads();
    if (moves) tv_move(x, g, n, scale, lo);
}

// tv_apply_kernel with the ASD-POCS step on the device: state = (alpha, dp2, dg2)
// with dp2 the squared size of the data step, so the RMS move of the sub-step
// is alpha * sqrt(dp2 / n), i.e. scale = alpha * sqrt(dp2 / sum g^2).
__global__ void __launch_bounds__(256)
tv_apply_asd_kernel(float *__restrict__ x, const float *__restrict__ g, long long n, float lo,
                    const double *__restrict__ sumsq, const double *__restrict__ state) {
    __shared__ float scale;
    __shared__ bool moves;
    if (threadIdx.x < 32) {
        const double ss = *sumsq, dp2 = state[1];
        moves = ss > 0.0 && dp2 > 0.0;
        scale = (float)(state[0] * sqrt(dp2 / ss));
    }
    __syncthreads();
    if (moves) tv_move(x, g, n, scale, lo);
}

// alpha <- alpha * alpha_red when the TV phase moved x more than r_max times the data step
__global__ void asd_alpha_kernel(double *state, float alpha_red, float r_max) {
    if (sqrt(state[2]) > (double)r_max * sqrt(state[1])) state[0] *= (double)alpha_red;
}

__global__ void __launch_bounds__(256)
sq_diff_kernel(const float *__restrict__ a, const float *__restrict__ b, long long n, double *__restrict__ out) {
    // FP32 partial sums of 16 terms, flushed into an FP64 sum (FP64 per
    // element would bound this kernel on GB300)
    double s = 0.0;
    float f = 0.0f;
    int c = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float d = a[i] - b[i];
        f = fmaf(d, d, f);
        if (++c == 16) {
            s += (double)f;
            f = 0.0f;
            c = 0;
        }
    }
    s += (double)f;
    block_sum_atomic<8>(s, out);
}

// Warps of 30 x TV_RY columns, and runs of kc planes: up to 32, fewer when that
// leaves under ~16 warps per scheduler
dim3 tv_grid(int nx, int ny, int nz, int &kc) {
    const long long gx = (nx + TV_WX - 1) / TV_WX, gy = (ny + TV_WARPS * TV_RY - 1) / (TV_WARPS * TV_RY);
    const long long fill = gx * gy * nz / (16LL * sm_count());
    kc = (int)std::min<long long>(nz, std::max<long long>(4, std::min<long long>(32, fill)));
    while ((nz + kc - 1) / kc > 65535) kc *= 2;
    return dim3((unsigned)gx, (unsigned)gy, (unsigned)((nz + kc - 1) / kc));
}

}  // namespace

int tv_flow_launch(float *x, float *work, double *scratch, int nx, int ny, int nz, int iters, float step, float eps,
                   float lo, cudaStream_t st) {
    CT_REQUIRE(nx > 0 && ny > 0 && nz > 0, "tv: sizes must be positive");
    CT_REQUIRE((long long)nx * ny * nz < (1LL << 31), "tv: volume too large");
    const long long n = (long long)nx * ny * nz;
    int kc = 1;
    const dim3 grid = tv_grid(nx, ny, nz, kc);
    const int ablocks = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 8);
    for (int it = 0; it < iters; ++it) {
        CT_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double), st), "tv memset");
        tv_grad_launch(grid, st, eps * eps, x, work, nx, ny, nz, kc, scratch);
        CT_LAUNCH_CHECK("tv_grad_kernel");
        tv_apply_kernel<<<ablocks, 256, 0, st>>>(x, work, n, step, lo, scratch);
        CT_LAUNCH_CHECK("tv_apply_kernel");
    }
    return CT_OK;
}

int tv_flow_asd_launch(float *x, float *prev, float *work, double *scratch, double *state, int nx, int ny, int nz,
                       int iters, float eps, float lo, float alpha_red, float r_max, cudaStream_t st) {
    CT_REQUIRE(nx > 0 && ny > 0 && nz > 0, "tv: sizes must be positive");
    CT_REQUIRE((long long)nx * ny * nz < (1LL << 31), "tv: volume too large");
    const long long n = (long long)nx * ny * nz;
    int kc = 1;
    const dim3 grid = tv_grid(nx, ny, nz, kc);
    const int ablocks = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 8);
    CT_CUDA(cudaMemsetAsync(state + 1, 0, 2 * sizeof(double), st), "asd memset");
    if (int s = sq_diff_sum_launch(x, prev, n, state + 1, st)) return s;        // dp2
    CT_CUDA(cudaMemcpyAsync(prev, x, n * sizeof(float), cudaMemcpyDeviceToDevice, st), "asd copy");
    for (int it = 0; it < iters; ++it) {
        CT_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double), st), "tv memset");
        tv_grad_launch(grid, st, eps * eps, x, work, nx, ny, nz, kc, scratch);
        CT_LAUNCH_CHECK("tv_grad_kernel");
        tv_apply_asd_kernel<<<ablocks, 256, 0, st>>>(x, work, n, lo, scratch, state);
        CT_LAUNCH_CHECK("tv_apply_asd_kernel");
    }
    if (int s = sq_diff_sum_launch(x, prev, n, state + 2, st)) return s;        // dg2
    asd_alpha_kernel<<<1, 1, 0, st>>>(state, alpha_red, r_max);
    CT_LAUNCH_CHECK("asd_alpha_kernel");
    return CT_OK;
}

int sq_diff_sum_launch(const float *a, const float *b, long long n, double *out, cudaStream_t st) {
    const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 8);
    if (blocks <= 0) return CT_OK;
    sq_diff_kernel<<<blocks, 256, 0, st>>>(a, b, n, out);
    CT_LAUNCH_CHECK("sq_diff_kernel");
    return CT_OK;
}

}  // namespace ct

extern "C" {

int ct_tv_flow(float *d_x, float *d_work, double *d_scratch, int nx, int ny, int nz, int iters, float step, float eps,
               float lo, void *stream) {
    CT_REQUIRE(d_x && d_work && d_scratch, "ct_tv_flow: null argument");
    CT_REQUIRE(iters >= 0, "ct_tv_flow: negative iteration count");
    return ct::tv_flow_launch(d_x, d_work, d_scratch, nx, ny, nz, iters, step, eps, lo, ct::as_stream(stream));
}

int ct_tv_flow_asd(float *d_x, float *d_prev, float *d_work, double *d_scratch, double *d_state, int nx, int ny,
                   int nz, int iters, float eps, float lo, float alpha_red, float r_max, void *stream) {
    CT_REQUIRE(d_x && d_prev && d_work && d_scratch && d_state, "ct_tv_flow_asd: null argument");
    CT_REQUIRE(iters >= 0, "ct_tv_flow_asd: negative iteration count");
    return ct::tv_flow_asd_launch(d_x, d_prev, d_work, d_scratch, d_state, nx, ny, nz, iters, eps, lo, alpha_red, r_max,
                                  ct::as_stream(stream));
}

int ct_sq_diff_sum(const float *d_a, const float *d_b, long long n, double *d_norm, void *stream) {
    CT_REQUIRE(d_a && d_b && d_norm && n >= 0, "ct_sq_diff_sum: bad argument");
    return ct::sq_diff_sum_launch(d_a, d_b, n, d_norm, ct::as_stream(stream));
}

}  // extern "C"

// filter.cu -- pre-weight + Shepp-Logan-form ramp filtering of detector rows.
//
// out[p] = dP * sum_q in'[q] * G[(np-1) + p - q], G the taps of GFunction
// (FDK.cu:6-19): G[np-1] = 1/(pi dP)^2, G[np-1 +- n] = -1/(pi dP)^2/(4n^2-1).
// in' is the row after the cosine pre-weight w (FDK: D/sqrt(D^2+P^2+xi^2),
// FDK.cu:34; FBPfan: R/sqrt(R^2+P^2), FBPfan.cu:32; FBPparallel: none).
//
// The reference applies w in place inside the same kernel that convolves the
// row, one P-tile (256 samples for FDK, 128 for FBPfan) per launch and
// `limit` taps per launch chunk (FDK.cu:333-477).  LAUNCH_ORDER mode models
// what that produces on a GPU: the outputs of a P-tile see the tiles launched
// before it fully weighted, their own tile weighted once per chunk processed
// so far, and later tiles unweighted; rows of the residual row tile launch
// the residual P-tile first.  CLEAN mode weights the whole row once.
//
// Options beyond the reference's GPU path: other ramp taps (Ram-Lak) only
// change G; short-scan (Parker) weights multiply the raw row as it is loaded,
// as a caller weighting the sinogram before the call would; a Hamming
// smoothing window runs over each finished filtered row.
//
// row_filter_kernel: the row, its weighted copy and the taps live in shared
// memory; a thread computes 4 consecutive outputs, whose taps at 4 consecutive
// samples are 7 consecutive ones, read as one 16-byte load per 4 samples.
// row_filter_repeat_kernel: launch order on rows longer than `limit`, where the
// weight is applied several times.
#include "kernels.cuh"

namespace ct {


namespace {

constexpr int FT = 256;
constexpr int FJ = 4;        // consecutive outputs per thread
constexpr int kFlush = 256;  // samples between flushes of the float pair into a double

// Position in the launch sequence of P-tile k for a row: rows of the residual
// row tile launch the residual P-tile first.
__device__ __forceinline__ int tile_pos(int k, int nfull, bool resid_first) {
    return resid_first ? (k == nfull ? 0 : k + 1) : k;
}

// Exact sums in FP32.  The row is scaled by a power of two to |m| < 1 and the
// taps to G[np-1] in [1/4, 1/2), so that (both kinds of taps sum to at most twice
// their centre) every partial sum of the products is within 1 of 0.  Started at
// 6, the running sum s stays within [4, 8), where it is a multiple of 2^-21 larger
// than any product: t = s + m w rounded, then t - s is exact and one more FMA
// gives the error of t, m w - (t - s), to 2^-47.  The errors are summed in a
// second float, and both go into a double every 256 samples: to ~2^-39 of the
// largest product per flush (the reference rounds each product to a float,
// 2^-25, before its double sum).  4 operations per tap instead of the 8 of a
// rounded product and TwoSum.
//
// FP32-bound: 16 operations per sample of a thread against 0.5 shared loads.
// 360 x 384 rows of 512 (FDK of 256^3) 8.9 -> 5.1 ms, 720 rows of 1024 (FBP) 0.31 -> 0.134 ms.
//
// grid: rows x split, each block a run of the row's outputs (split > 1 where the
// rows alone would leave the GPU idle).  A row filtered in place takes one block, which
// has read the whole row before it writes.
__global__ void __launch_bounds__(FT)
row_filter_kernel(const RowFilter f, const float *__restrict__ R, float *__restrict__ out, int split) {
    extern __shared__ float4 sm4[];
    __shared__ float part_max[FT / 32];
    const int np = f.np, np4 = (np + 3) & ~3;
    const int pad = 4 + ((4 - ((np + 3) & 3)) & 3);        // taps start at `pad`: np - 1 + pad is a multiple of 4
    float *raw = reinterpret_cast<float *>(sm4);
    float *wgt = raw + np4;
    float *G = wgt + np4;
    const int row = blockIdx.x / split, part = blockIdx.x % split;
    const float *in = R + (long long)row * np;
    float *o = out + (long long)row * np;
    const double *w = f.w ? f.w + (long long)(row % f.wrows) * np : nullptr;
    const float *pw = f.pw ? f.pw + (long long)(row / f.pw_div) * np : nullptr;
    float amax = 0.0f;
    for (int q = threadIdx.x; q < np4; q += blockDim.x) {
        const float v = q < np ? (pw ? __fmul_rn(in[q], pw[q]) : in[q]) : 0.0f;
        raw[q] = v;
        wgt[q] = (w && q < np) ? (float)((double)v * w[q]) : v;
        amax = fmaxf(amax, fabsf(v));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    if ((threadIdx.x & 31) == 0) part_max[threadIdx.x >> 5] = amax;
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) amax = fmaxf(amax, part_max[i]);
    // powers of two: the row's, clamped to normal floats, and the taps'; 1 for a row of
    // zeros or with infinities
    const int em = (amax > 0.0f && amax < __int_as_float(0x7f800000)) ? max(min(ilogbf(amax) + 1, 126), -125) : 0;
    const float g0 = fabsf(f.G[np - 1]);
    const int eg = (g0 > 0.0f && g0 < __int_as_float(0x7f800000)) ? max(min(ilogbf(g0) + 2, 126), -125) : 0;
    const float ms = ldexpf(1.0f, -em), gs = ldexpf(1.0f, -eg);
    for (int q = threadIdx.x; q < np4; q += blockDim.x) {
        raw[q] *= ms;
        wgt[q] *= ms;
    }
    for (int i = threadIdx.x; i < 2 * np - 1 + pad + 8; i += blockDim.x)
        G[i] = (i >= pad && i < 2 * np - 1 + pad) ? f.G[i - pad] * gs : 0.0f;
    __syncthreads();

    const bool order = f.launch_order && w;
    const int tile = order ? f.tile : np4;
    const int nfull = np / f.tile, resid = np % f.tile;
    const int ridx = row % f.rowmod;
    const bool resid_first = resid && (f.rowmod % f.row_block) != 0 && ridx >= (f.rowmod / f.row_block) * f.row_block;
    const double unscale = (double)f.pint * ldexp(1.0, em + eg);
    const int groups = (np + FJ - 1) / FJ, per = (groups + split - 1) / split;
    const int gend = min(groups, (part + 1) * per);
    for (int gi = part * per + threadIdx.x; gi < gend; gi += blockDim.x) {
        const int pb = FJ * gi;
        const int kpos = order ? tile_pos(pb / tile, nfull, resid_first) : 0;
        const float *gp = G + pad + (np - 1) + pb;          // tap of output pb + j at sample q: gp[j - q]
        double dacc[FJ] = {0.0, 0.0, 0.0, 0.0};
        for (int t0 = 0, j = 0; t0 < np4; t0 += tile, ++j) {
            // the samples of this tile as the output's launch reads them
            const float *mix = (!order || tile_pos(j, nfull, resid_first) <= kpos) ? wgt : raw;
            const int t1 = min(t0 + tile, np4);
            for (int q0 = t0; q0 < t1; q0 += kFlush) {
                const int q1 = min(q0 + kFlush, t1);
                float s[FJ], l[FJ];
#pragma unroll
                for (int i = 0; i < FJ; ++i) {
                    s[i] = 6.0f;
                    l[i] = 0.0f;
                }
                float4 hi = *reinterpret_cast<const float4 *>(gp - q0);
#pragma unroll 2
                for (int q = q0; q < q1; q += 4) {
                    const float4 lo = *reinterpret_cast<const float4 *>(gp - q - 4);
                    const float4 m4 = *reinterpret_cast<const float4 *>(mix + q);
                    const float tap[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    const float m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
                    for (int d = 0; d < 4; ++d)
#pragma unroll
                        for (int i = 0; i < FJ; ++i) {
                            const float g = tap[4 + i - d];
                            const float t = __fmaf_rn(m[d], g, s[i]);
                            l[i] = __fadd_rn(l[i], __fmaf_rn(m[d], g, __fsub_rn(s[i], t)));
                            s[i] = t;
                        }
                    hi = lo;
                }
#pragma unroll
                for (int i = 0; i < FJ; ++i) dacc[i] += ((double)s[i] - 6.0) + (double)l[i];
            }
        }
#pragma unroll
        for (int i = 0; i < FJ; ++i)
            if (pb + i < np) o[pb + i] = (float)(unscale * dacc[i]);
    }
    if (f.win) {
        // smoothing of the filtered row (split = 1): o[p] = sum_i win[i] x[p + i - wlen/2] / wsum,
        // x zero outside the row; sequential double sum without contraction
        __syncthreads();
        for (int q = threadIdx.x; q < np; q += blockDim.x) raw[q] = o[q];
        __syncthreads();
        const int c = f.wlen / 2;
        for (int p = threadIdx.x; p < np; p += blockDim.x) {
            double acc = 0.0;
            for (int i = 0; i < f.wlen; ++i) {
                const int k = p + i - c;
                if (k >= 0 && k < np) acc = __dadd_rn(acc, __dmul_rn((double)raw[k], f.win[i]));
            }
            o[p] = (float)__ddiv_rn(acc, f.wsum);
        }
    }
}

// Launch order on rows of more than `limit` samples: the weight is applied once
// more per chunk of `limit` samples, so the row is mixed anew for every P-tile
// and chunk, and each chunk's sum is added into the float output.  One block
// per row, one output per thread.
__global__ void __launch_bounds__(FT)
row_filter_repeat_kernel(const RowFilter f, const float *__restrict__ R, float *__restrict__ out) {
    extern __shared__ float sm[];
    const int np = f.np;
    float *raw = sm;
    float *mix = sm + np;
    float *G = sm + 2 * np;
    const int row = blockIdx.x;
    const float *in = R + (long long)row * np;
    float *o = out + (long long)row * np;
    const double *w = f.w + (long long)(row % f.wrows) * np;
    const float *pw = f.pw ? f.pw + (long long)(row / f.pw_div) * np : nullptr;
    for (int q = threadIdx.x; q < np; q += blockDim.x) {
        raw[q] = pw ? __fmul_rn(in[q], pw[q]) : in[q];
        o[q] = 0.0f;
    }
    for (int q = threadIdx.x; q < 2 * np - 1; q += blockDim.x) G[q] = f.G[q];
    __syncthreads();

    const int gtime = (np + f.limit - 1) / f.limit;
    const int nfull = np / f.tile, resid = np % f.tile;
    const int ntiles = nfull + (resid ? 1 : 0);
    const int ridx = row % f.rowmod;
    const bool resid_first = resid && (f.rowmod % f.row_block) != 0 && ridx >= (f.rowmod / f.row_block) * f.row_block;
    for (int step = 0; step < ntiles; ++step) {
        int k = 0;
        for (int j = 0; j < ntiles; ++j)
            if (tile_pos(j, nfull, resid_first) == step) k = j;
        const int p0 = k * f.tile, p1 = (k == nfull) ? np : p0 + f.tile;
        for (int c = 0; c < gtime; ++c) {
            const int g0 = c * f.limit, g1 = (c == gtime - 1) ? np : (c + 1) * f.limit;
            // the row as this chunk's launch reads it
            for (int q = g0 + threadIdx.x; q < g1; q += blockDim.x) {
                const int j = q / f.tile;
                const int e = (tile_pos(j, nfull, resid_first) < step) ? gtime : (j == k ? c + 1 : 0);
                float v = raw[q];
                for (int i = 0; i < e; ++i) v = (float)((double)v * w[q]);
                mix[q] = v;
            }
            __syncthreads();
            for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
                // rounded products, summed as an unevaluated pair (s + l) with the TwoSum
                // error-free transformation (Knuth), flushed into a double
                double dacc = 0.0;
                const float *gp = G + (np - 1) + p;
                for (int q0 = g0; q0 < g1; q0 += kFlush) {
                    const int q1 = min(q0 + kFlush, g1);
                    float s = 0.0f, l = 0.0f;
#pragma unroll 4
                    for (int q = q0; q < q1; ++q) {
                        const float prod = __fmul_rn(mix[q], gp[-q]);
                        const float t = __fadd_rn(s, prod);
                        const float bp = __fsub_rn(t, s);
                        l = __fadd_rn(l, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(prod, bp)));
                        s = t;
                    }
                    dacc += (double)s + (double)l;
                }
                o[p] = (float)((double)o[p] + (double)f.pint * dacc);
            }
            __syncthreads();
        }
    }
    if (f.win) {
        for (int q = threadIdx.x; q < np; q += blockDim.x) raw[q] = o[q];
        __syncthreads();
        const int c = f.wlen / 2;
        for (int p = threadIdx.x; p < np; p += blockDim.x) {
            double acc = 0.0;
            for (int i = 0; i < f.wlen; ++i) {
                const int k = p + i - c;
                if (k >= 0 && k < np) acc = __dadd_rn(acc, __dmul_rn((double)raw[k], f.win[i]));
            }
            o[p] = (float)__ddiv_rn(acc, f.wsum);
        }
    }
}

}  // namespace

int row_filter_launch(const RowFilter &f, const float *R, float *out, cudaStream_t st) {
    CT_REQUIRE(f.np >= 2, "row filter: at least 2 detector samples");
    CT_REQUIRE(f.np <= 12800, "row filter: detector row too long for shared memory");
    const bool repeat = f.launch_order && f.w && f.np > f.limit;
    const size_t smem = sizeof(float) * (size_t)(repeat ? 4 * f.np : 2 * ((f.np + 3) & ~3) + 2 * f.np + 16);
    if (smem > 48 * 1024)
        CT_CUDA(cudaFuncSetAttribute(repeat ? (const void *)row_filter_repeat_kernel : (const void *)row_filter_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                "row_filter smem attribute");
    if (repeat) {
        const int block = std::min(FT, std::max(32, (f.tile + 31) / 32 * 32));
        row_filter_repeat_kernel<<<f.nrow, block, smem, st>>>(f, R, out);
        CT_LAUNCH_CHECK("row_filter_repeat_kernel");
        return CT_OK;
    }
    // threads for the row's groups of outputs, in blocks of 32 to 128 (a warp's 128
    // outputs then lie in one P-tile); where the rows give fewer than 8 warps per
    // scheduler, a block per warp
    const int warps = ((f.np + FJ - 1) / FJ + 31) / 32;
    const size_t n = (size_t)f.nrow * f.np;
    const bool in_place = R < out + n && out < R + n;      // the input's rows overlap the output's
    int per_block = std::min(warps, 4);
    if (!f.win && !in_place && (long long)f.nrow * warps < 32LL * sm_count()) per_block = 1;
    const int split = f.win || in_place ? 1 : (warps + per_block - 1) / per_block;
    CT_REQUIRE((long long)f.nrow * split < (1LL << 31), "row filter: too many rows");
    row_filter_kernel<<<(unsigned)((long long)f.nrow * split), 32 * per_block, smem, st>>>(f, R, out, split);
    CT_LAUNCH_CHECK("row_filter_kernel");
    return CT_OK;
}

}  // namespace ct

// unet_conv.cu -- BF16 3x3x3 / 1x1x1 convolutions of the warm-start U-Net on
// the sm_103a tensor cores (tcgen05), with FP32 accumulation in tensor memory.
//
// Both kernels are one GEMM D[128 x N] = sum_k A[128 x 32k] B[N x 32k]^T whose
// 32-wide K slices are fetched by TMA into shared memory (64-byte rows,
// 64-byte swizzle), multiplied by tcgen05.mma (M = 128, K = 16 per
// instruction) issued by one thread, and accumulated in TMEM:
//
// * conv_fwd_kernel (forward, and data gradient with the flipped weights):
//   rows = 128 output voxels (a bx x by x bz block), columns = the
//   output channels, K = taps x input channels.  Activations are channels-last
//   bf16 [n][z][y][x][c]; the tap offset moves the TMA box, whose zero fill
//   outside the volume is the convolution's zero padding.  Two inputs are
//   concatenated along K (the skip connection) without a copy.  The epilogue
//   adds the bias, applies ReLU or the ReLU-derivative mask of a saved
//   activation, rounds to bf16 and splits the channels over one or two outputs.
//   conv_march_kernel is the same convolution for few channels: it keeps the
//   filters in shared memory and reads each input slice once.
// * conv_first_kernel: the one-channel input's 27 taps built in shared memory.
// * conv_wgrad_cl_kernel (weight gradient): the channels-last tensors as they
//   are, see below.  conv_wgrad_kernel, for volumes that its segments do not fit
//   and for 128 x 128 channels and more:
//   rows = (tap, input channel), columns = output channels, K = voxels in
//   64-voxel slices (128-byte rows, 128-byte swizzle).  Activations and output
//   gradients are read channel-major [n][c][z][y*x]; x offsets come from three
//   x-shifted copies (so the innermost TMA coordinate stays on the 16-byte
//   grid), y and z offsets move the box.  Split-K over voxel ranges; partial
//   sums are added to an FP32 gradient with atomics.
//
// A warp-specialised pipeline per CTA: warp 0 issues TMA loads into a 3- or
// 4-stage ring, warp 1 the MMAs (one elected lane of a converged warp each), and
// after the last MMA all four warps read the accumulator from TMEM (tcgen05.ld)
// for the epilogue.  Every mbarrier wait is bounded by a 2 s timer; a timeout
// sets a device error flag (read by ct_unet_status), the loads in flight are
// waited for and TMEM is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "ct_common.cuh"

namespace ct {

namespace {

__device__ int g_unet_err;

constexpr int kStages = 4;
constexpr int kRowBytes = 64;                 // one K slice: 32 bf16
constexpr int kTileM = 128;
constexpr uint32_t kABytes = kTileM * kRowBytes;
constexpr unsigned long long kWaitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase of the given parity; false after limit_ns (kWaitNs).
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, unsigned long long limit_ns = kWaitNs) {
    if (mbar_try(b, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 256; ++i)
            if (mbar_try(b, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// Flag bit of a bounded wait that gave up in wait_selftest_kernel.
constexpr int kErrSelftest = 8;

// One thread waits, through the convolutions' own bounded wait, on an
// mbarrier that nothing arrives on; the wait gives up after limit_ns and sets
// the error flag as a timed-out convolution does.  No copy or tensor-memory
// operation is in flight, so the kernel simply returns.
__global__ void __launch_bounds__(32) wait_selftest_kernel(unsigned long long limit_ns) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        if (!mbar_wait(&bar, 0, limit_ns)) atomicOr(&g_unet_err, kErrSelftest);
    }
}

__device__ __forceinline__ void tma_load5(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2,
                                          int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2,
                                          int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

__device__ __forceinline__ void tma_load3(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// Shared-memory matrix descriptor of a K-major operand in the 64-byte swizzle
// layout: 64-byte rows, 8-row atoms of 512 bytes (stride byte offset), the
// leading byte offset unused, descriptor version 1, layout code 4.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
    uint64_t d = static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(512 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(4) << 61;
    return d;
}

// The same for the 128-byte swizzle layout: 128-byte rows, 8-row atoms of
// 1024 bytes, layout code 2.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// Descriptor of an MN-major operand in the 64-byte swizzle layout: atoms of 32
// MN elements (64 bytes) x 8 k rows; mn_step bytes from one atom to the next
// along MN (leading byte offset), 512 along k (stride byte offset).
__device__ __forceinline__ uint64_t sw64_mn_desc(uint32_t saddr, uint32_t mn_step) {
    uint64_t d = static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(mn_step >> 4) << 16;
    d |= static_cast<uint64_t>(512 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(4) << 61;
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(m >> 4) << 24);
}

// The same with both operands MN-major.
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int m, int n) { return idesc_bf16(m, n) | (1u << 15) | (1u << 16); }

__device__ __forceinline__ void umma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
    return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

// Shared control block after the stage ring.
struct Ctrl {
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t done;
    uint32_t tmem;
};

// A wait gave up: each role then ends on its own waits, all bounded.
__device__ __forceinline__ void flag_error(int code) { atomicOr(&g_unet_err, code); }

__device__ __forceinline__ void tap_offsets(int tap, int ntaps, int &dz, int &dy, int &dx) {
    if (ntaps == 27) {
        dz = tap / 9 - 1;
        dy = (tap / 3) % 3 - 1;
        dx = tap % 3 - 1;
    } else {
        dz = dy = dx = 0;
    }
}

// Wait (bounded) until every load into the S stages has landed: no CTA leaves with one in flight, whichever wait gave up.
template <int S>
__device__ void drain_loads(Ctrl *c, int issued) {
    for (int s = 0; s < S && s < issued; ++s) {
        const int last = (issued - 1 - s) / S;   // use index of the last load into stage s
        mbar_wait(&c->full[s], static_cast<uint32_t>(last & 1));
    }
}

// One lane of a converged warp; the compiler then keeps the operands of the
// instructions in uniform registers instead of selecting them lane by lane.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// The MMA side of one CTA, called by a whole warp, over an S-stage ring of
// (A_BYTES of A, NG * N rows of B) stages with ROWB-byte rows (64: 64-byte
// swizzle, 128: 128-byte swizzle): per K step, NG groups of ROWB / 32
// instructions of 128 x N x 16, group g reading A from byte offset g * A_STEP
// and the g-th B tile.
template <int N, int S, uint32_t A_BYTES, int NG, uint32_t A_STEP, int ROWB = kRowBytes>
__device__ __forceinline__ void mma_loop(Ctrl *c, uint8_t *ring, uint32_t tmem, int ksteps) {
    constexpr uint32_t stage = A_BYTES + NG * N * ROWB;
    constexpr uint32_t idesc = idesc_bf16(kTileM, N);
    constexpr int KK = ROWB / 32;
    const uint32_t ra = smem_u32(ring);
    const uint64_t ad0 = ROWB == 128 ? sw128_desc(ra) : sw64_desc(ra);
    const uint64_t bd0 = ROWB == 128 ? sw128_desc(ra + A_BYTES) : sw64_desc(ra + A_BYTES);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int k = 0; k < ksteps; ++k) {
        ok = __all_sync(0xffffffffu, mbar_wait(&c->full[s], ph));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
            const uint64_t so = static_cast<uint64_t>(s) * (stage / 16);
#pragma unroll
            for (int g = 0; g < NG; ++g)
#pragma unroll
                for (int kk = 0; kk < KK; ++kk)
                    umma_bf16(tmem, ad0 + so + (g * A_STEP + kk * 32) / 16, bd0 + so + (g * N * ROWB + kk * 32) / 16,
                              idesc, k | g | kk);
            umma_commit(&c->empty[s]);
        }
        __syncwarp();
        if (++s == S) {
            s = 0;
            ph ^= 1;
        }
    }
    if (!ok) flag_error(2);
    if (elect_one()) umma_commit(&c->done);
}

// y-halo mode of the forward kernel: 8 x 16 voxel tiles of one slice; one box of
// 8 x 18 voxels per (dz, dx, channel chunk) serves the three dy taps, whose A
// operands start 0, 8 and 16 rows (512-byte swizzle atoms) into it.
constexpr int kYBx = 8, kYBy = 16;
constexpr uint32_t kYABytes = kYBx * (kYBy + 2) * kRowBytes;
constexpr int kYStages = 3;

// weight-gradient ring: K slices of 64 voxels (128-byte rows, 128-byte swizzle)
constexpr int kWK = 64;
constexpr int kWRowBytes = 2 * kWK;
constexpr int kWStages = 3;

struct FwdArgs {
    int c1, c2;              // channels of input 1 and input 2 (0: one input)
    int ntaps;               // 27 (3x3x3) or 1
    int nx, ny, nz;          // volume size, x fastest
    int bx, by, bz;          // voxel block of one tile (bx * by * bz = 128)
    int ksteps;              // ntaps * (c1 + c2) / 32
    const float *bias;       // [N] or null
    int relu;
    __nv_bfloat16 *out1, *out2;
    int co1, co2;            // channels written to out1 / out2 (co1 + co2 = N)
    const __nv_bfloat16 *mask1, *mask2;   // ReLU-derivative masks (same layout as out1 / out2) or null
    const float *head_w, *head_b, *base;  // conv_march_kernel's HEAD mode: 32 weights, bias, added volume or null
    float *head_out;
};

// ReLU-derivative mask values of columns c0 .. c0 + 15 of a voxel.
struct Mask16 {
    uint4 q0, q1;
};

__device__ __forceinline__ Mask16 load_mask(const FwdArgs &a, long long vox, int c0) {
    const bool first = c0 < a.co1;
    const __nv_bfloat16 *m = first ? a.mask1 : a.mask2;
    Mask16 r{};
    if (m) {
        const uint4 *mp = reinterpret_cast<const uint4 *>(m + vox * (first ? a.co1 : a.co2) + (first ? c0 : c0 - a.co1));
        r.q0 = __ldg(mp);
        r.q1 = __ldg(mp + 1);
    }
    return r;
}

// Bias, ReLU, mask, rounding and the store of columns c0 .. c0 + 15 of a voxel.
__device__ __forceinline__ void store16(const FwdArgs &a, long long vox, int c0, float (&v)[16], const Mask16 &mask) {
    const bool first = c0 < a.co1;
    __nv_bfloat16 *o = first ? a.out1 : a.out2;
    const int cc = first ? c0 : c0 - a.co1, stride = first ? a.co1 : a.co2;
    if (a.bias) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __ldg(a.bias + c0 + j);
    }
    if (a.relu) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f);
    }
    if (first ? a.mask1 : a.mask2) {
        const __nv_bfloat16 *mb0 = reinterpret_cast<const __nv_bfloat16 *>(&mask.q0);
        const __nv_bfloat16 *mb1 = reinterpret_cast<const __nv_bfloat16 *>(&mask.q1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (!(__bfloat162float(mb0[j]) > 0.0f)) v[j] = 0.0f;
            if (!(__bfloat162float(mb1[j]) > 0.0f)) v[8 + j] = 0.0f;
        }
    }
    uint4 w0, w1;
    uint32_t *p0 = reinterpret_cast<uint32_t *>(&w0), *p1 = reinterpret_cast<uint32_t *>(&w1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        const __nv_bfloat162 h1 = __floats2bfloat162_rn(v[8 + 2 * j], v[8 + 2 * j + 1]);
        p0[j] = *reinterpret_cast<const uint32_t *>(&h0);
        p1[j] = *reinterpret_cast<const uint32_t *>(&h1);
    }
    uint4 *op = reinterpret_cast<uint4 *>(o + vox * stride + cc);
    op[0] = w0;
    op[1] = w1;
}

template <int N, bool YR>
__global__ void __launch_bounds__(128, 1)
conv_fwd_kernel(const __grid_constant__ CUtensorMap mx1, const __grid_constant__ CUtensorMap mx2,
                const __grid_constant__ CUtensorMap mw, const FwdArgs a) {
    constexpr int S = YR ? kYStages : kStages;
    constexpr uint32_t a_bytes = YR ? kYABytes : kABytes;
    constexpr int ng = YR ? 3 : 1;
    constexpr uint32_t stage = a_bytes + ng * N * kRowBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *ring = align1024(smem_raw);
    Ctrl *c = reinterpret_cast<Ctrl *>(ring + S * stage);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    int t = blockIdx.x;
    const int tx = a.nx / a.bx, ty = a.ny / a.by, tz = a.nz / a.bz;
    const int x0 = (t % tx) * a.bx;
    t /= tx;
    const int y0 = (t % ty) * a.by;
    t /= ty;
    const int z0 = (t % tz) * a.bz, n0 = t / tz;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&c->full[s], 1);
            mbar_init(&c->empty[s], 1);
        }
        mbar_init(&c->done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc(&c->tmem, N);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = c->tmem;

    if (warp == 0) {
        // K order: (tap or (dz, dx) group) major, 32-channel chunks inner
        const int cin = a.c1 + a.c2, ngrp = YR ? 9 : a.ntaps;
        int s = 0, issued = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int grp = 0; ok && grp < ngrp; ++grp) {
            int dz, dy, dx;
            if (YR) {
                dz = grp / 3 - 1;
                dx = grp % 3 - 1;
                dy = -1;                          // the box starts one row above the tile
            } else {
                tap_offsets(grp, a.ntaps, dz, dy, dx);
            }
            for (int ch = 0; ch < cin; ch += 32) {
                if (issued >= S) ok = __all_sync(0xffffffffu, mbar_wait(&c->empty[s], ph ^ 1));
                if (!ok) break;
                if (elect_one()) {
                    uint8_t *sa = ring + s * stage;
                    mbar_expect_tx(&c->full[s], stage);
                    if (ch < a.c1)
                        tma_load5(sa, &mx1, &c->full[s], ch, x0 + dx, y0 + dy, z0 + dz, n0);
                    else
                        tma_load5(sa, &mx2, &c->full[s], ch - a.c1, x0 + dx, y0 + dy, z0 + dz, n0);
                    if (YR) {
#pragma unroll
                        for (int g = 0; g < 3; ++g)         // dy = g - 1
                            tma_load3(sa + a_bytes + g * N * kRowBytes, &mw, &c->full[s], ch,
                                      (dz + 1) * 9 + g * 3 + (dx + 1), 0);
                    } else {
                        tma_load3(sa + a_bytes, &mw, &c->full[s], ch, grp, 0);
                    }
                }
                __syncwarp();
                ++issued;
                if (++s == S) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        if (!ok) flag_error(1);
        drain_loads<S>(c, issued);
    } else if (warp == 1) {
        mma_loop<N, S, a_bytes, ng, kYBx * kRowBytes>(c, ring, tmem, a.ksteps);
    }
    __syncwarp();

    // epilogue: thread = tile row = voxel
    const bool ok = mbar_wait(&c->done, 0);
    if (!ok) flag_error(4);
    tc_fence_after();
    const int r = warp * 32 + lane;
    const int rxy = a.bx * a.by;
    const long long vox = ((static_cast<long long>(n0) * a.nz + z0 + r / rxy) * a.ny + (y0 + (r % rxy) / a.bx)) *
                              a.nx +
                          (x0 + r % a.bx);
    const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
#pragma unroll 1
    for (int c0 = 0; c0 < N; c0 += 16) {
        float v[16];
        tmem_ld16(trow + c0, v);
        if (!ok) continue;
        const Mask16 m = load_mask(a, vox, c0);
        store16(a, vox, c0, v, m);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) tmem_dealloc(tmem, N);
}

// ---------------------------------------------------------------------------
// z-marching mode of the 3x3x3 convolution, for filters that fit in shared
// memory (32 outputs from 32 or 64 channels, 64 outputs from 32).
//
// conv_fwd_kernel reads 9 boxes of each 32-channel chunk and all 27 filter
// slices for every 128-voxel tile (138 KB of L2 reads for 32 -> 32 channels:
// the L2's rate sets its time), in 54 instructions of N = 32 that the
// reading of A from shared memory holds to a quarter of the tensor cores' rate.
// Here a CTA keeps all filter slices and walks 8 x 16 voxel columns along z: each
// input slice is fetched once (three boxes, one per dx) and multiplied by the
// filters of the three dz at once, one 128 x 3N x 16 instruction per (dx, dy,
// 16 channels): the accumulators of the outputs z - 1, z, z + 1 are neighbours
// in a ring of tensor-memory columns, and the filter rows are stored in the order
// dz = +1, 0, -1.  An output still sums its taps in conv_fwd_kernel's order
// (dz, dx, chunk, dy), so the results are the same bits.
//
// An instruction takes 56 cycles at 3N = 96 (7 KB of operands from shared memory
// at 128 B/clock; 48 at the tensor cores' rate) and 96 at 3N = 192; issuing, waiting
// and committing cost the issuing thread about as long again per slice, so a
// CTA holds two groups of warps that share the filters, each with its own
// columns, load ring and half of the tensor memory, and one's waits pass under the
// other's instructions.  Per group: four warps store finished slices, one issues
// the loads, one the instructions.  Persistent, one CTA per SM: a group takes
// items = (sample, z chunk, tile) in turn.
//
// GB300, 256^3: 32 -> 32 channels 1542 -> 662 us (1.4 PFLOP/s), 64 -> 32 2518 ->
// 1314; 128^3: 32 -> 64 324 -> 181, 64 -> 64 489 -> 363.  One group per CTA: 1125 us for
// 32 -> 32; with one thread of an undivided warp issuing (operands moved to
// uniform registers for each instruction) 2386 us.
// ---------------------------------------------------------------------------
constexpr int kMGroups = 2;
constexpr int kMBoxes = 6;                    // boxes (8 x 18 voxels, 32 channels) in a group's load ring
constexpr int kMCols = 256;                   // tensor-memory columns of a group's accumulator ring

struct MarchGroup {
    uint64_t full[kMBoxes / 2];
    uint64_t empty[kMBoxes / 2];
    uint64_t accfull[kMCols / 32];
    uint64_t accempty[kMCols / 32];
    uint64_t done;
};

struct MarchCtrl {
    MarchGroup g[kMGroups];
    uint64_t wfull;
    uint32_t tmem;
};

struct MarchArgs {
    FwdArgs f;
    int tx, ty;              // tiles along x and y
    int zc, nzc;             // output slices per item, items along z
    int parts;               // CTAs b, b + parts, ... compute outputs (b % parts) * N .. + N - 1
    long long items;
};

struct MarchItem {
    int x0, y0, z0, z1, n;   // outputs z0 .. z1 - 1 of the tile at (x0, y0)
};

__device__ __forceinline__ MarchItem march_item(const MarchArgs &a, long long i) {
    MarchItem it;
    it.x0 = static_cast<int>(i % a.tx) * kYBx;
    i /= a.tx;
    it.y0 = static_cast<int>(i % a.ty) * kYBy;
    i /= a.ty;
    it.z0 = static_cast<int>(i % a.nzc) * a.zc;
    it.z1 = min(it.z0 + a.zc, a.f.nz);
    it.n = static_cast<int>(i / a.nzc);
    return it;
}

// N outputs, NCH 32-channel chunks of the input.  HEAD (N = 32): instead of the 32
// channels, their 1 x 1 convolution to one, added to `base`: the bf16 values and the
// order of the sum are those of storing them and reading them back, without that
// gigabyte at 256^3: 635 + 194 us as two launches, about 580 as one (a whole forward
// pass 6.60 -> 6.35 ms).
template <int N, int NCH, bool HEAD>
__global__ void __launch_bounds__(192 * kMGroups, 1)
conv_march_kernel(const __grid_constant__ CUtensorMap mx1, const __grid_constant__ CUtensorMap mx2,
                  const __grid_constant__ CUtensorMap mw, const MarchArgs a) {
    constexpr int R = kMCols / N;                          // accumulators in a group's ring
    // a stage: all boxes of a slice (one chunk), or those of one dx (two chunks)
    constexpr int DXS = NCH == 1 ? 3 : 1, S = kMBoxes / (DXS * NCH);
    constexpr uint32_t stage = DXS * NCH * kYABytes;
    constexpr uint32_t wblock = N * kRowBytes;             // filter rows of one tap and chunk
    constexpr uint32_t wbytes = 27 * NCH * wblock;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *wsm = align1024(smem_raw);                    // [dx][chunk][dy][dz = +1, 0, -1][N] filter rows
    uint8_t *rings = wsm + wbytes;
    MarchCtrl *ctrl = reinterpret_cast<MarchCtrl *>(rings + kMGroups * S * stage);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // warps 0 .. 4 G - 1: stores, four per group; then the groups' loading warps, then their multiplying warps
    const int role = warp < 4 * kMGroups ? 0 : (warp < 5 * kMGroups ? 1 : 2);
    const int grp = role == 0 ? warp / 4 : warp % kMGroups;
    MarchGroup *c = ctrl->g + grp;
    uint8_t *ring = rings + grp * S * stage;
    const int n0 = blockIdx.x % a.parts * N;               // first output channel
    const long long item0 = blockIdx.x / a.parts * kMGroups + grp;
    const long long istep = static_cast<long long>(gridDim.x / a.parts) * kMGroups;
    const int nz = a.f.nz;

    if (threadIdx.x < kMGroups) {
        MarchGroup *q = ctrl->g + threadIdx.x;
        for (int s = 0; s < S; ++s) {
            mbar_init(&q->full[s], 1);
            mbar_init(&q->empty[s], 1);
        }
        for (int s = 0; s < R; ++s) {
            mbar_init(&q->accfull[s], 1);
            mbar_init(&q->accempty[s], 4);
        }
        mbar_init(&q->done, 1);
        if (threadIdx.x == 0) mbar_init(&ctrl->wfull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 6 * kMGroups - 1) tmem_alloc(&ctrl->tmem, kMGroups * kMCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctrl->tmem + grp * kMCols;

    if (role == 1) {
        if (grp == 0 && lane == 0) {
            mbar_expect_tx(&ctrl->wfull, wbytes);
            for (int b = 0; b < 27 * NCH; ++b) {           // b = ((dx * NCH + chunk) * 3 + dy) * 3 + j, dz = 1 - j
                const int tap = (2 - b % 3) * 9 + (b / 3 % 3) * 3 + b / (9 * NCH);
                tma_load3(wsm + b * wblock, &mw, &ctrl->wfull, b / 9 % NCH * 32, tap, n0);
            }
        }
        __syncwarp();
        int s = 0, used = 0;                               // stage, stages filled so far (up to S)
        uint32_t ph = 0;
        bool ok = true;
        for (long long i = item0; ok && i < a.items; i += istep) {
            const MarchItem it = march_item(a, i);
            const int ze = min(it.z1, nz - 1);
            for (int z = max(it.z0 - 1, 0); ok && z <= ze; ++z) {
#pragma unroll
                for (int g = 0; g < 3 / DXS; ++g) {
                    if (used == S) ok = __all_sync(0xffffffffu, mbar_wait(&c->empty[s], ph ^ 1));
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_expect_tx(&c->full[s], stage);
#pragma unroll
                        for (int j = 0; j < DXS * NCH; ++j) {
                            const int dx = g * DXS + j / NCH - 1, ch = j % NCH * 32;
                            const bool second = ch >= a.f.c1;
                            tma_load5(ring + s * stage + j * kYABytes, second ? &mx2 : &mx1, &c->full[s],
                                      second ? ch - a.f.c1 : ch, it.x0 + dx, it.y0 - 1, z, it.n);
                        }
                    }
                    __syncwarp();
                    used = min(used + 1, S);
                    if (++s == S) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
        if (!ok && lane == 0) flag_error(1);
        // every load has landed before the CTA may leave: the last use of stage j
        mbar_wait(&ctrl->wfull, 0);
        for (int j = 0; j < used; ++j) mbar_wait(&c->full[j], j < s ? ph : ph ^ 1);
    } else if (role == 2) {
        bool ok = __all_sync(0xffffffffu, mbar_wait(&ctrl->wfull, 0));
        const uint64_t wdesc = sw64_desc(smem_u32(wsm)), adesc = sw64_desc(smem_u32(ring));
        unsigned obase = 0;                                // outputs of earlier items
        int s = 0;
        uint32_t ph = 0;
        for (long long i = item0; ok && i < a.items; i += istep) {
            const MarchItem it = march_item(a, i);
            const int ze = min(it.z1, nz - 1);
            for (int z = max(it.z0 - 1, 0); ok && z <= ze; ++z) {
                const int lo = max(z - 1, it.z0), hi = min(z + 1, it.z1 - 1), cnt = hi - lo + 1;
                const unsigned olo = obase + lo - it.z0, blo = olo % R;
                // this slice is the first input of output z + 1 (and of output 0): it starts in a free accumulator
                for (int zo = max(z ? z + 1 : 0, lo); zo <= hi; ++zo) {
                    const unsigned o = olo + zo - lo;
                    if (o >= R && !mbar_wait(&c->accempty[o % R], (o / R - 1) & 1)) ok = false;
                }
                const bool whole = cnt == 3 && blo + 3 <= R;   // and z > 0: outputs z - 1, z go on, z + 1 starts
                const int la = min(cnt, static_cast<int>(R - blo)), lb = cnt - la;
                const uint64_t b0 = wdesc + static_cast<uint64_t>(lo - z + 1) * (wblock / 16);
                const uint32_t d0 = tmem + blo * N;
#pragma unroll
                for (int g = 0; g < 3 / DXS; ++g) {
                    if (!mbar_wait(&c->full[s], ph)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t a0 = adesc + static_cast<uint64_t>(s) * (stage / 16);
#pragma unroll
                        for (int q = 0; q < DXS * NCH * 6; ++q) {   // q = ((dx * NCH + chunk) * 3 + dy) * 2 + half
                            const uint64_t ad = a0 + (q / 6) * (kYABytes / 16) + (q / 2 % 3) * (kYBx * kRowBytes / 16) +
                                                (q % 2) * 2;
                            const uint64_t bd = b0 + (g * DXS * NCH * 3 + q / 2) * (3 * wblock / 16) + (q % 2) * 2;
                            if (g == 0 && q == 0) {
                                if (whole) {
                                    umma_bf16(d0, ad, bd, idesc_bf16(kTileM, 2 * N), 1);
                                    umma_bf16(d0 + 2 * N, ad, bd + 2 * wblock / 16, idesc_bf16(kTileM, N), 0);
                                } else {
                                    for (int j = 0; j < cnt; ++j)
                                        umma_bf16(tmem + (blo + j) % R * N, ad, bd + j * (wblock / 16),
                                                  idesc_bf16(kTileM, N), z != max(lo + j - 1, 0));
                                }
                            } else if (whole) {
                                umma_bf16(d0, ad, bd, idesc_bf16(kTileM, 3 * N), 1);
                            } else {
                                umma_bf16(d0, ad, bd, idesc_bf16(kTileM, N * la), 1);
                                if (lb)                    // the ring's end lies between the outputs
                                    umma_bf16(tmem, ad, bd + la * (wblock / 16), idesc_bf16(kTileM, N * lb), 1);
                            }
                        }
                        umma_commit(&c->empty[s]);
                        if (g == 3 / DXS - 1) {            // outputs that this slice is the last input of
                            if (lo < z) umma_commit(&c->accfull[blo]);
                            if (z == nz - 1 && hi == z) umma_commit(&c->accfull[(blo + z - lo) % R]);
                        }
                    }
                    __syncwarp();
                    if (++s == S) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            obase += it.z1 - it.z0;
        }
        if (!ok && lane == 0) flag_error(2);
        if (elect_one()) umma_commit(&c->done);
    } else {
        const int r = (warp & 3) * 32 + lane;
        const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        unsigned o = 0;
        bool ok = true;
        float hw[HEAD ? 32 : 1];
        if (HEAD) {
#pragma unroll
            for (int j = 0; j < (HEAD ? 32 : 1); ++j) hw[j] = __ldg(a.f.head_w + j);
        }
        for (long long i = item0; ok && i < a.items; i += istep) {
            const MarchItem it = march_item(a, i);
            long long vox = ((static_cast<long long>(it.n) * nz + it.z0) * a.f.ny + it.y0 + r / kYBx) * a.f.nx + it.x0 +
                            r % kYBx;
            for (int z = it.z0; z < it.z1; ++z, ++o, vox += static_cast<long long>(a.f.ny) * a.f.nx) {
                Mask16 m[N / 16];
                float sum = 0.0f;
                if (HEAD) {
                    sum = __ldg(a.f.head_b) + (a.f.base ? __ldg(a.f.base + vox) : 0.0f);
                } else {
#pragma unroll
                    for (int j = 0; j < N / 16; ++j) m[j] = load_mask(a.f, vox, n0 + 16 * j);
                }
                ok = __all_sync(0xffffffffu, mbar_wait(&c->accfull[o % R], (o / R) & 1));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < N / 16; ++j) {
                    float v[16];
                    tmem_ld16(trow + o % R * N + 16 * j, v);
                    if (j == N / 16 - 1) {                 // the accumulator is in registers: free it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&c->accempty[o % R]))
                                         : "memory");
                    }
                    if (HEAD) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            float x = a.f.bias ? v[e] + __ldg(a.f.bias + 16 * j + e) : v[e];
                            if (a.f.relu) x = fmaxf(x, 0.0f);
                            sum = fmaf(hw[HEAD ? 16 * j + e : 0], __bfloat162float(__float2bfloat16_rn(x)), sum);
                        }
                    } else {
                        store16(a.f, vox, n0 + 16 * j, v, m[j]);
                    }
                }
                if (HEAD) a.f.head_out[vox] = sum;
            }
        }
        if (!ok && lane == 0) flag_error(4);
    }
    __syncwarp();
    if (!mbar_wait(&c->done, 0)) flag_error(4);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 6 * kMGroups - 1) tmem_dealloc(ctrl->tmem, kMGroups * kMCols);
}

// ---------------------------------------------------------------------------
// The first convolution: one FP32 input channel, 32 outputs.  Its 27 taps are a
// K of 32 (5 zeros): what im2col27 gathers into a [v][32] tensor and a 1-tap
// convolution reads back is built here in shared memory, one voxel per
// thread and row, and multiplied by the same two instructions, so the outputs
// are the same bits without the 2 GB the tensor moves at 256^3.  256^3: 455 us
// against 302 + 691; bound by the 27 loads and the packing per voxel (619 us
// with 64-bit index divisions and the bias read per tile).
// ---------------------------------------------------------------------------
// CTAs per SM (48 registers): a 256^3 forward pass takes 6.38 ms at 8, 6.33 at 10 or 12.
constexpr int kFirstCtas = 10;
struct FirstArgs {
    const float *vol;
    const __nv_bfloat16 *w;  // [32][32]
    int nx, ny, nz;
    long long tiles;         // of 128 consecutive voxels
    int small;               // voxels below 2^32
    int relu;
    const float *bias;       // [32] or null
    __nv_bfloat16 *out;      // [v][32]
};

// 16 bytes of row r (64 bytes) at chunk q of a 64-byte swizzled tile.
__device__ __forceinline__ void put_sw64(uint8_t *tile, int r, int q, const uint4 &v) {
    *reinterpret_cast<uint4 *>(tile + r * 64 + ((q ^ ((r >> 1) & 3)) << 4)) = v;
}

__global__ void __launch_bounds__(128, kFirstCtas)
conv_first_kernel(const FirstArgs a) {
    __shared__ __align__(1024) uint8_t atile[128 * 64];
    __shared__ __align__(1024) uint8_t btile[32 * 64];
    __shared__ __align__(16) float bias[32];
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_slot;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), r = threadIdx.x;
    if (r == 0) {
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc(&tmem_slot, 32);
    if (r < 32) bias[r] = a.bias ? a.bias[r] : 0.0f;
    put_sw64(btile, r / 4, r % 4, __ldg(reinterpret_cast<const uint4 *>(a.w) + r));
    uint32_t ph = 0, tmem = 0;
    bool ok = true;
    const long long plane = static_cast<long long>(a.nx) * a.ny;
    for (long long t = blockIdx.x; t < a.tiles; t += gridDim.x) {
        const long long vox = t * 128 + r;
        int x, y, z;
        if (a.small) {                                     // 32-bit divisions
            const unsigned v = static_cast<unsigned>(vox), row = v / a.nx, zy = row / a.ny;
            x = v - row * a.nx;
            y = row - zy * a.ny;
            z = zy % a.nz;
        } else {
            const long long row = vox / a.nx;
            x = static_cast<int>(vox - row * a.nx);
            y = static_cast<int>(row % a.ny);
            z = static_cast<int>(row / a.ny % a.nz);
        }
        const float *c = a.vol + vox;
        float val[32];
        const bool xl = x > 0, xh = x < a.nx - 1;
        const bool inner = y > 0 && y < a.ny - 1 && z > 0 && z < a.nz - 1;   // of most warps, all lanes
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            val[k] = 0.0f;
            if (k < 27) {
                const int dz = k / 9 - 1, dy = k / 3 % 3 - 1, dx = k % 3 - 1;
                const bool in = (dx < 0 ? xl : (dx > 0 ? xh : true)) &&
                                (inner || (static_cast<unsigned>(y + dy) < static_cast<unsigned>(a.ny) &&
                                           static_cast<unsigned>(z + dz) < static_cast<unsigned>(a.nz)));
                if (in) val[k] = __ldg(c + (dz * plane + dy * a.nx) + dx);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 w;
            uint32_t *p = reinterpret_cast<uint32_t *>(&w);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(val[q * 8 + 2 * j], val[q * 8 + 2 * j + 1]);
                p[j] = *reinterpret_cast<const uint32_t *>(&h);
            }
            put_sw64(atile, r, q, w);
        }
        // the tiles as the tensor cores see them; the last tile's accumulator has been read
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tmem = tmem_slot;
        if (warp == 0) {
            if (elect_one()) {
                const uint64_t ad = sw64_desc(smem_u32(atile)), bd = sw64_desc(smem_u32(btile));
                umma_bf16(tmem, ad, bd, idesc_bf16(kTileM, 32), 0);
                umma_bf16(tmem, ad + 2, bd + 2, idesc_bf16(kTileM, 32), 1);
                umma_commit(&done);
            }
            __syncwarp();
        }
        ok = mbar_wait(&done, ph);
        ph ^= 1;
        ok = __syncthreads_and(ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
        uint4 *op = reinterpret_cast<uint4 *>(a.out + vox * 32);
#pragma unroll
        for (int c0 = 0; c0 < 32; c0 += 16) {
            float v[16];
            tmem_ld16(trow + c0, v);
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const float4 b = *reinterpret_cast<const float4 *>(bias + c0 + j);
                v[j] += b.x;
                v[j + 1] += b.y;
                v[j + 2] += b.z;
                v[j + 3] += b.w;
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo = v[8 * q + 2 * j], hi = v[8 * q + 2 * j + 1];
                    if (a.relu) {
                        lo = fmaxf(lo, 0.0f);
                        hi = fmaxf(hi, 0.0f);
                    }
                    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
                    w[j] = *reinterpret_cast<const uint32_t *>(&h);
                }
                op[c0 / 8 + q] = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
    if (!ok && r == 0) flag_error(4);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 2) tmem_dealloc(tmem_slot, 32);
}

struct WgradArgs {
    int cin, ntaps;
    int rows_per_tap, taps_per_tile, cblocks;
    int nxy, nx, nz;         // y*x plane size, x size, slices
    long long kchunks;       // 64-voxel K slices over all samples
    int pchunks;             // 64-voxel slices per y*x plane (the last may run past the plane: zero fill)
    int kper;                // K slices per CTA
    float *dw;               // [N][ntaps][cin], FP32, accumulated
};

template <int N>
__global__ void __launch_bounds__(128, 1)
conv_wgrad_kernel(const __grid_constant__ CUtensorMap mxm, const __grid_constant__ CUtensorMap mx0,
                  const __grid_constant__ CUtensorMap mxp, const __grid_constant__ CUtensorMap mdy,
                  const WgradArgs a) {
    constexpr uint32_t a_bytes = kTileM * kWRowBytes;
    constexpr uint32_t stage = a_bytes + N * kWRowBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *ring = align1024(smem_raw);
    Ctrl *c = reinterpret_cast<Ctrl *>(ring + kWStages * stage);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    const int tgroup = blockIdx.x / a.cblocks, cb = blockIdx.x % a.cblocks;
    const int tap0 = tgroup * a.taps_per_tile, ci0 = cb * a.rows_per_tap;
    const long long k0 = static_cast<long long>(blockIdx.y) * a.kper;
    const int ksteps = static_cast<int>(min(static_cast<long long>(a.kper), a.kchunks - k0));

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&c->full[s], 1);
            mbar_init(&c->empty[s], 1);
        }
        mbar_init(&c->done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc(&c->tmem, N);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = c->tmem;

    if (warp == 0) {
        // slice k0: voxels p .. p + 63 of the y*x plane z of sample n
        int p = static_cast<int>(k0 % a.pchunks) * kWK;
        int z = static_cast<int>(k0 / a.pchunks % a.nz), n = static_cast<int>(k0 / a.pchunks / a.nz);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        int k = 0;
        for (; k < ksteps; ++k) {
            if (k >= kWStages) ok = __all_sync(0xffffffffu, mbar_wait(&c->empty[s], ph ^ 1));
            if (!ok) break;
            if (elect_one()) {
                uint8_t *sa = ring + s * stage;
                mbar_expect_tx(&c->full[s], stage);
                for (int j = 0; j < a.taps_per_tile; ++j) {
                    const int tap = min(tap0 + j, a.ntaps - 1);
                    int dz, dy, dx;
                    tap_offsets(tap, a.ntaps, dz, dy, dx);
                    const CUtensorMap *m = dx < 0 ? &mxm : (dx > 0 ? &mxp : &mx0);
                    tma_load4(sa + j * a.rows_per_tap * kWRowBytes, m, &c->full[s], p + dy * a.nx, z + dz, ci0, n);
                }
                tma_load4(sa + a_bytes, &mdy, &c->full[s], p, z, 0, n);
            }
            __syncwarp();
            if (++s == kWStages) {
                s = 0;
                ph ^= 1;
            }
            p += kWK;
            if (p >= a.pchunks * kWK) {
                p = 0;
                if (++z == a.nz) {
                    z = 0;
                    ++n;
                }
            }
        }
        if (!ok) flag_error(1);
        drain_loads<kWStages>(c, k);
    } else if (warp == 1) {
        mma_loop<N, kWStages, a_bytes, 1, 0, kWRowBytes>(c, ring, tmem, ksteps);
    }
    __syncwarp();

    const bool ok = mbar_wait(&c->done, 0);
    if (!ok) flag_error(4);
    tc_fence_after();
    const int r = warp * 32 + lane;
    const int tap = tap0 + r / a.rows_per_tap, ci = ci0 + r % a.rows_per_tap;
    const bool valid = ok && ksteps > 0 && tap < a.ntaps;
    const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    float *dst = a.dw + (valid ? static_cast<long long>(tap) * a.cin + ci : 0);   // rows past the last tap: unused
    const long long cstride = static_cast<long long>(a.ntaps) * a.cin;
#pragma unroll 1
    for (int c0 = 0; c0 < N; c0 += 16) {
        float v[16];
        tmem_ld16(trow + c0, v);
        if (valid) {
#pragma unroll
            for (int j = 0; j < 16; ++j) atomicAdd(dst + (c0 + j) * cstride, v[j]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) tmem_dealloc(tmem, N);
}

// ---------------------------------------------------------------------------
// Weight gradient straight from channels-last tensors: 32 input x 32 output
// channels and the nine taps of one dz per item.
//
// conv_wgrad_kernel wants its K dimension (voxels) contiguous, so the tensors
// are first copied channel-major, X three times, and each of its boxes gathers
// 128-byte rows that lie a whole volume apart.  Here the channels-last tensors are the
// operands as they are (MN-major: 32 channels of a voxel contiguous, voxels along
// K).  A K step is 16 consecutive voxels of X.  M = 3 boxes of X, one per dx, of 32 channels
// each (a fourth quarter of M reads what follows them and is dropped); N = the
// three dy: the voxels of dY one row before, at and one row after those of X, which
// lie one row apart in a ring of dY.  (Its first two rows are fetched a second time
// behind its end: a product split at the end costs 88 cycles of operand reads
// instead of 56, in 4 of 7 steps of 128-voxel rows.)  The CTA walks X in memory order in
// segments (rows or parts of one), so each row of either tensor is fetched once per dz.
//
// The sums are conv_wgrad_kernel's: a partial sum takes the same kper * 64 voxels of
// dY, every tap meets them in the same order and groups of 16, and it is added
// to dw the same way.  Adam divides a gradient by its own size, so a weight whose
// gradient is near zero follows its last bits, and one bf16 weight more or less
// moves the next step's gradients by 1e-3 of their norm.  (8 x 16 voxel tiles walked
// along z, with one fetch of X for all dz, took three quarters of the time, but sum in
// another order.)
//
// Bound by shared memory: 224 cycles of operand reads and 140 of TMA writes per 64
// voxels of one dz.  GB300, with the copies that conv_wgrad_kernel needs (before /
// after): 128^3, 32 x 32 channels 935 / 161 us, 64 x 32 1789 / 296; 64^3, 64 x 64 131 / 86,
// 128 x 64 225 / 162; 32^3, 64 x 128 40 / 35, but 128 x 128 54 / 59 (there every row of
// conv_wgrad_kernel's products is of use); 16^3, 256 x 256 38 / 53.
// ---------------------------------------------------------------------------
constexpr int kClStages = 16;

struct ClCtrl {
    uint64_t full[kClStages];
    uint64_t empty[kClStages];
    uint64_t accfull;
    uint64_t accempty[3];
    uint64_t done;
    uint32_t tmem;
};

struct ClArgs {
    int c1, cin, nz;
    int seg, bx, by;         // K steps of a segment; its x and y extent
    int nseg, spp;           // segments side by side along x, and per plane
    int boxes;               // 32-channel boxes of X per stage: the three dx, or (one tap) channel chunks
    int stages;              // of X
    int steps, chain;        // K steps of the volume and of a partial sum
    int items;
    float *dw;               // [cout][taps][cin], FP32, accumulated
};

// grid (CTAs, 32-channel chunks of X (`boxes` of them for one tap), 32-channel chunks of dY)
template <int TAPS>
__global__ void __launch_bounds__(192, 1)
conv_wgrad_cl_kernel(const __grid_constant__ CUtensorMap mx1, const __grid_constant__ CUtensorMap mx2,
                     const __grid_constant__ CUtensorMap mdy, const ClArgs a) {
    constexpr int NZ = TAPS == 27 ? 3 : 1;                 // dz per partial sum, dy per item
    constexpr uint32_t cols = TAPS == 27 ? 128 : 32;       // 32 NZ used
    extern __shared__ uint8_t smem_raw[];
    uint8_t *ring = align1024(smem_raw);
    const int h = TAPS == 27 ? a.nseg : 0;                 // segments from a voxel to the next row's
    const int S = a.stages, W = S + 2 * h;                 // stages of X, segments in the ring of dY (and 2 h twice)
    const uint32_t box = a.seg * 16 * kRowBytes, xstage = a.boxes * box;
    uint8_t *yring = ring + S * xstage;
    ClCtrl *c = reinterpret_cast<ClCtrl *>(yring + (W + 2 * h) * box);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int ci0 = blockIdx.y * 32 * (TAPS == 27 ? 1 : a.boxes), co0 = blockIdx.z * 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&c->full[s], 1);
            mbar_init(&c->empty[s], 1);
        }
        mbar_init(&c->accfull, 1);
        for (int e = 0; e < NZ; ++e) mbar_init(&c->accempty[e], a.boxes);
        mbar_init(&c->done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(&c->tmem, cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = c->tmem;

    // item i: K steps v0 .. v1 - 1 of dY in memory order, the taps of one dz
    auto item = [&](int i, int &v0, int &v1) {
        v0 = i / NZ * a.chain;
        v1 = min(v0 + a.chain, a.steps);
        return TAPS == 27 ? i % 3 - 1 : 0;
    };
    // Its segments ka .. kb - 1 of one plane, from segment sg of all planes.  The steps of such a run are the
    // segments k of X from ka - h to kb - 1 + h; dY of segment k + h comes with X of segment k.
    auto run = [&](int sg, int v1, int &plane, int &ka, int &kb) {
        plane = sg / a.spp;
        ka = sg - plane * a.spp;
        kb = min((v1 + a.seg - 1) / a.seg - plane * a.spp, a.spp);
    };
    int v0, v1, plane, ka, kb;

    if (warp == 4) {
        int s = 0, used = 0, w = 0;                        // stage, stages filled so far (up to S), slot of dY
        uint32_t ph = 0;
        bool ok = true;
        for (int i = blockIdx.x; ok && i < a.items; i += gridDim.x) {
            const int dz = item(i, v0, v1);
            for (int sg = v0 / a.seg; ok && sg * a.seg < v1; sg += kb - ka) {
                run(sg, v1, plane, ka, kb);
                const int n = plane / a.nz, z = plane - n * a.nz;
                int row = (ka - h + a.nseg) / a.nseg - 1;  // ka - h >= -nseg
                int x0 = (ka - h - row * a.nseg) * a.bx, y0 = row * a.by;
                for (int k = ka - h; k < kb + h; ++k) {
                    // step k's stage is free: so is the slot, whose dY the step before that stage's was the last to read
                    if (used == S) ok = __all_sync(0xffffffffu, mbar_wait(&c->empty[s], ph ^ 1));
                    if (!ok) break;
                    if (elect_one()) {
                        const bool dy = k + h >= ka && k + h < kb, twice = dy && w < 2 * h;
                        mbar_expect_tx(&c->full[s], xstage + (dy ? box : 0) + (twice ? box : 0));
                        for (int j = 0; j < a.boxes; ++j) {
                            const int ch = TAPS == 27 ? ci0 : ci0 + 32 * j;
                            const bool second = ch >= a.c1;
                            tma_load5(ring + s * xstage + j * box, second ? &mx2 : &mx1, &c->full[s],
                                      second ? ch - a.c1 : ch, TAPS == 27 ? x0 + j - 1 : x0, y0, z + dz, n);
                        }
                        const int yd = TAPS == 27 ? y0 + a.by : y0;
                        if (dy) tma_load5(yring + w * box, &mdy, &c->full[s], co0, x0, yd, z, n);
                        if (twice) tma_load5(yring + (W + w) * box, &mdy, &c->full[s], co0, x0, yd, z, n);
                    }
                    __syncwarp();
                    x0 += a.bx;
                    if (x0 == a.nseg * a.bx) {
                        x0 = 0;
                        y0 += a.by;
                    }
                    used = min(used + 1, S);
                    if (++w == W) w = 0;
                    if (++s == S) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
        if (!ok && lane == 0) flag_error(1);
        // every load has landed before the CTA may leave: the last use of stage j
        for (int j = 0; j < used; ++j) mbar_wait(&c->full[j], j < s ? ph : ph ^ 1);
    } else if (warp == 5) {
        // in K steps (1024 bytes): a row, and the part of it in a segment
        const int row = a.nseg * a.bx / 16, line = a.bx / 16;
        const uint64_t xd = sw64_mn_desc(smem_u32(ring), a.boxes > 1 ? box : 512);
        const uint64_t yd = sw64_mn_desc(smem_u32(yring), row * 1024);
        int s = 0, w = 0;
        uint32_t ph = 0, sums = 0;
        bool ok = true;
        for (int i = blockIdx.x; ok && i < a.items; i += gridDim.x) {
            item(i, v0, v1);
            for (int sg = v0 / a.seg; ok && sg * a.seg < v1; sg += kb - ka) {
                run(sg, v1, plane, ka, kb);
                const int pv = plane * a.spp * a.seg;                  // the plane's first K step
                const bool start = v0 >= pv;                           // the sum starts in this run
                const int pa = start ? v0 - pv : 0, pb = min(v1 - pv, a.spp * a.seg);   // the sum's dY in this plane
                for (int k = ka - h; k < kb + h; ++k) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&c->full[s], ph));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t xb = xd + static_cast<uint64_t>(s) * (xstage / 16);
                    const int y0 = (w >= h ? w - h : w - h + W) * a.seg;   // where dY of the same voxels is
                    // the segment's rows (or part of one): what holds for a row's first K step holds for all.  dY of
                    // p + (e - 1) row is met for dy = 1 - e.
                    for (int r = 0; r < a.seg; r += line) {
                        const int p = k * a.seg + r;
                        int e = TAPS == 1 ? 1 : (p >= pa + row ? 0 : (p >= pa ? 1 : (p >= pa - row ? 2 : 3)));
                        const int ee = TAPS == 1 ? 2 : (p + row < pb ? 3 : (p < pb ? 2 : (p - row < pb ? 1 : 0)));
                        while (e < ee) {
                            // a sum's first K step for e starts its accumulator, once it has been read
                            const bool first = start && p + (e - 1) * row == pa;
                            if (first && sums)
                                ok = __all_sync(0xffffffffu, mbar_wait(&c->accempty[TAPS == 1 ? 0 : e], (sums - 1) & 1));
                            if (!ok) break;
                            tc_fence_after();
                            const int len = first ? 1 : ee - e;
                            const int y = y0 + r + (e - 1) * row;
                            if (elect_one()) {
                                const uint64_t xg = xb + r * 64, yg = yd + (y < 0 ? y + W * a.seg : y) * 64;
                                const uint32_t d = tmem + (TAPS == 1 ? 0 : e * 32);
                                const uint32_t id = idesc_bf16_mn(kTileM, 32) + (len - 1) * (4u << 17);
#pragma unroll
                                for (int g = 0; g < 4; ++g)
                                    if (g < line) umma_bf16(d, xg + g * 64, yg + g * 64, id, g > 0 || !first);
                            }
                            __syncwarp();
                            e += len;
                        }
                        if (!ok) break;
                    }
                    if (!ok) break;
                    if (elect_one()) {
                        umma_commit(&c->empty[s]);
                        if (k == kb + h - 1 && pv + kb * a.seg >= v1) umma_commit(&c->accfull);
                    }
                    __syncwarp();
                    if (++w == W) w = 0;
                    if (++s == S) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            ++sums;
        }
        if (!ok && lane == 0) flag_error(2);
        if (elect_one()) umma_commit(&c->done);
    } else if (warp < a.boxes) {                           // warp = dx + 1 (or channel chunk), lane = input channel
        const long long cstride = static_cast<long long>(TAPS) * a.cin;
        const uint32_t trow = tmem + (static_cast<uint32_t>(warp * 32) << 16);
        uint32_t sums = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < a.items; i += gridDim.x, ++sums) {
            const int dz = item(i, v0, v1);
            ok = __all_sync(0xffffffffu, mbar_wait(&c->accfull, sums & 1));
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int e = NZ - 1; e >= 0; --e) {            // in the order in which the next sum wants them
                const int tap = TAPS == 27 ? (dz + 1) * 9 + (2 - e) * 3 + warp : 0;
                const int ci = ci0 + lane + (TAPS == 27 ? 0 : 32 * warp);
                float *dst = a.dw + co0 * cstride + static_cast<long long>(tap) * a.cin + ci;
#pragma unroll
                for (int b = 0; b < 32; b += 16) {
                    float v[16];
                    tmem_ld16(trow + e * 32 + b, v);
#pragma unroll
                    for (int q = 0; q < 16; ++q) atomicAdd(dst + (b + q) * cstride, v[q]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&c->accempty[e])) : "memory");
            }
        }
        if (!ok && lane == 0) flag_error(4);
    }
    __syncwarp();
    if (!mbar_wait(&c->done, 0)) flag_error(4);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 5) tmem_dealloc(tmem, cols);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// bf16 tensor map of the given rank; dims innermost first, strides in bytes
// for dims 1.., 64-byte swizzle, zero fill outside.
int make_map(CUtensorMap *m, const void *base, int rank, const uint64_t *dims, const uint64_t *strides,
             const uint32_t *box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_64B) {
    auto fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return CT_ERR_CUDA;
    }
    cuuint64_t gd[5], gs[4];
    cuuint32_t bd[5], es[5];
    for (int i = 0; i < rank; ++i) {
        gd[i] = dims[i];
        bd[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) gs[i] = strides[i];
    }
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(base), gd, gs, bd, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (" + std::to_string(static_cast<int>(r)) + ")");
        return CT_ERR_ARG;
    }
    return CT_OK;
}

// channels-last activation [n][z][y][x][c]: box 32 channels x bx x by x bz
int map_ndhwc(CUtensorMap *m, const void *p, int c, int nx, int ny, int nz, int nb, int bx, int by, int bz) {
    const uint64_t dims[5] = {(uint64_t)c, (uint64_t)nx, (uint64_t)ny, (uint64_t)nz, (uint64_t)nb};
    const uint64_t e = 2;
    const uint64_t st[4] = {c * e, (uint64_t)nx * c * e, (uint64_t)ny * nx * c * e, (uint64_t)nz * ny * nx * c * e};
    const uint32_t box[5] = {32, (uint32_t)bx, (uint32_t)by, (uint32_t)bz, 1};
    return make_map(m, p, 5, dims, st, box);
}

// channel-major activation [n][c][z][y*x]: box 64 voxels x rows channels, 128-byte swizzle
int map_ncdhw(CUtensorMap *m, const void *p, int c, int nxy, int nz, int nb, int rows) {
    const uint64_t dims[4] = {(uint64_t)nxy, (uint64_t)nz, (uint64_t)c, (uint64_t)nb};
    const uint64_t e = 2;
    const uint64_t st[3] = {(uint64_t)nxy * e, (uint64_t)nz * nxy * e, (uint64_t)c * nz * nxy * e};
    const uint32_t box[4] = {(uint32_t)kWK, 1, (uint32_t)rows, 1};
    return make_map(m, p, 4, dims, st, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Dynamic shared memory of a ring (plus alignment slack and the control block).
// Every size here keeps the CTAs an SM can hold at <= 512 TMEM columns in total.
template <int N>
size_t ring_smem() {
    return 1024 + kStages * (kABytes + N * kRowBytes) + sizeof(Ctrl);
}

template <int N>
size_t wring_smem() {
    return 1024 + kWStages * (kTileM * kWRowBytes + N * kWRowBytes) + sizeof(Ctrl);
}

template <int N>
size_t yring_smem() {
    return 1024 + kYStages * (kYABytes + 3 * N * kRowBytes) + sizeof(Ctrl);
}

// A kernel's shared memory above 48 KB is granted per device: asked for at each launch.
int grant_smem(const void *kernel, size_t smem) {
    CT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "convolution smem");
    return CT_OK;
}

template <int N, bool YR>
int launch_fwd(const CUtensorMap &m1, const CUtensorMap &m2, const CUtensorMap &mw, const FwdArgs &a, int tiles,
               cudaStream_t st) {
    const size_t smem = YR ? yring_smem<N>() : ring_smem<N>();
    if (int e = grant_smem((const void *)conv_fwd_kernel<N, YR>, smem)) return e;
    conv_fwd_kernel<N, YR><<<tiles, 128, smem, st>>>(m1, m2, mw, a);
    CT_LAUNCH_CHECK("conv_fwd_kernel");
    return CT_OK;
}

template <int N, int NCH>
constexpr size_t march_smem() {
    return 1024 + 27 * NCH * N * kRowBytes + kMGroups * kMBoxes * kYABytes + sizeof(MarchCtrl);
}

// Slices per item: the groups of the persistent CTAs share ceil(items / groups) items each, and an item of zc outputs
// reads zc + 2 slices; the zc with the fewest slices read by the busiest group, the longer one of equals.
template <int N, int NCH, bool HEAD = false>
int launch_march(const CUtensorMap &m1, const CUtensorMap &m2, const CUtensorMap &mw, const FwdArgs &f, int nb,
                 cudaStream_t st) {
    MarchArgs a{};
    a.f = f;
    a.tx = f.nx / kYBx;
    a.ty = f.ny / kYBy;
    a.parts = (f.co1 + f.co2) / N;
    const long long cols = (long long)nb * a.tx * a.ty, groups = (long long)kMGroups * std::max(1, sm_count() / a.parts);
    long long best = -1;
    for (int chunks = 1; chunks <= f.nz; ++chunks) {
        const int zc = (f.nz + chunks - 1) / chunks;
        const long long items = cols * ((f.nz + zc - 1) / zc), cost = (items + groups - 1) / groups * (zc + 2);
        if (best >= 0 && cost >= best) continue;
        best = cost;
        a.zc = zc;
        a.items = items;
    }
    a.nzc = (f.nz + a.zc - 1) / a.zc;
    constexpr size_t smem = march_smem<N, NCH>();
    if (int e = grant_smem((const void *)conv_march_kernel<N, NCH, HEAD>, smem)) return e;
    conv_march_kernel<N, NCH, HEAD><<<(unsigned)((std::min(a.items, groups) + kMGroups - 1) / kMGroups * a.parts), 192 * kMGroups, smem, st>>>(m1, m2, mw, a);
    CT_LAUNCH_CHECK("conv_march_kernel");
    return CT_OK;
}

template <int N>
int launch_wgrad(const CUtensorMap &mm, const CUtensorMap &m0, const CUtensorMap &mp, const CUtensorMap &md,
                 const WgradArgs &a, dim3 grid, cudaStream_t st) {
    const size_t smem = wring_smem<N>();
    if (int e = grant_smem((const void *)conv_wgrad_kernel<N>, smem)) return e;
    conv_wgrad_kernel<N><<<grid, 128, smem, st>>>(mm, m0, mp, md, a);
    CT_LAUNCH_CHECK("conv_wgrad_kernel");
    return CT_OK;
}

// Bytes of a CTA's rings and control block, and the stages of X that fit beside `per_sm` CTAs on an SM (1 KB of each is
// the system's).
size_t cl_smem(const ClArgs &a, int h, int stages) {
    return 1024 + (size_t)a.seg * 16 * kRowBytes * (stages * a.boxes + stages + 4 * h) + sizeof(ClCtrl);
}

int cl_stages(const ClArgs &a, int h, int per_sm) {
    int s = 0;
    while (s < kClStages && cl_smem(a, h, s + 1) <= (228u / per_sm - 1) * 1024) ++s;
    return s;
}

template <int TAPS>
int launch_wgrad_cl(const CUtensorMap &m1, const CUtensorMap &m2, const CUtensorMap &md, ClArgs a, int cout, cudaStream_t st) {
    const int h = TAPS == 27 ? a.nseg : 0;
    // CTAs per SM, one's waits under the others' instructions: 3 where each can load two segments ahead, else 2.  128^3,
    // 32 x 32 channels (2 stages with 3 CTAs): 161 / 178 / 179 us with 2 / 3 / 4; 64^3, 64 x 64 (3 stages): 89 / 86 / 136;
    // 32^3, 128 x 128: 66 / 59 / 73.
    int per_sm = cl_stages(a, h, 3) >= 3 ? 3 : (cl_stages(a, h, 2) >= 2 ? 2 : 1);
    a.stages = cl_stages(a, h, per_sm);
    const size_t smem = cl_smem(a, h, a.stages);
    if (int e = grant_smem((const void *)conv_wgrad_cl_kernel<TAPS>, smem)) return e;
    const int gy = a.cin / (TAPS == 27 ? 32 : 32 * a.boxes), gz = cout / 32;
    const int ctas = std::max(1, per_sm * sm_count() / (gy * gz));
    conv_wgrad_cl_kernel<TAPS><<<dim3((unsigned)std::min(a.items, ctas), gy, gz), 192, smem, st>>>(m1, m2, md, a);
    CT_LAUNCH_CHECK("conv_wgrad_cl_kernel");
    return CT_OK;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

bool valid_n(int n) { return n == 32 || n == 64 || n == 128 || n == 256; }

}  // namespace

}  // namespace ct

using namespace ct;

extern "C" {

int ct_unet_conv3d(const void *x1, int c1, const void *x2, int c2, int nb, int nz, int ny, int nx, const void *w,
                   int ntaps, const float *bias, int relu, void *out1, int co1, void *out2, int co2,
                   const void *mask1, const void *mask2, void *stream) {
    CT_REQUIRE(x1 && w && out1, "conv3d: null pointer");
    CT_REQUIRE(ntaps == 1 || ntaps == 27, "conv3d: ntaps must be 1 or 27");
    CT_REQUIRE(c1 > 0 && c1 % 32 == 0 && c2 >= 0 && c2 % 32 == 0 && (c2 == 0 || x2),
               "conv3d: input channels must be positive multiples of 32");
    const int n = co1 + co2;
    CT_REQUIRE(valid_n(n) && co1 > 0 && co1 % 16 == 0 && co2 % 16 == 0 && (co2 == 0 || out2),
               "conv3d: output channels must total 32, 64, 128 or 256, split at a multiple of 16");
    CT_REQUIRE(nb > 0 && nz > 0 && ny > 0 && nx > 0, "conv3d: empty volume");
    // y-halo tiles (8 x 16 voxels, the three dy taps from one box) where they fit
    const bool yr = ntaps == 27 && n <= 128 && nx % kYBx == 0 && ny % kYBy == 0;
    int bx, by, bz;
    if (yr) {
        bx = kYBx;
        by = kYBy;
        bz = 1;
    } else {
        bx = nx >= 128 ? 128 : nx;
        CT_REQUIRE(128 % bx == 0 && nx % bx == 0, "conv3d: x must be a divisor or a multiple of 128");
        by = ny >= 128 / bx ? 128 / bx : ny;
        CT_REQUIRE((128 / bx) % by == 0 && ny % by == 0, "conv3d: y must fit the 128-voxel tile");
        bz = 128 / (bx * by);
        CT_REQUIRE(nz % bz == 0, "conv3d: z must be a multiple of 128 / (x * y) for small slices");
    }
    CT_REQUIRE(aligned16(x1) && aligned16(w) && aligned16(out1) && (!x2 || aligned16(x2)) &&
                   (!out2 || aligned16(out2)) && (!mask1 || aligned16(mask1)) && (!mask2 || aligned16(mask2)),
               "conv3d: pointers must be 16-byte aligned");
    const long long tiles = (long long)nb * (nz / bz) * (ny / by) * (nx / bx);
    CT_REQUIRE(tiles < (1ll << 31), "conv3d: too many tiles");
    // Outputs per CTA of the z-marching kernel where its filters fit in shared memory (64 outputs of 64 channels in
    // two halves), else 0.  It starts by loading the filters (about 8 us for 110 KB) and walks several slices per CTA:
    // a volume that conv_fwd_kernel covers in about one wave of its four CTAs per SM is left to that.  32^3 (256 tiles):
    // 12.5 us there, 16.0 here for 64 -> 32 channels, 8.8 / 8.6 for 32 -> 32; 48^3 (864 tiles): 25.1 / 21.9, 16.3 / 11.9.
    const int march = !yr || n > 64 || tiles <= 4LL * sm_count() ? 0 : (c1 + c2 == 32 ? n : (c1 + c2 == 64 ? 32 : 0));
    CUtensorMap m1, m2, mw;
    int s;
    const int box_y = yr ? by + 2 : by;
    if ((s = map_ndhwc(&m1, x1, c1, nx, ny, nz, nb, bx, box_y, bz))) return s;
    if ((s = map_ndhwc(&m2, c2 ? x2 : x1, c2 ? c2 : c1, nx, ny, nz, nb, bx, box_y, bz))) return s;
    {
        const int cin = c1 + c2;
        const uint64_t dims[3] = {(uint64_t)cin, (uint64_t)ntaps, (uint64_t)n};
        const uint64_t st[2] = {(uint64_t)cin * 2, (uint64_t)ntaps * cin * 2};
        const uint32_t box[3] = {32, 1, (uint32_t)(march ? march : n)};
        if ((s = make_map(&mw, w, 3, dims, st, box))) return s;
    }
    FwdArgs a{};
    a.c1 = c1;
    a.c2 = c2;
    a.ntaps = ntaps;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.bx = bx;
    a.by = by;
    a.bz = bz;
    a.ksteps = (yr ? 9 : ntaps) * (c1 + c2) / 32;
    a.bias = bias;
    a.relu = relu;
    a.out1 = static_cast<__nv_bfloat16 *>(out1);
    a.out2 = static_cast<__nv_bfloat16 *>(out2);
    a.co1 = co1;
    a.co2 = co2;
    a.mask1 = static_cast<const __nv_bfloat16 *>(mask1);
    a.mask2 = static_cast<const __nv_bfloat16 *>(mask2);
    cudaStream_t st = as_stream(stream);
    if (march) {
        if (c1 + c2 == 64) return launch_march<32, 2>(m1, m2, mw, a, nb, st);
        return march == 32 ? launch_march<32, 1>(m1, m2, mw, a, nb, st) : launch_march<64, 1>(m1, m2, mw, a, nb, st);
    }
    if (yr) {
        switch (n) {
            case 32: return launch_fwd<32, true>(m1, m2, mw, a, (int)tiles, st);
            case 64: return launch_fwd<64, true>(m1, m2, mw, a, (int)tiles, st);
            default: return launch_fwd<128, true>(m1, m2, mw, a, (int)tiles, st);
        }
    }
    switch (n) {
        case 32: return launch_fwd<32, false>(m1, m2, mw, a, (int)tiles, st);
        case 64: return launch_fwd<64, false>(m1, m2, mw, a, (int)tiles, st);
        case 128: return launch_fwd<128, false>(m1, m2, mw, a, (int)tiles, st);
        default: return launch_fwd<256, false>(m1, m2, mw, a, (int)tiles, st);
    }
}

int ct_unet_conv3d_wgrad(const void *xm, const void *x0, const void *xp, int cin, const void *dy, int cout, int nb,
                         int nz, int ny, int nx, int ntaps, int kper, float *dw, void *stream) {
    CT_REQUIRE(x0 && dy && dw && (ntaps == 1 || (xm && xp)), "conv3d_wgrad: null pointer");
    CT_REQUIRE(ntaps == 1 || ntaps == 27, "conv3d_wgrad: ntaps must be 1 or 27");
    CT_REQUIRE(cin > 0 && cin % 32 == 0, "conv3d_wgrad: input channels must be a positive multiple of 32");
    CT_REQUIRE(valid_n(cout), "conv3d_wgrad: output channels must be 32, 64, 128 or 256");
    CT_REQUIRE(nb > 0 && nz > 0 && ny > 0 && nx > 0 && nx % 8 == 0 && (long long)nx * ny < (1ll << 30),
               "conv3d_wgrad: x must be a multiple of 8");
    CT_REQUIRE(kper > 0, "conv3d_wgrad: kper must be positive");
    CT_REQUIRE(aligned16(x0) && aligned16(dy) && (!xm || aligned16(xm)) && (!xp || aligned16(xp)),
               "conv3d_wgrad: pointers must be 16-byte aligned");
    const int nxy = nx * ny;
    const int rows = cin >= 128 ? 128 : cin;
    CUtensorMap mm, m0, mp, md;
    int s;
    if ((s = map_ncdhw(&m0, x0, cin, nxy, nz, nb, rows))) return s;
    if ((s = map_ncdhw(&mm, ntaps == 27 ? xm : x0, cin, nxy, nz, nb, rows))) return s;
    if ((s = map_ncdhw(&mp, ntaps == 27 ? xp : x0, cin, nxy, nz, nb, rows))) return s;
    if ((s = map_ncdhw(&md, dy, cout, nxy, nz, nb, cout))) return s;
    WgradArgs a{};
    a.cin = cin;
    a.ntaps = ntaps;
    a.rows_per_tap = rows;
    a.taps_per_tile = 128 / rows;
    a.cblocks = cin / rows;
    a.nxy = nxy;
    a.nx = nx;
    a.nz = nz;
    // a slice past the end of a plane reads zeros for dY, so it adds nothing
    a.pchunks = (nxy + kWK - 1) / kWK;
    a.kchunks = (long long)nb * nz * a.pchunks;
    a.kper = kper;
    a.dw = dw;
    const int ttiles = (ntaps + a.taps_per_tile - 1) / a.taps_per_tile;
    const long long ksplit = (a.kchunks + kper - 1) / kper;
    CT_REQUIRE(ksplit <= 65535, "conv3d_wgrad: too many K splits (raise kper)");
    dim3 grid(ttiles * a.cblocks, (unsigned)ksplit);
    cudaStream_t st = as_stream(stream);
    switch (cout) {
        case 32: return launch_wgrad<32>(mm, m0, mp, md, a, grid, st);
        case 64: return launch_wgrad<64>(mm, m0, mp, md, a, grid, st);
        case 128: return launch_wgrad<128>(mm, m0, mp, md, a, grid, st);
        default: return launch_wgrad<256>(mm, m0, mp, md, a, grid, st);
    }
}

int ct_unet_conv3d_wgrad_cl(const void *x1, int c1, const void *x2, int c2, const void *dy, int cout, int nb, int nz,
                            int ny, int nx, int ntaps, int kper, float *dw, void *stream) {
    CT_REQUIRE(x1 && dy && dw && (c2 == 0 || x2), "conv3d_wgrad_cl: null pointer");
    CT_REQUIRE(ntaps == 1 || ntaps == 27, "conv3d_wgrad_cl: ntaps must be 1 or 27");
    CT_REQUIRE(c1 > 0 && c1 % 32 == 0 && c2 >= 0 && c2 % 32 == 0 && cout > 0 && cout % 32 == 0 &&
                   c1 <= 32 * 65535 - c2 && cout <= 32 * 65535,
               "conv3d_wgrad_cl: channels must be positive multiples of 32");
    CT_REQUIRE(nb > 0 && nz > 0 && ny > 0 && nx > 0 && (long long)nx * ny < (1ll << 30),
               "conv3d_wgrad_cl: empty volume, or a plane too large");
    CT_REQUIRE(kper > 0, "conv3d_wgrad_cl: kper must be positive");
    CT_REQUIRE(aligned16(x1) && aligned16(dy) && (!x2 || aligned16(x2)),
               "conv3d_wgrad_cl: pointers must be 16-byte aligned");
    // Segments: 64 voxels, in whole rows where x is 16 or 32, or the largest power of two that
    // divides x: partial sums (of 64 voxels) then end with one.
    ClArgs a{};
    a.by = nx == 16 || nx == 32 ? 64 / nx : 1;
    a.bx = std::min(nx & -nx, 64);
    CT_REQUIRE(nx % 16 == 0 && ny % a.by == 0 && nx * ny % kWK == 0,
               "conv3d_wgrad_cl: x must be a multiple of 16 and x * y of 64");
    const int seg = a.bx * a.by;
    a.seg = seg / 16;
    a.nseg = nx / a.bx;
    a.spp = nx * ny / seg;
    a.c1 = c1;
    a.cin = c1 + c2;
    a.nz = nz;
    a.boxes = 3;
    if (ntaps == 1)
        for (a.boxes = 2; a.cin / 32 % a.boxes;) --a.boxes;
    CT_REQUIRE(cl_stages(a, ntaps == 27 ? a.nseg : 0, 1) >= 2, "conv3d_wgrad_cl: rows too long");
    const long long vox = (long long)nb * nz * ny * nx, ksplit = (vox / kWK + kper - 1) / kper;
    CT_REQUIRE(ksplit <= 65535, "conv3d_wgrad_cl: too many K splits (raise kper)");
    CT_REQUIRE(vox / 16 < (1ll << 30), "conv3d_wgrad_cl: volume too large");
    a.steps = (int)(vox / 16);
    a.chain = (int)std::min<long long>(4ll * kper, a.steps);
    a.items = (int)ksplit * (ntaps == 27 ? 3 : 1);
    a.dw = dw;
    CUtensorMap m1, m2, md;
    int s;
    if ((s = map_ndhwc(&m1, x1, c1, nx, ny, nz, nb, a.bx, a.by, 1))) return s;
    if ((s = map_ndhwc(&m2, c2 ? x2 : x1, c2 ? c2 : c1, nx, ny, nz, nb, a.bx, a.by, 1))) return s;
    if ((s = map_ndhwc(&md, dy, cout, nx, ny, nz, nb, a.bx, a.by, 1))) return s;
    cudaStream_t st = as_stream(stream);
    return ntaps == 27 ? launch_wgrad_cl<27>(m1, m2, md, a, cout, st) : launch_wgrad_cl<1>(m1, m2, md, a, cout, st);
}

int ct_unet_conv3d_head(const void *x, int nb, int nz, int ny, int nx, const void *w, const float *bias, int relu,
                        const float *head_w, const float *head_b, const float *base, float *out, void *stream) {
    CT_REQUIRE(x && w && head_w && head_b && out, "conv3d_head: null pointer");
    CT_REQUIRE(nb > 0 && nz > 0 && ny > 0 && nx > 0 && nx % kYBx == 0 && ny % kYBy == 0,
               "conv3d_head: x must be a multiple of 8, y of 16");
    CT_REQUIRE(aligned16(x) && aligned16(w), "conv3d_head: pointers must be 16-byte aligned");
    const long long tiles = (long long)nb * nz * (ny / kYBy) * (nx / kYBx);
    CT_REQUIRE(tiles < (1ll << 31), "conv3d_head: too many tiles");
    CUtensorMap m, mw;
    int s;
    if ((s = map_ndhwc(&m, x, 32, nx, ny, nz, nb, kYBx, kYBy + 2, 1))) return s;
    const uint64_t dims[3] = {32, 27, 32}, st[2] = {64, 27 * 64};
    const uint32_t box[3] = {32, 1, 32};
    if ((s = make_map(&mw, w, 3, dims, st, box))) return s;
    FwdArgs a{};
    a.c1 = 32;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.bias = bias;
    a.relu = relu;
    a.co1 = 32;
    a.head_w = head_w;
    a.head_b = head_b;
    a.base = base;
    a.head_out = out;
    return launch_march<32, 1, true>(m, m, mw, a, nb, as_stream(stream));
}

int ct_unet_conv_first(const float *vol, int nb, int nz, int ny, int nx, const void *w, const float *bias, int relu,
                       void *out, void *stream) {
    CT_REQUIRE(vol && w && out, "conv_first: null pointer");
    CT_REQUIRE(nb > 0 && nz > 0 && ny > 0 && nx > 0, "conv_first: empty volume");
    CT_REQUIRE(aligned16(w) && aligned16(out), "conv_first: pointers must be 16-byte aligned");
    const long long nvox = (long long)nb * nz * ny * nx;
    CT_REQUIRE(nvox % 128 == 0 && nvox / 128 < (1ll << 31), "conv_first: voxels must be a multiple of 128");
    FirstArgs a{};
    a.vol = vol;
    a.w = static_cast<const __nv_bfloat16 *>(w);
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.tiles = nvox / 128;
    a.small = nvox <= 0xffffffffll;
    a.relu = relu;
    a.bias = bias;
    a.out = static_cast<__nv_bfloat16 *>(out);
    // as many CTAs as fit at once: one's gathers run under another's instructions and stores
    const unsigned grid = (unsigned)std::min<long long>(a.tiles, kFirstCtas * (long long)sm_count());
    conv_first_kernel<<<grid, 128, 0, as_stream(stream)>>>(a);
    CT_LAUNCH_CHECK("conv_first_kernel");
    return CT_OK;
}

int ct_unet_wait_selftest(long long limit_ns, void *stream) {
    CT_REQUIRE(limit_ns >= 1000 && limit_ns <= 1000000000LL, "unet_wait_selftest: limit must be in [1 us, 1 s]");
    wait_selftest_kernel<<<1, 32, 0, as_stream(stream)>>>((unsigned long long)limit_ns);
    CT_LAUNCH_CHECK("wait_selftest_kernel");
    return CT_OK;
}

int ct_unet_status(int *flags) {
    CT_REQUIRE(flags, "unet_status: null pointer");
    int zero = 0;
    CT_CUDA(cudaMemcpyFromSymbol(flags, g_unet_err, sizeof(int)), "unet_status read");
    CT_CUDA(cudaMemcpyToSymbol(g_unet_err, &zero, sizeof(int)), "unet_status reset");
    if (*flags) {
        set_error("a tensor-core convolution gave up on a bounded wait (flags " + std::to_string(*flags) + ")");
        return CT_ERR_TIMEOUT;
    }
    return CT_OK;
}

}  // extern "C"

// kernels_learn.cu -- the learned warm start on the 5th-generation tensor cores (sm_103a).
//
// Every convolution of the encoder-decoder, forward and backward, is an implicit GEMM on tcgen05: BF16 operands
// staged in shared memory, FP32 accumulation in tensor memory (TMEM), one thread issuing tcgen05.mma for the CTA,
// completion signalled by tcgen05.commit on an mbarrier, and an epilogue that reads the accumulator with
// tcgen05.ld and applies bias / skip addend / ReLU / ReLU-derivative mask before writing FP32 or BF16.
//
//   forward  : Y[pixel][co]  = sum_(tap,ci) X[pixel * s + tap][ci] W[co][tap,ci]            (k_conv_tc)
//   data grad: dX[pixel][ci] = sum_(tap,co) dY[(pixel - tap) / s][co] W[co][tap,ci]         (k_conv_tc, dgrad)
//   weight   : dW[co][tap,ci] = sum_pixel X[pixel * s + tap][ci] dY[pixel][co]            (k_wgrad_tc, split-K)
//
// Activations are NHWC BF16 (channels contiguous, a multiple of 8), so one 16-byte load of the gather moves 8
// consecutive K elements of one tap. Shared-memory operand layout (K-major, no swizzle): 8 x 16-byte "core
// matrices" (8 rows x 8 bf16). Element (row r, k) of a 64-wide K stage sits at byte
// ((r / 8) * 8 + k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2: core matrices adjacent in K are 128 B apart (leading
// byte offset), 8-row groups 1 KB apart (stride byte offset); one MMA (K = 16) reads two core matrices along K, so
// the descriptor start advances 256 B per MMA.
#include <algorithm>
#include <atomic>

#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include "device_common.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace lfrv {

namespace {

constexpr int kBM = 128, kBK = 64, kThreads = 128, kStages = 4;

// Shared-memory matrix descriptor: start >> 4 in bits 0-13, leading byte offset >> 4 in 16-29, stride byte
// offset >> 4 in 32-45, the fixed version field (1) in 46-47, base offset 0, layout type 0 (no swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo = 128, uint32_t sbo = 1024) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::f16: D = F32 (bits 4-5 = 1), A = B = BF16 (bits 7-9 = 1, 10-12 = 1), both
// K-major (bits 15, 16 = 0; kMnMajor sets both), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
constexpr uint32_t kMnMajor = (1u << 15) | (1u << 16);
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int acc) {
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

// Arrives on the mbarrier once every tcgen05.mma this thread issued before it has completed.
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, int cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_free(uint32_t tmem, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

// 16 consecutive accumulator columns of this thread's TMEM lane (warp w of the CTA reads lanes 32 w .. 32 w + 31).
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16-byte global -> shared copy; bytes = 0 writes zeros (the source is not read).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Byte offset of the 16-byte chunk (row r, K chunk kc) of a 64-wide stage in the core-matrix layout.
__device__ __forceinline__ uint32_t tile_off(int r, int kc) {
    return (uint32_t)(((r >> 3) * 8 + kc) << 7) + (uint32_t)((r & 7) << 4);
}

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
    return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 1023) & ~(uintptr_t)1023);
}

__device__ __forceinline__ void unpack8(const uint4 &u, float f[8]) {
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float f[8]) {
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return u;
}

// Source pixel of tap (ky, kx) for GEMM row (y, x): forward rows are output pixels (input = y * s - 1 + ky for
// 3 x 3 with padding 1); data-gradient rows are the forward input pixels, whose contributions come from the output
// pixel (y + 1 - ky) / s when that division is exact.
__device__ __forceinline__ bool conv_src(const ConvGemm &g, int y, int x, int ky, int kx, int &iy, int &ix) {
    if (!g.dgrad) {
        iy = y * g.stride + (g.ks == 3 ? ky - 1 : 0);
        ix = x * g.stride + (g.ks == 3 ? kx - 1 : 0);
    } else {
        const int ty = y + (g.ks == 3 ? 1 - ky : 0), tx = x + (g.ks == 3 ? 1 - kx : 0);
        if (ty < 0 || tx < 0) return false;
        if (g.stride == 2) {
            if ((ty | tx) & 1) return false;
            iy = ty >> 1;
            ix = tx >> 1;
        } else {
            iy = ty;
            ix = tx;
        }
    }
    return iy >= 0 && iy < g.Hs && ix >= 0 && ix < g.Ws;
}

// What the epilogue of 16 columns reads besides the accumulator: the skip values of a 2 x 2 block ([2 d], [2 d + 1] for
// pixel d) with upskip (UP), else the addend ([0], [1]) and the mask ([2], [3]). Loaded ahead of the accumulator, so that its
// latency passes during the matrix products.
template <bool UP>
struct EpilogueIn {
    uint4 u[UP ? 8 : 4];
};

__device__ __forceinline__ size_t upskip_row(const ConvGemm &g, size_t row, int d) {
    const size_t HW = (size_t)g.Ho * g.Wo, b = row / HW, rem = row - b * HW;
    const int y = (int)(rem / g.Wo), x = (int)(rem - (size_t)y * g.Wo);
    return (b * 2 * g.Ho + 2 * y + (d >> 1)) * (size_t)(2 * g.Wo) + 2 * x + (d & 1);
}

template <bool UP>
__device__ __forceinline__ void conv_load16(const ConvGemm &g, size_t row, int col, EpilogueIn<UP> &in) {
    if constexpr (UP) {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const uint4 *sp = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(g.upskip) +
                                                              upskip_row(g, row, d) * g.N + col);
            in.u[2 * d] = sp[0];
            in.u[2 * d + 1] = sp[1];
        }
        return;
    }
    const size_t o = row * g.N + col;
    if (g.add) {
        const uint4 *ap = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(g.add) + o);
        in.u[0] = ap[0];
        in.u[1] = ap[1];
    }
    if (g.mask) {
        const uint4 *mp = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(g.mask) + o);
        in.u[2] = mp[0];
        in.u[3] = mp[1];
    }
}

// Epilogue of 16 accumulator columns (col .. col + 15) of GEMM row `row` (an output pixel, row-major over batch,
// Ho, Wo): + bias, + add, ReLU, zero where mask <= 0, then the FP32 and / or BF16 stores. With upskip (and no addend)
// the row's value goes, as relu(v + skip), to its 2 x 2 block of the doubled-resolution BF16 output. `bias`: the 16
// columns' biases in shared memory.
template <bool UP>
__device__ __forceinline__ void conv_store16(const ConvGemm &g, size_t row, int col, float v[16],
                                             const EpilogueIn<UP> &in, const float *bias) {
    const size_t o = row * g.N + col;
    if (g.bias) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 b = reinterpret_cast<const float4 *>(bias)[k];
            v[4 * k] += b.x;
            v[4 * k + 1] += b.y;
            v[4 * k + 2] += b.z;
            v[4 * k + 3] += b.w;
        }
    }
    if constexpr (UP) {
        __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(g.outb);
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            float a[8], c[8], w0[8], w1[8];
            unpack8(in.u[2 * d], a);
            unpack8(in.u[2 * d + 1], c);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                w0[k] = fmaxf(v[k] + a[k], 0.f);
                w1[k] = fmaxf(v[8 + k] + c[k], 0.f);
            }
            uint4 *bp = reinterpret_cast<uint4 *>(out + upskip_row(g, row, d) * g.N + col);
            bp[0] = pack8(w0);
            bp[1] = pack8(w1);
        }
        return;
    }
    if (g.add) {
        float tt[8];
        unpack8(in.u[0], tt);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] += tt[k];
        unpack8(in.u[1], tt);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[8 + k] += tt[k];
    }
    if (g.relu) {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k], 0.f);
    }
    if (g.mask) {
        float tt[8];
        unpack8(in.u[2], tt);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = tt[k] > 0.f ? v[k] : 0.f;
        unpack8(in.u[3], tt);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[8 + k] = tt[k] > 0.f ? v[8 + k] : 0.f;
    }
    if (g.outf && g.outf_head) {
        if (col == 0) *reinterpret_cast<float4 *>(g.outf + row * 4) = make_float4(v[0], v[1], v[2], v[3]);
    } else if (g.outf) {
        float4 *fp = reinterpret_cast<float4 *>(g.outf + o);
#pragma unroll
        for (int k = 0; k < 4; ++k) fp[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
    if (g.outb) {
        uint4 *bp = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(g.outb) + o);
        bp[0] = pack8(v);
        bp[1] = pack8(v + 8);
    }
}

}  // namespace

// One CTA: 128 GEMM rows (pixels) x BN output channels (columns n0 = blockIdx.y * BN ..), K in 64-wide stages through a kStages-deep
// cp.async ring. Thread 0 issues the four K = 16 MMAs of a stage once the stage has landed and commits them to
// the stage's mbarrier; a slot is refilled only after the mbarrier shows that the MMAs reading it completed.
template <int BN, bool UP>
__global__ void __launch_bounds__(kThreads) k_conv_tc(const ConvGemm g, int *err) {
    extern __shared__ uint8_t dsm[];
    constexpr int kAB = kBM * kBK * 2, kStage = kAB + BN * kBK * 2;
    constexpr int kCols = BN < 32 ? 32 : BN;
    __shared__ __align__(8) uint64_t bars[kStages];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ __align__(16) float s_bias[BN];
    uint8_t *base = align1024(dsm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int M = g.batch * g.Ho * g.Wo, HWo = g.Ho * g.Wo;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(&bars[s], 1);
        s_fail = 0;
        fence_proxy_async_smem();
    }
    // this thread's eight gather rows (fixed over K) and K chunk
    const int rlo = tid & 7, kc = (tid >> 3) & 7, rhi = tid >> 6;
    int rbase[8], ry[8], rx[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = m0 + (rhi + 2 * j) * 8 + rlo;
        if (m < M) {
            const int b = m / HWo, rem = m - b * HWo, y = rem / g.Wo;
            rbase[j] = b * g.Hs * g.Ws;
            ry[j] = y;
            rx[j] = rem - y * g.Wo;
        } else {
            rbase[j] = 0;
            ry[j] = -(1 << 28);
            rx[j] = -(1 << 28);
        }
    }
    const __nv_bfloat16 *src = static_cast<const __nv_bfloat16 *>(g.src);
    const __nv_bfloat16 *wt = static_cast<const __nv_bfloat16 *>(g.wt);
    const uint32_t sbase = smem_u32(base);
    auto load_stage = [&](int kt, int slot) {
        const uint32_t sa = sbase + slot * kStage, sb = sa + kAB;
        const int k = kt * kBK + kc * 8;
        const bool kvalid = k < g.K;
        int tap = 0, ci = 0;
        if (kvalid) {
            tap = k / g.C;
            ci = k - tap * g.C;
        }
        const int ky = (g.ks == 3) ? tap / 3 : 0, kx = (g.ks == 3) ? tap - ky * 3 : 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int iy = 0, ix = 0;
            const bool ok = kvalid && conv_src(g, ry[j], rx[j], ky, kx, iy, ix);
            const __nv_bfloat16 *p = ok ? src + (size_t)(rbase[j] + iy * g.Ws + ix) * g.C + ci : src;
            cp_async16(sa + tile_off((rhi + 2 * j) * 8 + rlo, kc), p, ok ? 16 : 0);
        }
#pragma unroll
        for (int j = 0; j < BN / 16; ++j) {
            const int r = (rhi + 2 * j) * 8 + rlo;
            cp_async16(sb + tile_off(r, kc), wt + (size_t)(n0 + r) * g.ldw + kt * kBK + kc * 8, 16);
        }
    };
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();
    pdl_wait();
    for (int c = tid; g.bias && c < BN; c += kThreads) s_bias[c] = __ldcg(g.bias + n0 + c);  // read after the loop's barriers
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16_f32(kBM, BN);
    const int nk = (g.K + kBK - 1) / kBK;
#pragma unroll 1
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_async_commit();
    }
    int issued = 0;  // stages whose MMAs were committed
#pragma unroll 1
    for (int kt = 0; kt < nk; ++kt) {
        const int slot = kt % kStages;
        cp_async_wait<kStages - 2>();  // stage kt has landed
        fence_proxy_async_smem();      // make this thread's shared-memory writes visible to the tensor core
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (s_fail) break;
        if (tid == 0) {
            const uint32_t a = sbase + slot * kStage, b = a + kAB;
#pragma unroll
            for (int s = 0; s < kBK / 16; ++s)
                tc_mma(tmem, smem_desc(a + s * 256), smem_desc(b + s * 256), idesc, (kt > 0 || s > 0) ? 1 : 0);
            tc_commit(&bars[slot]);
        }
        issued = kt + 1;
        const int nxt = kt + kStages - 1;
        if (nxt < nk) {
            bool ok = true;
            if (kt >= 1) ok = mbar_wait(&bars[(kt - 1) % kStages], ((kt - 1) / kStages) & 1, kSpinLimit);
            if (ok) load_stage(nxt, nxt % kStages);
            else {
                s_fail = 1;
                atomicExch(err, 1);
            }
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    // the last commit covers every MMA issued before it
    bool done = true;
    if (issued > 0) done = mbar_wait(&bars[(issued - 1) % kStages], ((issued - 1) / kStages) & 1, kSpinLimit);
    if (!done) {
        s_fail = 1;
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!s_fail && issued == nk) {
        const int m = m0 + warp * 32 + lane;
        const bool row_ok = m < M;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            EpilogueIn<UP> in;
            if (row_ok) conv_load16(g, (size_t)m, n0 + c0, in);
            tc_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            if (!row_ok) continue;
            conv_store16(g, (size_t)m, n0 + c0, v, in, s_bias + c0);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, kCols);
}

// Stride-1 3 x 3 convolution (or its data gradient, taps mirrored) with the input tile resident in shared memory.
// A CTA computes R output rows x 128 columns (x0 .. x0 + 127) x BN channels: it loads the (R + 2) x 130 input pixels
// around them once, in a layout where consecutive pixels are consecutive 16-byte rows of the core matrices
// (stride byte offset 128) and the 8-channel chunks are kLboA apart (leading byte offset), so the A operand of
// tap (ky, kx) for output row i is the same tile read from pixel (i + ky) * 130 + kx on: nine shifted descriptors
// instead of nine gathers. The weights stream per tap through a 3-slot cp.async ring. TMEM: R accumulators of BN
// columns. Needs W % 128 == 0, H % R == 0, C % 16 == 0. Bound by the latency of a CTA's phases and by shared-memory
// wavefronts: with 64 registers and 57 KB, four CTAs of 256 threads share an SM at 32 channels (one 1024^2 image, the 32 ->
// 32 and 32 -> 16 layers: 75 and 69 us with the weights' rows 16 bytes a lane and the biases read a column at a time, 69
// and 57 now).
constexpr int kTileW = 130, kTapStages = 3;
constexpr int kEpiThreads = 256;  // two groups of four warps share an epilogue (a warp reads TMEM lanes 32 (w % 4) ..)

__host__ __device__ constexpr int tile_lbo_px(int R) { return ((R + 2) * kTileW) | 1; }  // odd: spreads the banks

template <int BN, int R>
__global__ void __launch_bounds__(kEpiThreads) k_conv_tile_tc(const ConvGemm g, int *err) {
    extern __shared__ uint8_t dsm[];
    constexpr int kCols = (R * BN) < 32 ? 32 : (R * BN);
    constexpr int lbo_px = tile_lbo_px(R);
    __shared__ __align__(8) uint64_t bars[kTapStages];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ __align__(16) float s_bias[BN];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(dsm) + 127) & ~(uintptr_t)127);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int C = g.C, chunks = C >> 3;
    const int strips = g.Wo >> 7, yblocks = g.Ho / R;
    int blk = blockIdx.x;
    const int strip = blk % strips;
    blk /= strips;
    const int yb = blk % yblocks, b = blk / yblocks;
    const int x0 = strip << 7, y0 = yb * R, n0 = blockIdx.y * BN;
    const uint32_t lboA = (uint32_t)lbo_px * 16u;
    const uint32_t sA = smem_u32(base), sB = sA + (uint32_t)chunks * lboA;
    constexpr uint32_t kLboB = (BN + 2) * 16;
    const uint32_t bstage = (uint32_t)chunks * kLboB;  // one tap's weights
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    if (tid == 0) {
        for (int s = 0; s < kTapStages; ++s) mbar_init(&bars[s], 1);
        s_fail = 0;
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();
    pdl_wait();
    if (g.bias && tid < BN) s_bias[tid] = __ldcg(g.bias + n0 + tid);  // read after the loop's barriers
    const __nv_bfloat16 *src = static_cast<const __nv_bfloat16 *>(g.src);
    const __nv_bfloat16 *wt = static_cast<const __nv_bfloat16 *>(g.wt);
    // the input tile (zero outside the image): thread q -> pixel q / chunks of a row, chunk q % chunks (coalesced reads), in
    // every row of the tile
    // unit u of the epilogue: 16 columns of one row; the two groups of four warps take every other one
    const int m = (warp & 3) * 32 + lane;
    constexpr int kUnits = R * (BN / 16);
    auto unit_row = [&](int u) { return ((size_t)b * g.Ho + y0 + u / (BN / 16)) * g.Wo + x0 + m; };
    auto unit_col = [&](int u) { return n0 + u % (BN / 16) * 16; };
    EpilogueIn<false> in;
    if ((warp >> 2) < kUnits) conv_load16(g, unit_row(warp >> 2), unit_col(warp >> 2), in);
    const size_t img = (size_t)b * g.Hs * g.Ws;
    for (int q = tid; q < kTileW * chunks; q += kEpiThreads) {
        const int cc = q / chunks, j = q - cc * chunks;
        const int ix = x0 - 1 + cc;
        const bool okx = ix >= 0 && ix < g.Ws;
        const __nv_bfloat16 *col = src + (img + (size_t)(okx ? ix : 0)) * C + j * 8;
        const uint32_t dst = sA + (uint32_t)j * lboA + (uint32_t)cc * 16u;
#pragma unroll
        for (int rr = 0; rr < R + 2; ++rr) {
            const int iy = y0 - 1 + rr;
            const bool ok = okx && iy >= 0 && iy < g.Hs;
            cp_async16(dst + (uint32_t)(rr * kTileW) * 16u, ok ? col + (size_t)iy * g.Ws * C : src, ok ? 16 : 0);
        }
    }
    cp_async_commit();
    // one tap's weights: B[n][c] = wt[n0 + n][tap * C + c], chunk-major (chunk j at j * kLboB, row n at n * 16). Adjacent
    // threads take adjacent chunks of a row; the two rows of padding of a plane put four chunks of two rows, a quarter
    // warp's, in different banks
    const int wn = tid / chunks, wj = tid - wn * chunks;
    auto load_tap = [&](int t, int slot) {
        const uint32_t dst = sB + (uint32_t)slot * bstage;
        int n = wn, j = wj;
        for (int q = tid; q < BN * chunks; q += kEpiThreads) {
            cp_async16(dst + (uint32_t)j * kLboB + (uint32_t)n * 16u, wt + (size_t)(n0 + n) * g.ldw + t * C + j * 8, 16);
            if (BN * chunks > kEpiThreads) {
                n = (q + kEpiThreads) / chunks;
                j = q + kEpiThreads - n * chunks;
            }
        }
    };
    load_tap(0, 0);
    cp_async_commit();
    load_tap(1, 1);
    cp_async_commit();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16_f32(kBM, BN);
    int issued = 0;
#pragma unroll 1
    for (int t = 0; t < 9; ++t) {
        cp_async_wait<1>();  // the tile and this tap's weights have landed
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (s_fail) break;
        if (tid == 0) {
            const int ky = t / 3, kx = t - 3 * (t / 3);
            const int sy = g.dgrad ? 2 - ky : ky, sx = g.dgrad ? 2 - kx : kx;
            const uint32_t bb = sB + (uint32_t)(t % kTapStages) * bstage;
            for (int i = 0; i < R; ++i) {
                const uint32_t a0 = sA + (uint32_t)((i + sy) * kTileW + sx) * 16u;
                for (int s = 0; s < C / 16; ++s)
                    tc_mma(tmem + (uint32_t)(i * BN), smem_desc(a0 + (uint32_t)(2 * s) * lboA, lboA, 128),
                           smem_desc(bb + (uint32_t)(2 * s) * kLboB, kLboB, 128), idesc,
                           (t > 0 || s > 0) ? 1 : 0);
            }
            tc_commit(&bars[t % kTapStages]);
        }
        issued = t + 1;
        if (t + 2 < 9) {
            bool ok = true;
            if (t >= 1) ok = mbar_wait(&bars[(t - 1) % kTapStages], ((t - 1) / kTapStages) & 1, kSpinLimit);
            if (ok) load_tap(t + 2, (t + 2) % kTapStages);
            else {
                s_fail = 1;
                atomicExch(err, 1);
            }
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    bool done = true;
    if (issued > 0) done = mbar_wait(&bars[(issued - 1) % kTapStages], ((issued - 1) / kTapStages) & 1, kSpinLimit);
    if (!done) {
        s_fail = 1;
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!s_fail && issued == 9) {
#pragma unroll 1
        for (int u = warp >> 2; u < kUnits; u += 2) {
            float v[16];
            tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(u * 16), v);
            conv_store16(g, unit_row(u), unit_col(u), v, in, s_bias + u % (BN / 16) * 16);
            if (u + 2 < kUnits) conv_load16(g, unit_row(u + 2), unit_col(u + 2), in);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, kCols);
}

// TMA-fed convolution with warp-specialised roles. A CTA owns a patch of bh x bw = 128 output pixels of one image
// (one row of 128, or 128 / Wo whole rows) and BN output channels. The K loop runs over (tap, 64-channel block):
// per stage, one thread issues a strided 4-D TMA box of the activations (64 channels x the patch's input pixels,
// element stride = the convolution stride; padding and channels past C arrive as zeros) and a 2-D box of the
// weights, both 128-byte swizzled, onto a full mbarrier with the stage's byte count. A second thread waits for the
// stage, issues its four K = 16 MMAs and commits them to the stage's empty mbarrier, which releases the slot to the
// producer. After the last stage the MMA thread commits to `done`, and the four warps read the accumulator.
// Forward convolutions of stride 1 or 2 (3 x 3 or 1 x 1) and the data gradient of stride-1 layers (taps mirrored).
// The data gradient of a stride-2 3 x 3 layer (PARITY) is four convolutions of stride 1 on the output gradient's grid,
// one for each parity of the input pixel (blockIdx.z, the one with most taps first): of the nine taps an even
// coordinate meets only the middle one and an odd one the outer two, 1, 2, 2 and 4 taps instead of nine with three
// quarters zeros. The sums skip exact zeros only, in the order of the taps. Layers 1 to 3 of four 256^2 images: 131, 86
// and 68 us with the gather kernel, 27, 16 and 14 us now.
constexpr int kTmaMaxStages = 4;

// K-major operand in the 128-byte swizzle: 128-byte rows (64 bf16), 8-row atoms of 1 KB (stride byte offset),
// layout type 2 in bits 61-63; successive K = 16 slices start 32 B apart inside the atom.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

template <int BN, bool PARITY, bool UP>
__global__ void __launch_bounds__(kEpiThreads) k_conv_tma(const ConvGemm g, const __grid_constant__ CUtensorMap mapA,
                                                       const __grid_constant__ CUtensorMap mapB, int bw, int bh,
                                                       int cblocks, int stages, int *err) {
    extern __shared__ uint8_t dsm[];
    constexpr int kA = kBM * 128, kStage = kA + BN * 128;
    constexpr int kCols = BN < 32 ? 32 : BN;
    __shared__ __align__(8) uint64_t full[kTmaMaxStages], empty[kTmaMaxStages], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ __align__(16) float s_bias[BN];
    uint8_t *base = align1024(dsm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gw = PARITY ? g.Ws : g.Wo, gh = PARITY ? g.Hs : g.Ho;  // the grid that is cut into patches
    const int pxn = gw / bw, pyn = gh / bh;
    int blk = blockIdx.x;
    const int pxi = blk % pxn;
    blk /= pxn;
    const int pyi = blk % pyn, b = blk / pyn;
    const int ox0 = pxi * bw, oy0 = pyi * bh, n0 = blockIdx.y * BN;
    const int odd_y = PARITY ? 1 - (int)(blockIdx.z >> 1) : 0, odd_x = PARITY ? 1 - (int)(blockIdx.z & 1) : 0;
    const int nk = (PARITY ? (1 + odd_y) * (1 + odd_x) : g.ks * g.ks) * cblocks;
    const int m = (warp & 3) * 32 + lane;
    int oy = oy0 + m / bw, ox = ox0 + m % bw;
    if constexpr (PARITY) {
        oy = 2 * oy + odd_y;
        ox = 2 * ox + odd_x;
    }
    const size_t row = ((size_t)b * g.Ho + oy) * g.Wo + ox;
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&done, 1);
        s_fail = 0;
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();
    pdl_wait();
    if (g.bias && tid < BN) s_bias[tid] = __ldcg(g.bias + n0 + tid);  // read after the loop's barriers
    EpilogueIn<UP> in;
    // the upsampled output of a pass of up to 32 columns: chunk k of this thread (8 channels of one high-resolution pixel,
    // adjacent threads in adjacent memory), its low-resolution pixel and its offset in the output and in the skip
    constexpr int kUpCols = BN < 32 ? BN : 32, kUpChunks = kUpCols / 8, kUpPer = 2 * kUpChunks, kUpPitch = kUpCols + 4;
    auto up_pixel = [&](int k) { return (tid + kEpiThreads * k) / kUpChunks; };
    const int up_shift = 32 - __clz(bw);  // a patch's output row has 2 bw pixels, a power of two
    auto up_lr = [&](int k) {
        const int hp = up_pixel(k), hy = hp >> up_shift, hx = hp - (hy << up_shift);
        return (hy >> 1) * bw + (hx >> 1);
    };
    auto up_offset = [&](int k, int c0) {
        const int hp = up_pixel(k), hy = hp >> up_shift, hx = hp - (hy << up_shift);
        return (((size_t)b * 2 * g.Ho + 2 * oy0 + hy) * (size_t)(2 * g.Wo) + 2 * ox0 + hx) * g.N + n0 + c0 +
               tid % kUpChunks * 8;
    };
    auto up_load = [&](int c0) {
#pragma unroll
        for (int k = 0; k < (UP ? kUpPer : 0); ++k)
            in.u[k] = *reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(g.upskip) + up_offset(k, c0));
    };
    if constexpr (UP) up_load(0);
    else if ((warp >> 2) * 16 < BN) conv_load16(g, row, n0 + (warp >> 2) * 16, in);
    const uint32_t tmem = tmem_slot;
    if (warp == 0 && lane == 0) {
        // producer
        for (int kt = 0; kt < nk; ++kt) {
            const int use = kt / stages, slot = kt - use * stages;
            if (kt >= stages && !mbar_wait(&empty[slot], (use - 1) & 1, kSpinLimit)) {
                s_fail = 1;
                atomicExch(err, 1);
                break;
            }
            int tap = kt / cblocks;
            const int cb = kt - tap * cblocks;
            int sx = ox0 * g.stride, sy = oy0 * g.stride;
            if constexpr (PARITY) {
                // tap 0 or 2 along an odd coordinate (source one on, or in place), tap 1 along an even one
                const int ty = tap >> odd_x, tx = tap & odd_x;
                sx = ox0 + (odd_x & (tx ^ 1));
                sy = oy0 + (odd_y & (ty ^ 1));
                tap = 3 * (odd_y ? 2 * ty : 1) + (odd_x ? 2 * tx : 1);
            } else if (g.ks == 3) {
                const int ky = tap / 3, kx = tap - 3 * (tap / 3);
                if (!g.dgrad) {
                    sx += kx - 1;
                    sy += ky - 1;
                } else {
                    sx = ox0 + 1 - kx;
                    sy = oy0 + 1 - ky;
                }
            }
            uint8_t *sa = base + slot * kStage;
            mbar_arrive_expect_tx(&full[slot], (unsigned)kStage);
            tma_load_4d(sa, &mapA, cb * 64, sx, sy, b, &full[slot]);
            tma_load_2d(sa + kA, &mapB, tap * g.C + cb * 64, n0, &full[slot]);
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        const uint32_t idesc = idesc_bf16_f32(kBM, BN);
        for (int kt = 0; kt < nk; ++kt) {
            const int use = kt / stages, slot = kt - use * stages;
            if (!mbar_wait(&full[slot], use & 1, kSpinLimit)) {
                s_fail = 1;
                atomicExch(err, 1);
                break;
            }
            tc_fence_after();
            const uint32_t a = smem_u32(base + slot * kStage), bb = a + kA;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                tc_mma(tmem, smem_desc_sw128(a + 32 * k), smem_desc_sw128(bb + 32 * k), idesc, (kt > 0 || k > 0) ? 1 : 0);
            tc_commit(&empty[slot]);
        }
        tc_commit(&done);  // arrives once every MMA issued above has completed
    }
    __syncthreads();
    if (!mbar_wait(&done, 0, kSpinLimit)) {
        s_fail = 1;
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (UP && !s_fail) {
        // A thread's own pixel would write 32 of every 128 bytes a store touches, and read the skip likewise: the values go
        // through shared memory (the stages' memory, whose reads are over) and leave in the order of the output (the three
        // decoder layers of a 1024^2 image: 19, 30 and 45 -> 13, 21 and 36 us)
        float *vs = reinterpret_cast<float *>(base);
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += kUpCols) {
            if (c0) up_load(c0);
            const int cw = (warp >> 2) * 16;
            if (cw < kUpCols) {
                float v[16];
                tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(c0 + cw), v);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 bv = g.bias ? reinterpret_cast<const float4 *>(s_bias + c0 + cw)[k]
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
                    reinterpret_cast<float4 *>(vs + m * kUpPitch + cw)[k] =
                        make_float4(v[4 * k] + bv.x, v[4 * k + 1] + bv.y, v[4 * k + 2] + bv.z, v[4 * k + 3] + bv.w);
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < (UP ? kUpPer : 0); ++k) {
                const float4 *pv = reinterpret_cast<const float4 *>(vs + up_lr(k) * kUpPitch + tid % kUpChunks * 8);
                const float4 v0 = pv[0], v1 = pv[1];
                float f[8];
                unpack8(in.u[k], f);
                const float r[8] = {fmaxf(v0.x + f[0], 0.f), fmaxf(v0.y + f[1], 0.f), fmaxf(v0.z + f[2], 0.f),
                                    fmaxf(v0.w + f[3], 0.f), fmaxf(v1.x + f[4], 0.f), fmaxf(v1.y + f[5], 0.f),
                                    fmaxf(v1.z + f[6], 0.f), fmaxf(v1.w + f[7], 0.f)};
                *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(g.outb) + up_offset(k, c0)) = pack8(r);
            }
            __syncthreads();  // the next pass overwrites vs
        }
    }
    if constexpr (!UP) {
#pragma unroll 1
        for (int c0 = (warp >> 2) * 16; !s_fail && c0 < BN; c0 += 32) {
            float v[16];
            tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
            conv_store16(g, row, n0 + c0, v, in, s_bias + c0);
            if (c0 + 32 < BN) conv_load16(g, row, n0 + c0 + 32, in);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, kCols);
}

// Weight gradient: GEMM rows are the (tap, ci) rows of dW^T (padded to 128), N = the stored output channels, the
// reduction runs over the output pixels of this split. Both operands are pixel-major in global memory, that is
// MN-major: eight channels of one pixel are one 16-byte row of a core matrix (8 pixels x 8 channels), so a gather is
// one 16-byte cp.async and nothing is transposed. Core matrices adjacent in channels lie kWgSbo apart (stride byte
// offset; 128 B and 32 of padding, which spreads a quarter warp's four chunks of two pixels over all banks), 8-pixel
// blocks one row of those apart (leading byte offset). Stages of 64 pixels run through a ring of cp.async groups as in
// k_conv_tc; its depth leaves two CTAs an SM up to 128 columns. Bound by the gather's L1 and L2 traffic (every input
// pixel is read once a tap). Four 256^2 images, twelve layers: 691 us with 2-byte transposing stores and one stage in
// flight, 333 us now. Result: FP32 partial[split][row][co].
constexpr int kWgSbo = 160;
__host__ __device__ constexpr int wg_stage_bytes(int BN) { return 8 * kWgSbo * (kBM / 8 + BN / 8); }
__host__ __device__ constexpr int wg_stages(int BN) { return BN <= 32 ? 4 : BN == 64 ? 3 : BN == 128 ? 2 : 3; }

template <int BN>
__global__ void __launch_bounds__(kEpiThreads) k_wgrad_tc(const WgradGemm g, int *err) {
    extern __shared__ uint8_t dsm[];
    constexpr int kWgStages = wg_stages(BN), kStage = wg_stage_bytes(BN);
    constexpr int kLboA = kBM / 8 * kWgSbo, kLboB = BN / 8 * kWgSbo, kA = 8 * kLboA;
    constexpr int kCols = BN < 32 ? 32 : BN;
    constexpr int kBC = BN < 32 ? 2 : 4;  // dY chunks that adjacent threads take
    __shared__ __align__(8) uint64_t bars[kWgStages];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    uint8_t *base = align1024(dsm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int HWo = g.Ho * g.Wo, P = g.batch * HWo;
    const int m0 = blockIdx.x * kBM;
    const int p0 = blockIdx.y * g.chunk, p1 = min(P, p0 + g.chunk);
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    if (tid == 0) {
        for (int s = 0; s < kWgStages; ++s) mbar_init(&bars[s], 1);
        s_fail = 0;
        fence_proxy_async_smem();
    }
    // this thread's four X chunks (8 channels of one tap each), channel blocks 4 q + (tid & 3) of the tile, all of pixel
    // tid / 4 of a stage: the tap's step, and the chunk's offset from the pixel's first channel
    int ady[4], adx[4], aoff[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r0 = m0 + (4 * q + (tid & 3)) * 8;
        const int tap = r0 / g.Cin;
        ady[q] = g.ks == 3 ? tap / 3 - 1 : 0;
        adx[q] = g.ks == 3 ? tap - (tap / 3) * 3 - 1 : 0;
        aoff[q] = (ady[q] * g.Wx + adx[q]) * g.Cin + r0 - tap * g.Cin;
        if (r0 >= g.Kf) ady[q] = -(1 << 28);  // past the last row: outside every image
    }
    const __nv_bfloat16 *X = static_cast<const __nv_bfloat16 *>(g.x);
    const __nv_bfloat16 *DY = static_cast<const __nv_bfloat16 *>(g.dy);
    const uint32_t sbase = smem_u32(base);
    const int pk = tid >> 2, yk = tid / kBC;  // this thread's pixel of a stage for X and for dY
    int p = p0 + pk, b = p / HWo, oy = (p - b * HWo) / g.Wo, ox = p - b * HWo - oy * g.Wo;
    // stages are loaded in order: the pixel moves on by one stage a call, without a division where a row holds a stage
    auto load_stage = [&](int kt, int slot) {
        const uint32_t sa = sbase + slot * kStage, sb = sa + kA;
        const bool pv = p < p1;
        const int y0 = oy * g.stride, x0 = ox * g.stride;
        const __nv_bfloat16 *px = X + (size_t)((b * g.Hx + y0) * g.Wx + x0) * g.Cin;
        const uint32_t dst = sa + (uint32_t)((pk >> 3) * kLboA + (tid & 3) * kWgSbo + ((pk & 7) << 4));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool ok = pv && (unsigned)(y0 + ady[q]) < (unsigned)g.Hx && (unsigned)(x0 + adx[q]) < (unsigned)g.Wx;
            cp_async16(dst + q * 4 * kWgSbo, ok ? px + aoff[q] : X, ok ? 16 : 0);
        }
        if (yk < kBK) {
            const int py = p0 + kt * kBK + yk;
            const bool yv = py < p1;
            const __nv_bfloat16 *src = yv ? DY + (size_t)py * BN + tid % kBC * 8 : DY;
            const uint32_t ydst = sb + (uint32_t)((yk >> 3) * kLboB + tid % kBC * kWgSbo + ((yk & 7) << 4));
#pragma unroll
            for (int c = 0; c < BN / 8; c += kBC) cp_async16(ydst + c * kWgSbo, yv ? src + c * 8 : DY, yv ? 16 : 0);
        }
        p += kBK;
        if (g.Wo >= kBK) {
            ox += kBK;
            if (ox >= g.Wo) {
                ox -= g.Wo;
                if (++oy == g.Ho) {
                    oy = 0;
                    ++b;
                }
            }
        } else {
            b = p / HWo;
            oy = (p - b * HWo) / g.Wo;
            ox = p - b * HWo - oy * g.Wo;
        }
    };
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16_f32(kBM, BN) | kMnMajor;
    const int nk = (p1 - p0 + kBK - 1) / kBK;
#pragma unroll 1
    for (int s = 0; s < kWgStages - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_async_commit();
    }
    int issued = 0;
#pragma unroll 1
    for (int kt = 0; kt < nk; ++kt) {
        const int slot = kt % kWgStages;
        cp_async_wait<kWgStages - 2>();  // stage kt has landed
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (s_fail) break;
        if (tid == 0) {
            const uint32_t a = sbase + slot * kStage, bb = a + kA;
#pragma unroll
            for (int s = 0; s < kBK / 16; ++s)
                tc_mma(tmem, smem_desc(a + s * 2 * kLboA, kLboA, kWgSbo), smem_desc(bb + s * 2 * kLboB, kLboB, kWgSbo),
                       idesc, (kt > 0 || s > 0) ? 1 : 0);
            tc_commit(&bars[slot]);
        }
        issued = kt + 1;
        const int nxt = kt + kWgStages - 1;
        if (nxt < nk) {
            // the slot of stage kt - 1 is free once its MMAs have completed
            bool ok = true;
            if (kt >= 1) ok = mbar_wait(&bars[(kt - 1) % kWgStages], ((kt - 1) / kWgStages) & 1, kSpinLimit);
            if (ok) load_stage(nxt, nxt % kWgStages);
            else {
                s_fail = 1;
                atomicExch(err, 1);
            }
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    bool done = true;
    if (issued > 0) done = mbar_wait(&bars[(issued - 1) % kWgStages], ((issued - 1) / kWgStages) & 1, kSpinLimit);
    if (!done) {
        s_fail = 1;
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!s_fail) {
        const int r = (warp & 3) * 32 + lane;
        float *out = g.partial + ((size_t)blockIdx.y * g.Mpad + m0 + r) * BN;
#pragma unroll 1
        for (int c0 = (warp >> 2) * 16; c0 < BN; c0 += 32) {
            float v[16];
            if (issued > 0) tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
            else {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.f;
            }
            float4 *fp = reinterpret_cast<float4 *>(out + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) fp[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    pdl_wait();  // the column sums this kernel ran beside
    if (warp == 0) tmem_free(tmem, kCols);
}

// Column sums of a BF16 [P][C] tensor (bias gradients): per-block partials[block][C], fixed order. A thread keeps eight
// channels of every (256 / (C / 8))-th pixel, so a warp's loads are contiguous 512 bytes; four are in flight a thread.
constexpr int kColsumUnroll = 4;
__global__ void __launch_bounds__(256) k_colsum(int P, int C, const __nv_bfloat16 *__restrict__ dy,
                                                float *__restrict__ partial) {
    pdl_trigger();
    __shared__ float sh[256 * 9];  // nine floats a thread: eight and one of padding
    const int chunks = C >> 3, lanes = 256 / chunks, j = threadIdx.x % chunks, l = threadIdx.x / chunks;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int step = gridDim.x * lanes;
    const uint4 *src = reinterpret_cast<const uint4 *>(dy) + j;
    for (long long p = (long long)blockIdx.x * lanes + l; p < P; p += (long long)kColsumUnroll * step) {
        uint4 u[kColsumUnroll];
#pragma unroll
        for (int k = 0; k < kColsumUnroll; ++k) {
            const long long q = p + (long long)k * step;
            u[k] = q < P ? __ldg(src + (size_t)q * chunks) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int k = 0; k < kColsumUnroll; ++k) {
            float f[8];
            unpack8(u[k], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] += f[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sh[threadIdx.x * 9 + i] = s[i];
    __syncthreads();
    if (threadIdx.x < C) {
        const int cj = threadIdx.x >> 3, ci = threadIdx.x & 7;
        float t = 0.f;
        for (int k = 0; k < lanes; ++k) t += sh[(k * chunks + cj) * 9 + ci];
        partial[(size_t)blockIdx.x * C + threadIdx.x] = t;
    }
}

// Sums of `count` partials of n elements each (partial[s * stride + i], i < n), element i = k * Cst + co going to
// out[co * Kf + k] where co < Cout: the weight gradient's splits (n = Kf * Cst) and, in the last blocks, the bias
// gradient's block partials (Kf = 1). 256 threads take 4 * 256 / lanes elements, `lanes` of them splitting the count:
// adjacent threads read adjacent 16 bytes, and a small layer with many splits (288 rows of 16 channels, 102 splits) still
// has all its loads in flight. One thread per element walking every split, its reads Cst floats apart, took 298 us for
// the twelve layers of four 256^2 images (95 now) and the bias sums with 2-byte loads 374 (62 now).
struct ReducePart {
    const float *partial;
    float *out;
    size_t stride;
    int count, Cst, Kf, Cout, lanes, blocks;
};

__global__ void __launch_bounds__(256) k_wgrad_reduce(const ReducePart w, const ReducePart bias) {
    __shared__ float4 sh[256];
    const bool isb = (int)blockIdx.x >= w.blocks;
    const ReducePart &r = isb ? bias : w;
    const int width = 256 / r.lanes, x = threadIdx.x % width, l = threadIdx.x / width;
    const int i = (((int)blockIdx.x - (isb ? w.blocks : 0)) * width + x) * 4, n = r.Kf * r.Cst;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
        const float *p = r.partial + i;
#pragma unroll 4
        for (int k = l; k < r.count; k += r.lanes) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p + (size_t)k * r.stride));
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
        }
    }
    sh[threadIdx.x] = s;
    for (int h = r.lanes >> 1; h > 0; h >>= 1) {
        __syncthreads();
        if (l < h) {
            const float4 v = sh[threadIdx.x + h * width];
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
            sh[threadIdx.x] = s;
        }
    }
    if (l == 0 && i < n) {
        const float f[4] = {s.x, s.y, s.z, s.w};
        const int k = i / r.Cst, co = i - k * r.Cst;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (co + c < r.Cout) r.out[(size_t)(co + c) * r.Kf + k] = f[c];
    }
}

// dt = sum of the 2 x 2 block of ds (the adjoint of nearest upsampling).
__global__ void k_down_sum(int batch, int Hl, int Wl, int C, const __nv_bfloat16 *__restrict__ ds,
                           __nv_bfloat16 *__restrict__ dt) {
    const int C8 = C >> 3, W = 2 * Wl;
    const size_t total = (size_t)batch * Hl * Wl * C8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c8 = (int)(i % C8);
        const size_t pix = i / C8;
        const int x = (int)(pix % Wl);
        const size_t r = pix / Wl;
        const int y = (int)(r % Hl), b = (int)(r / Hl);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, v[8];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const size_t hp = ((size_t)b * 2 * Hl + 2 * y + (d >> 1)) * W + 2 * x + (d & 1);
            unpack8(*reinterpret_cast<const uint4 *>(ds + hp * C + c8 * 8), v);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += v[j];
        }
        *reinterpret_cast<uint4 *>(dt + pix * C + c8 * 8) = pack8(acc);
    }
}

// Output head: pred = u0 + y[:, 0:3] (y: four floats a pixel; pred planar per image), and with a target the loss 1/(3 P) sum (pred - target)^2,
// its gradient dy = 2 (pred - target) / (3 P) as BF16 [P][Cy] (zero in the padding channels), per-block loss
// partials in FP64.
template <bool LOSS>
__global__ void __launch_bounds__(256) k_output_head(int batch, int HW, int Cy, const float4 *__restrict__ y,
                                                     const float *__restrict__ u0, const float *__restrict__ target,
                                                     float *__restrict__ pred, __nv_bfloat16 *__restrict__ dy,
                                                     double *__restrict__ loss_partial) {
    pdl_wait();
    __shared__ double sh[8];
    const size_t P = (size_t)batch * HW;
    const float scale = 2.0f / (3.0f * (float)P);
    double acc = 0.0;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < P; p += (size_t)gridDim.x * blockDim.x) {
        const size_t b = p / HW, o = p - b * HW;
        const float4 yp = __ldcg(y + p);
        const float yc[3] = {yp.x, yp.y, yp.z};
        float d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t q = (b * 3 + c) * HW + o;
            const float v = u0[q] + yc[c];
            if (pred) pred[q] = v;
            if constexpr (LOSS) {
                d[c] = v - target[q];
                acc += (double)d[c] * d[c];
            }
        }
        if constexpr (LOSS) {
            const float f[8] = {d[0] * scale, d[1] * scale, d[2] * scale, 0.f, 0.f, 0.f, 0.f, 0.f};
            uint4 *row = reinterpret_cast<uint4 *>(dy + p * Cy);
            row[0] = pack8(f);
            for (int c = 1; c < Cy / 8; ++c) row[c] = make_uint4(0, 0, 0, 0);
        }
    }
    if constexpr (LOSS) acc = block_sum<256>(acc, sh);
    if (LOSS && threadIdx.x == 0) loss_partial[blockIdx.x] = acc;
}

// Adam on the flat FP32 parameters (bias-corrected step sizes computed on the host).
__global__ void k_adam(size_t n, float *__restrict__ w, const float *__restrict__ grad, float *__restrict__ m,
                       float *__restrict__ v, float lr_t, float b1, float b2, float eps_t) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = grad[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr_t * mi / (sqrtf(vi) + eps_t);
    }
}

// BF16 GEMM copies of one layer's FP32 weights w[co][tap * Cin + ci]: Wb[co][k] (Cst x Kpad, zero padded) for the
// forward pass and Wt[ci][tap * Cst + co] (Cin x Kdpad) for the data gradient.
__global__ void k_pack_weights(int Cout, int Cst, int Cin, int taps, int Kpad, int Kdpad, const float *__restrict__ w,
                               __nv_bfloat16 *__restrict__ Wb, __nv_bfloat16 *__restrict__ Wt) {
    const int Kf = taps * Cin;
    const size_t nb = (size_t)Cst * Kpad, nt = (size_t)Cin * Kdpad;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nb + nt; i += (size_t)gridDim.x * blockDim.x) {
        if (i < nb) {
            const int co = (int)(i / Kpad), k = (int)(i % Kpad);
            Wb[i] = __float2bfloat16_rn((co < Cout && k < Kf) ? w[(size_t)co * Kf + k] : 0.f);
        } else {
            const size_t j = i - nb;
            const int ci = (int)(j / Kdpad), kd = (int)(j % Kdpad);
            const int tap = kd / Cst, co = kd - tap * Cst;
            float val = 0.f;
            if (tap < taps && co < Cout) val = w[(size_t)co * Kf + tap * Cin + ci];
            Wt[j] = __float2bfloat16_rn(val);
        }
    }
}

// ------------------------------------------------------------------ launchers
// A forward layer starts setting up (tensor memory, barriers, indices) while the layer before it ends: twelve layers of one
// 512^2 image 239 -> 222 us. The data gradients don't: their early blocks would hold shared memory that the weight
// gradients beside them use (a training step with and without: four images of 256^2 735 and 706 us, sixteen 1877 and 1850,
// one of 512^2 731 and 705; only the smallest would gain, one of 64^2 440 and 472).
template <typename... Params, typename... Args>
static cudaError_t launch_layer(const ConvGemm &g, void (*kernel)(Params...), dim3 grid, int threads, int smem,
                                cudaStream_t st, Args... args) {
    if (!g.dgrad) return launch_pdl(kernel, grid, dim3(threads), (size_t)smem, st, args...);
    kernel<<<grid, threads, smem, st>>>(args...);
    return cudaGetLastError();
}

template <int BN, bool UP>
static cudaError_t conv_launch(const ConvGemm &g, int *err, cudaStream_t st) {
    constexpr int smem = kStages * (kBM * kBK * 2 + BN * kBK * 2) + 1024;
    static bool attr = false;
    if (!attr) {
        const cudaError_t e = cudaFuncSetAttribute(k_conv_tc<BN, UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int M = g.batch * g.Ho * g.Wo;
    return launch_layer(g, k_conv_tc<BN, UP>, dim3((M + kBM - 1) / kBM, g.N / BN), kThreads, smem, st, g, err);
}

template <bool UP>
static cudaError_t launch_gather(const ConvGemm &g, int bn, int *err, cudaStream_t st) {
    switch (bn) {
        case 16: return conv_launch<16, UP>(g, err, st);
        case 32: return conv_launch<32, UP>(g, err, st);
        case 64: return conv_launch<64, UP>(g, err, st);
        case 128: return conv_launch<128, UP>(g, err, st);
        case 256: return conv_launch<256, UP>(g, err, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int BN, int R>
static cudaError_t tile_launch(const ConvGemm &g, int smem, int *err, cudaStream_t st) {
    static int attr = 0;
    if (smem > attr) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_conv_tile_tc<BN, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = smem;
    }
    const dim3 grid(g.batch * (g.Ho / R) * (g.Wo >> 7), g.N / BN);
    return launch_layer(g, k_conv_tile_tc<BN, R>, grid, kEpiThreads, smem, st, g, err);
}

// The resident-tile kernel's shape for a stride-1 3 x 3 layer (forward, or data gradient of a stride-1 layer), or
// false when it does not apply (rows not a multiple of 128, channels not a multiple of 16, no shape that fits).
static bool tile_shape(const ConvGemm &g, int &R, int &BN, int &smem) {
    if (g.ks != 3 || g.stride != 1 || g.Wo % 128 || g.C % 16 || g.Hs != g.Ho || g.Ws != g.Wo) return false;
    if (g.ldw < 9 * g.C) return false;
    int best = -1;
    for (int r : {4, 2, 1}) {
        if (g.Ho % r) continue;
        for (int bn = g.N; bn >= 16 && bn >= g.N / 2; bn >>= 1) {
            if (r * bn > 256 || bn > 128) continue;
            const int sm = (g.C / 8) * tile_lbo_px(r) * 16 + kTapStages * (g.C / 8) * (bn + 2) * 16 + 128;
            if (sm > 200 * 1024) continue;
            const int ctas = g.batch * (g.Ho / r) * (g.Wo / 128) * (g.N / bn);
            const int score = std::min(ctas, 2 * kSms);
            if (score > best) {
                best = score;
                R = r;
                BN = bn;
                smem = sm;
            }
        }
    }
    return best > 0;
}

static cudaError_t launch_tile(const ConvGemm &g, int R, int BN, int smem, int *err, cudaStream_t st) {
#define LFRV_TILE_CASE(bn, r) \
    if (BN == bn && R == r) return tile_launch<bn, r>(g, smem, err, st);
    LFRV_TILE_CASE(16, 1) LFRV_TILE_CASE(16, 2) LFRV_TILE_CASE(16, 4)
    LFRV_TILE_CASE(32, 1) LFRV_TILE_CASE(32, 2) LFRV_TILE_CASE(32, 4)
    LFRV_TILE_CASE(64, 1) LFRV_TILE_CASE(64, 2) LFRV_TILE_CASE(64, 4)
    LFRV_TILE_CASE(128, 1) LFRV_TILE_CASE(128, 2)
#undef LFRV_TILE_CASE
    return cudaErrorInvalidValue;
}

// The data gradient of a stride-2 layer that k_conv_tma takes by parity: an even image, so that every parity has the
// output gradient's grid, and whole 64-channel blocks, so that a tap's box holds no other tap's weights. Everything
// else of stride 2 (one row more or less, 1 x 1, 16 or 32 channels) is the gather kernel's.
static bool tma_parity(const ConvGemm &g) {
    return g.dgrad && g.stride == 2 && g.ks == 3 && g.C % 64 == 0 && g.Ho == 2 * g.Hs && g.Wo == 2 * g.Ws;
}

// Patch of the TMA kernel (bw x bh = 128 pixels of the grid it runs over), or false when the layer does not tile that
// way.
static bool tma_shape(const ConvGemm &g, int &bw, int &bh) {
    if (g.ks != 1 && g.ks != 3) return false;
    const bool parity = tma_parity(g);
    if (g.dgrad && g.stride != 1 && !parity) return false;
    if (g.C % 8 || g.C < 8) return false;
    const int gw = parity ? g.Ws : g.Wo, gh = parity ? g.Hs : g.Ho;
    if (gw >= 128) {
        if (gw % 128) return false;
        bw = 128;
        bh = 1;
    } else {
        if (128 % gw) return false;
        bw = gw;
        bh = 128 / gw;
        if (gh % bh) return false;
    }
    const int s = g.dgrad ? 1 : g.stride;
    return bw * s <= 256 && bh * s <= 256;
}

// Activation map: dims (C, W, H, batch) of NHWC BF16, box (64, bw s, bh s, 1) with element strides (1, s, s, 1);
// weight map: dims (ldw, N), box (64, BN). Both with the 128-byte swizzle and zero fill outside the tensor.
static bool encode_conv_maps(const ConvGemm &g, int bw, int bh, int BN, CUtensorMap *mA, CUtensorMap *mB) {
    const auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
    if (!encode) return false;
    const int s = g.dgrad ? 1 : g.stride;
    const cuuint64_t adims[4] = {(cuuint64_t)g.C, (cuuint64_t)g.Ws, (cuuint64_t)g.Hs, (cuuint64_t)g.batch};
    const cuuint64_t astr[3] = {(cuuint64_t)g.C * 2, (cuuint64_t)g.Ws * g.C * 2, (cuuint64_t)g.Hs * g.Ws * g.C * 2};
    const cuuint32_t abox[4] = {64, (cuuint32_t)(bw * s), (cuuint32_t)(bh * s), 1};
    const cuuint32_t aes[4] = {1, (cuuint32_t)s, (cuuint32_t)s, 1};
    if (encode(mA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(g.src), adims, astr, abox, aes,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    const cuuint64_t bdims[2] = {(cuuint64_t)g.ldw, (cuuint64_t)g.N};
    const cuuint64_t bstr[1] = {(cuuint64_t)g.ldw * 2};
    const cuuint32_t bbox[2] = {64, (cuuint32_t)BN};
    const cuuint32_t bes[2] = {1, 1};
    return encode(mB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(g.wt), bdims, bstr, bbox, bes,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool PARITY, bool UP>
static cudaError_t tma_launch(const ConvGemm &g, int bw, int bh, const CUtensorMap &mA, const CUtensorMap &mB, int *err,
                              cudaStream_t st) {
    constexpr int stage = kBM * 128 + BN * 128, limit = 200 * 1024;
    static bool attr = false;
    if (!attr) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_conv_tma<BN, PARITY, UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit + 1024);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int cblocks = (g.C + 63) / 64, parities = PARITY ? 4 : 1, nk = (PARITY ? 4 : g.ks * g.ks) * cblocks;
    const dim3 grid(g.batch * (g.Ho * g.Wo / parities) / (bh * bw), g.N / BN, parities);
    // four stages (what fits of them) when the grid leaves each SM one or two CTAs; two when there are more, which then
    // hide each other's latency: with four the layers of four 256^2 images took 260 us forward, with two 243, and rings
    // of six or eight gave the one-CTA layers nothing
    const int per_sm = ((int)(grid.x * grid.y * grid.z) + kSms - 1) / kSms;
    const int stages = std::min({nk, kTmaMaxStages, per_sm > 2 ? 2 : limit / per_sm / stage});
    return launch_layer(g, k_conv_tma<BN, PARITY, UP>, grid, kEpiThreads, stages * stage + 1024, st, g, mA, mB, bw, bh,
                        cblocks, stages, err);
}

template <bool PARITY, bool UP>
static cudaError_t launch_tma(const ConvGemm &g, int bn, int bw, int bh, const CUtensorMap &mA, const CUtensorMap &mB,
                              int *err, cudaStream_t st) {
    switch (bn) {
        case 16: return tma_launch<16, PARITY, UP>(g, bw, bh, mA, mB, err, st);
        case 32: return tma_launch<32, PARITY, UP>(g, bw, bh, mA, mB, err, st);
        case 64: return tma_launch<64, PARITY, UP>(g, bw, bh, mA, mB, err, st);
        case 128: return tma_launch<128, PARITY, UP>(g, bw, bh, mA, mB, err, st);
        default: return tma_launch<256, PARITY, UP>(g, bw, bh, mA, mB, err, st);
    }
}

// Which convolution kernel a layer uses: the TMA kernel where its patch tiling applies, else the resident-tile
// kernel (stride-1 3 x 3 on 128-pixel rows), else the cp.async gather. The preference (0 all, 1 no TMA kernel,
// 2 the gather only) restricts the choice; a kernel that does not apply falls through to the next.
static std::atomic<int> g_conv_pref{0};
void set_conv_kernel_pref(int pref) { g_conv_pref.store(pref); }
static int conv_kernel_pref() { return g_conv_pref.load(); }

cudaError_t launch_conv_tc(const ConvGemm &g, int *err, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, g.dgrad ? "conv_dgrad_tc" : "conv_fwd_tc", st);
    if (g.N != 16 && g.N != 32 && g.N != 64 && g.N != 128 && g.N != 256) return cudaErrorInvalidValue;
    const int pref = conv_kernel_pref();
    // the resident-tile kernel reads each input pixel ~1.5 times, the TMA kernel once per tap in 64-channel boxes:
    // with fewer than 64 channels the tile kernel moves fewer bytes
    {
        int R = 0, BN = 0, smem = 0;
        if (pref <= 1 && g.C < 64 && tile_shape(g, R, BN, smem)) {
            const cudaError_t e = launch_tile(g, R, BN, smem, err, st);
            lc.add(1);
            return e;
        }
    }
    {
        int bw = 0, bh = 0;
        CUtensorMap mA, mB;
        int bn = g.N;
        const bool tma = pref == 0 && tma_shape(g, bw, bh);
        if (tma) {
            const int mtiles = g.batch * g.Ho * g.Wo / kBM;
            while (bn > 32 && mtiles * (g.N / bn) < 120) bn >>= 1;
        }
        // a map the driver does not accept sends the layer to the other kernels
        if (tma && encode_conv_maps(g, bw, bh, bn, &mA, &mB)) {
            const cudaError_t e = tma_parity(g) ? launch_tma<true, false>(g, bn, bw, bh, mA, mB, err, st)
                                  : g.upskip    ? launch_tma<false, true>(g, bn, bw, bh, mA, mB, err, st)
                                                : launch_tma<false, false>(g, bn, bw, bh, mA, mB, err, st);
            lc.add(1);
            return e;
        }
    }
    if (pref <= 1) {
        int R = 0, BN = 0, smem = 0;
        if (tile_shape(g, R, BN, smem)) {
            const cudaError_t e = launch_tile(g, R, BN, smem, err, st);
            lc.add(1);
            return e;
        }
    }
    if (g.C % 8 || g.ldw % kBK || g.ldw < ((g.K + kBK - 1) / kBK) * kBK || g.K <= 0) return cudaErrorInvalidValue;
    if (g.stride != 1 && g.stride != 2) return cudaErrorInvalidValue;
    if (g.N != 16 && g.N != 32 && g.N != 64 && g.N != 128 && g.N != 256) return cudaErrorInvalidValue;
    // output columns per CTA: all N, halved while the grid would not fill the SMs (the low-resolution layers)
    const int mtiles = (g.batch * g.Ho * g.Wo + kBM - 1) / kBM;
    int bn = g.N;
    while (bn > 32 && mtiles * (g.N / bn) < 120) bn >>= 1;
    const cudaError_t e = g.upskip ? launch_gather<true>(g, bn, err, st) : launch_gather<false>(g, bn, err, st);
    lc.add(1);
    return e;
}

template <int BN>
static cudaError_t wgrad_launch(const WgradGemm &g, int splits, bool beside, int *err, cudaStream_t st) {
    constexpr int smem = wg_stages(BN) * wg_stage_bytes(BN) + 1024;
    static bool attr = false;
    if (!attr) {
        const cudaError_t e = cudaFuncSetAttribute(k_wgrad_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const dim3 grid(g.Mpad / kBM, splits);
    // beside: the launch before it is this layer's column sums, which started after all that this kernel reads was written
    if (beside) return launch_pdl(k_wgrad_tc<BN>, grid, dim3(kEpiThreads), smem, st, g, err);
    k_wgrad_tc<BN><<<grid, kEpiThreads, smem, st>>>(g, err);
    return cudaGetLastError();
}

cudaError_t launch_wgrad_tc(const WgradGemm &g, int splits, int Cout_real, float *grad, float *bias_partial,
                            int bias_blocks, float *bias_out, int *err, cudaStream_t st, LaunchCounter &lc) {
    if (g.Cin % 8 || g.Mpad % kBM || g.Mpad < g.Kf || g.chunk % kBK) return cudaErrorInvalidValue;
    if (g.Cout != 16 && g.Cout != 32 && g.Cout != 64 && g.Cout != 128 && g.Cout != 256) return cudaErrorInvalidValue;
    ReducePart w{}, bias{};
    auto part = [](ReducePart &r, const float *partial, float *out, size_t stride, int count, int Cst, int Kf, int Cout) {
        // threads per element: enough to fill the chip where the elements alone do not, at most one a partial
        const size_t vecs = (size_t)Kf * Cst / 4;
        int lanes = 1;
        while (lanes < 64 && lanes < count && vecs * lanes < (size_t)kSms * 2048) lanes *= 2;
        const int width = 256 / lanes;
        r = ReducePart{partial, out, stride, count, Cst, Kf, Cout, lanes, (int)((vecs + width - 1) / width)};
    };
    part(w, g.partial, grad, (size_t)g.Mpad * g.Cout, splits, g.Cout, g.Kf, Cout_real);
    if (bias_out) {  // before the products, which start while it runs
        ProfScope _ps(lc, "bias_grad", st);
        const int P = g.batch * g.Ho * g.Wo, lanes = 256 / (g.Cout / 8);
        const int blocks = std::min(bias_blocks, std::max(1, P / (lanes * kColsumUnroll)));
        k_colsum<<<blocks, 256, 0, st>>>(P, g.Cout, static_cast<const __nv_bfloat16 *>(g.dy), bias_partial);
        lc.add(1);
        part(bias, bias_partial, bias_out, (size_t)g.Cout, blocks, g.Cout, 1, Cout_real);
    }
    {
        ProfScope _ps(lc, "conv_wgrad_tc", st);
        const bool beside = bias_out != nullptr;
        cudaError_t e;
        switch (g.Cout) {
            case 16: e = wgrad_launch<16>(g, splits, beside, err, st); break;
            case 32: e = wgrad_launch<32>(g, splits, beside, err, st); break;
            case 64: e = wgrad_launch<64>(g, splits, beside, err, st); break;
            case 128: e = wgrad_launch<128>(g, splits, beside, err, st); break;
            default: e = wgrad_launch<256>(g, splits, beside, err, st); break;
        }
        lc.add(1);
        if (e != cudaSuccess) return e;
    }
    ProfScope _ps(lc, "wgrad_reduce", st);
    k_wgrad_reduce<<<w.blocks + bias.blocks, 256, 0, st>>>(w, bias);
    lc.add(1);
    return cudaGetLastError();
}

static int ew_blocks(size_t n) { return (int)std::min<size_t>((n + 255) / 256, kSms * 16); }

cudaError_t launch_down_sum(int batch, int Hl, int Wl, int C, const void *ds, void *dt, cudaStream_t st,
                            LaunchCounter &lc) {
    ProfScope _ps(lc, "down_sum", st);
    const size_t n = (size_t)batch * Hl * Wl * (C / 8);
    k_down_sum<<<ew_blocks(n), 256, 0, st>>>(batch, Hl, Wl, C, static_cast<const __nv_bfloat16 *>(ds),
                                            static_cast<__nv_bfloat16 *>(dt));
    lc.add(1);
    return cudaGetLastError();
}

cudaError_t launch_output_head(int batch, int HW, int Cy, const float *y, const float *u0, const float *target,
                               float *pred, void *dy, double *loss_partial, int blocks, cudaStream_t st,
                               LaunchCounter &lc) {
    ProfScope _ps(lc, "output_head", st);
    // `blocks` loss partials; without a target there is no FP64 sum and a thread takes one pixel (1024^2: 20 us with the
    // sum of zeros and 304 blocks, 10 now)
    const float4 *y4 = reinterpret_cast<const float4 *>(y);
    const int nb = target ? blocks : (int)(((size_t)batch * HW + 255) / 256);
    const cudaError_t e = launch_pdl(target ? k_output_head<true> : k_output_head<false>, dim3(nb), dim3(256), 0, st, batch,
                                     HW, Cy, y4, u0, target, pred, static_cast<__nv_bfloat16 *>(dy), loss_partial);
    lc.add(1);
    return e;
}

cudaError_t launch_adam(size_t n, float *w, const float *grad, float *m, float *v, float lr_t, float b1, float b2,
                        float eps_t, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "adam", st);
    k_adam<<<ew_blocks(n), 256, 0, st>>>(n, w, grad, m, v, lr_t, b1, b2, eps_t);
    lc.add(1);
    return cudaGetLastError();
}

cudaError_t launch_pack_weights(int Cout, int Cst, int Cin, int taps, int Kpad, int Kdpad, const float *w, void *Wb,
                                void *Wt, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "pack_weights", st);
    const size_t n = (size_t)Cst * Kpad + (size_t)Cin * Kdpad;
    k_pack_weights<<<ew_blocks(n), 256, 0, st>>>(Cout, Cst, Cin, taps, Kpad, Kdpad, w,
                                                 static_cast<__nv_bfloat16 *>(Wb), static_cast<__nv_bfloat16 *>(Wt));
    lc.add(1);
    return cudaGetLastError();
}

}  // namespace lfrv

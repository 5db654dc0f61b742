// kernels_cg.cu -- IBR_gradient: hole filling and the Poisson conjugate gradient (sm_103a).
//
// hole_filling (sources/gradientIBR.cu:87-152, compute_laplacian sources/gradientIBR_kernels.cuh:553-590)
// runs Jacobi diffusion on the non-visible pixels only: the hole list is built once, every iteration reads
// the previous iterate and writes the holes of the other buffer (both buffers share the visible pixels).
//
// possion_conj_grad (sources/solver.cu:526-699) solves (lambda I - Delta_N) u = lambda u0 + grad^T g per
// channel. Its per-pixel operator (updateAlpha :201-310), initial residual (initConjGrad :361-505) and the
// updates (updateSolution :130-198, updateDir :508-523) are restated here; the dot products are FP64
// block partials reduced in a fixed order (the reference accumulates float atomics in arbitrary order).
#include <algorithm>
#include <cstring>
#include <mutex>

#include <cooperative_groups.h>
#include <cudaTypedefs.h>

#include "batch_layout.h"
#include "cg_scalars.h"
#include "device_common.cuh"
#include "tma.cuh"
#include "kernels.h"
#include "lfrv_internal.h"

namespace lfrv {

namespace cg = cooperative_groups;

// Hole list in raster order: one warp per row counts its holes (ballot), one block scans the row counts,
// one warp per row writes its holes in order.
// Zero bytes of 16 visibility bytes (as a 16-bit mask, bit j = byte j) and their count.
__device__ __forceinline__ unsigned int zero_mask16(uint4 v) {
    const unsigned int w[4] = {v.x, v.y, v.z, v.w};
    unsigned int m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned int e = __vcmpeq4(w[i], 0u);  // 0xff in every zero byte
#pragma unroll
        for (int j = 0; j < 4; ++j) m |= ((e >> (8 * j)) & 1u) << (4 * i + j);
    }
    return m;
}

__global__ void k_hole_rows(int W, int H, const uint8_t *__restrict__ vis, int *__restrict__ row_count) {
    pdl_wait();
    pdl_trigger();
    const int y = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (y >= H) return;
    int c = 0;
    if (W % 16 == 0) {
        // 16 pixels per lane and load (rows start on 16-byte boundaries)
        const uint8_t *row = vis + (size_t)y * W;
        for (int x = lane * 16; x < W; x += 512) c += __popc(zero_mask16(*reinterpret_cast<const uint4 *>(row + x)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    } else {
        for (int x0 = 0; x0 < W; x0 += 32) {
            const int x = x0 + lane;
            const bool hole = (x < W) && !vis[(size_t)y * W + x];
            c += __popc(__ballot_sync(0xffffffffu, hole));
        }
    }
    if (lane == 0) row_count[y] = c;
}

// Exclusive scan of H row counts in one block of 1024 threads (chunks of 1024 rows).
__global__ void k_hole_scan(int H, int *__restrict__ row_count, int *__restrict__ total) {
    pdl_wait();
    pdl_trigger();
    __shared__ int warp_tot[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = 0; base < H; base += 1024) {
        const int y = base + threadIdx.x;
        const int v = (y < H) ? row_count[y] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int wt = warp_tot[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, wt, o);
                if (lane >= o) wt += t;
            }
            warp_tot[lane] = wt;  // inclusive over warps
        }
        __syncthreads();
        const int before = (wid > 0) ? warp_tot[wid - 1] : 0;
        if (y < H) row_count[y] = carry + before + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_tot[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_hole_write(int W, int H, const uint8_t *__restrict__ vis, const int *__restrict__ row_start,
                             int *__restrict__ holes) {
    pdl_wait();
    const int y = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (y >= H) return;
    int k = row_start[y];
    if (W % 16 == 0) {
        // 16 pixels per lane and load; a lane's holes go after the holes of the lanes before it
        const uint8_t *row = vis + (size_t)y * W;
        for (int x0 = 0; x0 < W; x0 += 512) {
            const int x = x0 + lane * 16;
            const unsigned int m = (x < W) ? zero_mask16(*reinterpret_cast<const uint4 *>(row + x)) : 0u;
            const int c = __popc(m);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int at = k + incl - c;
            for (unsigned int r = m; r; r &= r - 1) holes[at++] = y * W + x + (__ffs(r) - 1);
            k += __shfl_sync(0xffffffffu, incl, 31);
        }
        return;
    }
    for (int x0 = 0; x0 < W; x0 += 32) {
        const int x = x0 + lane;
        const bool hole = (x < W) && !vis[(size_t)y * W + x];
        const unsigned int m = __ballot_sync(0xffffffffu, hole);
        if (hole) holes[k + __popc(m & ((1u << lane) - 1u))] = y * W + x;
        k += __popc(m);
    }
}

// ------------------------------------------------------------------ conjugate gradient
constexpr int kCgBX = 32, kCgBY = 8;

// Phase 0 of the corrected CG at pixel o: the initial residual r = b - A x with b = lambda u0 + grad^T g
// (initConjGrad, solver.cu:383-467) for the starting iterate x = U, and the energy
// F(x) = lambda/2 |x - u0|^2 + 1/2 |grad x - g|^2 there (the loop lowers it by each step's decrease, so the
// certified gap always refers to the current iterate). Without a separate anchor (U0 == nullptr) x = u0, as in
// the reference; with one, U holds a seed (the learned warm start) while u0 keeps the problem unchanged.
// acc[0..2] += r^2 per channel, acc[3] += the energy. cg_start_values returns the residual of pixel (x, y)
// (o = y W + x) per channel in rv3; cg_start_pixel stores it in r.
__device__ __forceinline__ void cg_start_values(int W, int H, size_t N, size_t o, int x, int y,
                                                const float *__restrict__ gX, const float *__restrict__ gY,
                                                const float *__restrict__ U, const float *__restrict__ U0,
                                                float lambda, float rv3[3], float acc[4]) {
    const float gxo = __ldg(gX + o), gyo = __ldg(gY + o);
    const float gxl = (x > 0) ? __ldg(gX + o - 1) : 0.f, gyu = (y > 0) ? __ldg(gY + o - W) : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float *u = U + c * N;
        const float uc = __ldcg(u + o);
        float lx, ly;
        if (x == 0) lx = uc - __ldcg(u + o + 1) + gxo;
        else if (x < W - 1) lx = 2.f * uc - __ldcg(u + o - 1) - __ldcg(u + o + 1) + gxo - gxl;
        else lx = uc - __ldcg(u + o - 1) - gxl;
        if (y == 0) ly = uc - __ldcg(u + o + W) + gyo;
        else if (y < H - 1) ly = 2.f * uc - __ldcg(u + o - W) - __ldcg(u + o + W) + gyo - gyu;
        else ly = uc - __ldcg(u + o - W) - gyu;
        float rv = -(lx + ly);
        float e = 0.f;
        if (U0) {
            const float dv = __ldcg(U0 + c * N + o) - uc;
            rv += lambda * dv;
            e = lambda * dv * dv;
        }
        rv3[c] = rv;
        acc[c] += rv * rv;
        if (x < W - 1) {
            const float a = __ldcg(u + o + 1) - uc - gxo;
            e += a * a;
        }
        if (y < H - 1) {
            const float a = __ldcg(u + o + W) - uc - gyo;
            e += a * a;
        }
        acc[3] += 0.5f * e;
    }
}

__device__ __forceinline__ void cg_start_pixel(int W, int H, size_t N, size_t o, const float *__restrict__ gX,
                                               const float *__restrict__ gY, const float *__restrict__ U,
                                               const float *__restrict__ U0, float *__restrict__ r, float lambda,
                                               float acc[4]) {
    // 32-bit index arithmetic: images have fewer than 2^31 pixels
    const unsigned int ou = (unsigned int)o;
    const int y = (int)(ou / (unsigned int)W), x = (int)(ou - (unsigned int)y * (unsigned int)W);
    float rv[3];
    cg_start_values(W, H, N, o, x, y, gX, gY, U, U0, lambda, rv, acc);
#pragma unroll
    for (int c = 0; c < 3; ++c) r[c * N + o] = rv[c];
}

// partial layout: [3][nblocks]
__device__ __forceinline__ void cg_block3(double a0, double a1, double a2, double *partial) {
    __shared__ double red[3][8];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, off);
        a1 += __shfl_down_sync(0xffffffffu, a1, off);
        a2 += __shfl_down_sync(0xffffffffu, a2, off);
    }
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = a0;
        red[1][tid >> 5] = a1;
        red[2][tid >> 5] = a2;
    }
    __syncthreads();
    if (tid == 0) {
        const int nb = gridDim.x * gridDim.y, b = blockIdx.y * gridDim.x + blockIdx.x;
        double s0 = 0, s1 = 0, s2 = 0;
        for (int i = 0; i < (kCgBX * kCgBY) / 32; ++i) {
            s0 += red[0][i];
            s1 += red[1][i];
            s2 += red[2][i];
        }
        partial[b] = s0;
        partial[nb + b] = s1;
        partial[2 * nb + b] = s2;
    }
}

__global__ void __launch_bounds__(256) k_cg_energy(int W, int H, const float *__restrict__ U, const float *__restrict__ U0,
                                                   const float *__restrict__ gX, const float *__restrict__ gY,
                                                   double *__restrict__ partial) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const size_t N = (size_t)W * H;
    double acc[3] = {0, 0, 0};
    if (x < W && y < H) {
        const size_t o = (size_t)y * W + x;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float *u = U + c * N;
            const double dd = (double)u[o] - (double)U0[c * N + o];
            double e = 0.5 * dd * dd;
            if (x < W - 1) {
                const double a = (double)u[o + 1] - (double)u[o] - (double)gX[o];
                e += 0.5 * a * a;
            }
            if (y < H - 1) {
                const double a = (double)u[o + W] - (double)u[o] - (double)gY[o];
                e += 0.5 * a * a;
            }
            acc[c] = e;
        }
    }
    cg_block3(acc[0], acc[1], acc[2], partial);
}

// ====================================================================== persistent solvers
// One cooperative launch runs a whole iteration loop; phases are separated by the bounded grid barrier of
// device_common.cuh. Values written by other blocks inside the launch are read through L2 (__ldcg).
constexpr int kPersistThreads = 512;

// Sums of nslots slots of count FP64 values (slot s at p + s * stride) into out_smem[s], in FP64 and a fixed order:
// warp s takes slot s (lane l adds elements l, l + 32, ... in order, eight loads in flight at a time, then a
// shuffle tree). One warp per slot keeps each slot to one round trip to L2 and puts the slots' FP64 trees on
// separate warp schedulers (the FP64 pipe is narrow on this part). Needs a block of at least 32 * nslots threads.
__device__ void reduce_slots(const double *p, int count, size_t stride, int nslots, double *out_smem) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (wid < nslots) {
        const double *q = p + (size_t)wid * stride;
        double s = 0.0;
        for (int base = 0; base < count; base += 256) {
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int i = base + lane + 32 * j;
                v[j] = i < count ? __ldcg(q + i) : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s += v[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) out_smem[wid] = s;
    }
    __syncthreads();
}

__device__ void block_reduce_partials(const double *partial, int count, int nslots, double *out_smem) {
    reduce_slots(partial, count, (size_t)count, nslots, out_smem);
}

// Block sum of up to 4 per-thread FP32 values into partial[slot * stride + blockIdx.x]: warp trees in FP32 (each
// lane holds a handful of terms, the slots interleaved), then warp s adds the warp sums of slot s in FP64 (a
// shuffle tree, fixed order). Every call site reaches a grid barrier next, whose leading block barrier orders
// these stores before the barrier's release and the shared buffer before its next use.
__device__ void block_partials_f(const float v[4], int nslots, double *partial, int stride) {
    __shared__ float red[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    float s[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int sl = 0; sl < 4; ++sl) s[sl] += __shfl_down_sync(0xffffffffu, s[sl], o);
    if (lane == 0) {
#pragma unroll
        for (int sl = 0; sl < 4; ++sl) red[sl][wid] = s[sl];
    }
    __syncthreads();
    if (wid < nslots) {
        double t = lane < nw ? (double)red[wid][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) partial[(size_t)wid * stride + blockIdx.x] = t;
    }
}

// Block sum of up to 4 per-thread values into partial[slot * stride + blockIdx.x] (stride: gridDim.x, or
// the number of participating blocks).
__device__ void block_partials(const double v[4], int nslots, double *partial, int stride) {
    __shared__ double red[kPersistThreads / 32][4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int sl = 0; sl < nslots; ++sl) {
        double s = v[sl];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[wid][sl] = s;
    }
    __syncthreads();
    if (threadIdx.x < nslots) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x / 32); ++w) t += red[w][threadIdx.x];
        partial[(size_t)threadIdx.x * stride + blockIdx.x] = t;
    }
    __syncthreads();
}

__device__ __forceinline__ float ldcg_op(const float *d, int W, int H, int x, int y, size_t o, float lambda) {
    const float c = __ldcg(d + o);
    float lx, ly;
    if (x == 0) lx = c - __ldcg(d + o + 1);
    else if (x < W - 1) lx = 2.f * c - __ldcg(d + o - 1) - __ldcg(d + o + 1);
    else lx = c - __ldcg(d + o - 1);
    if (y == 0) ly = c - __ldcg(d + o + W);
    else if (y < H - 1) ly = 2.f * c - __ldcg(d + o - W) - __ldcg(d + o + W);
    else ly = c - __ldcg(d + o - W);
    return lambda * c + lx + ly;
}

// possion_conj_grad's loop (sources/solver.cu:526-699) as the reference runs it, iterations `first` .. first + count - 1
// in one cooperative launch: beta = 1, the step's denominator dAlpha accumulated over the iterations and receiving
// alpha + r . r after each, r0 . r0 counting the last row twice. Two grid barriers an iteration: after q = A d with d . q,
// and after the update of u, r and d with r . r. state: [0..2] r0 . r0, [3..5] dAlpha, carried from launch to launch.
// Bound by the barriers at small images and by the streams of r, d, q and U at large ones; the scalars stay on the device
// because a copy back for each (11 of them) cost more than the arithmetic: a whole call with host arrays, 8 views of 256^2,
// took 607 us with host-stepped kernels and takes 375 us.
__global__ void __launch_bounds__(kPersistThreads) k_cg_faithful(int W, int H, const float *__restrict__ gX,
                                                                 const float *__restrict__ gY, float *U, float *r,
                                                                 float *d, float *q, double *partA, double *partB,
                                                                 GridBarrier gb, int first, int count, double *state) {
    __shared__ double sh[4];
    const size_t N = (size_t)W * H, stride = (size_t)gridDim.x * blockDim.x;
    const size_t o0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned int gen = 0;
    double delta[3], dAlpha[3];
    if (first == 0) {
        double acc[4] = {0, 0, 0, 0};
        for (size_t o = o0; o < N; o += stride) {
            const int y = (int)(o / W), x = (int)(o - (size_t)y * W);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float *u = U + c * N;
                float lx, ly;
                if (x == 0) lx = u[o] - u[o + 1] + gX[o];
                else if (x < W - 1) lx = 2.f * u[o] - u[o - 1] - u[o + 1] + gX[o] - gX[o - 1];
                else lx = u[o] - u[o - 1] - gX[o - 1];
                if (y == 0) ly = u[o] - u[o + W] + gY[o];
                else if (y < H - 1) ly = 2.f * u[o] - u[o - W] - u[o + W] + gY[o] - gY[o - W];
                else ly = u[o] - u[o - W] - gY[o - W];
                const float rv = -(lx + ly);
                r[c * N + o] = rv;
                d[c * N + o] = rv;
                acc[c] += (double)rv * rv * (y == H - 1 ? 2.0 : 1.0);
            }
        }
        block_partials(acc, 3, partB, gridDim.x);
        if (!grid_sync(gb, gen)) return;
        block_reduce_partials(partB, gridDim.x, 3, sh);
        for (int c = 0; c < 3; ++c) {
            delta[c] = sh[c];
            dAlpha[c] = 0.0;
        }
    } else {
        for (int c = 0; c < 3; ++c) {
            delta[c] = state[c];
            dAlpha[c] = state[3 + c];
        }
    }
    for (int it = 0; it < count; ++it) {
        double acc[4] = {0, 0, 0, 0};
        for (size_t o = o0; o < N; o += stride) {
            const int y = (int)(o / W), x = (int)(o - (size_t)y * W);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float qv = ldcg_op(d + c * N, W, H, x, y, o, 1.0f);
                q[c * N + o] = qv;
                acc[c] += (double)__ldcg(d + c * N + o) * qv;
            }
        }
        block_partials(acc, 3, partA, gridDim.x);
        if (!grid_sync(gb, gen)) return;
        block_reduce_partials(partA, gridDim.x, 3, sh);
        float alpha[3];
        for (int c = 0; c < 3; ++c) {
            dAlpha[c] += sh[c];
            alpha[c] = (float)delta[c] / (float)dAlpha[c];
            acc[c] = 0;
        }
        for (size_t o = o0; o < N; o += stride) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const size_t i = c * N + o;
                const float dv = d[i];
                U[i] += alpha[c] * dv;
                const float rv = r[i] - alpha[c] * q[i];
                r[i] = rv;
                d[i] = rv + dv;
                acc[c] += (double)rv * rv;
            }
        }
        block_partials(acc, 3, partB, gridDim.x);
        if (!grid_sync(gb, gen)) return;
        block_reduce_partials(partB, gridDim.x, 3, sh);
        for (int c = 0; c < 3; ++c) dAlpha[c] = (double)alpha[c] + sh[c];
    }
    if (blockIdx.x == 0 && threadIdx.x < 3) {
        state[threadIdx.x] = delta[threadIdx.x];
        state[3 + threadIdx.x] = dAlpha[threadIdx.x];
    }
}

// Tiles of the persistent CG: kTileX x kTileY pixels staged with a one-pixel halo.
constexpr int kTileX = 64, kTileY = 16, kHaloX = kTileX + 2, kHaloY = kTileY + 2;

// Operator of updateAlpha (sources/solver.cu:222-271) on a shared-memory tile: (tx, ty) is the pixel's tile
// position (halo included), (x, y) its image position for the one-sided border differences.
__device__ __forceinline__ float tile_op(const float (*t)[kHaloX], int tx, int ty, int x, int y, int W, int H,
                                         float lambda) {
    const float c = t[ty][tx];
    float lx, ly;
    if (x == 0) lx = c - t[ty][tx + 1];
    else if (x < W - 1) lx = 2.f * c - t[ty][tx - 1] - t[ty][tx + 1];
    else lx = c - t[ty][tx - 1];
    if (y == 0) ly = c - t[ty + 1][tx];
    else if (y < H - 1) ly = 2.f * c - t[ty - 1][tx] - t[ty + 1][tx];
    else ly = c - t[ty - 1][tx];
    return lambda * c + lx + ly;
}

// TMA form of the operator phases: each tile's halo arrives as one 3-D box per array (all 3 planes), x origin
// rounded down to a 16-byte boundary (x0 - 4), double-buffered so the next tile's box is in flight while the
// current one is used. Box rows are padded to a 128-byte multiple in shared memory.
constexpr int kBoxX = kTileX + 8, kBoxY = kTileY + 2, kBoxPlane = kBoxX * kBoxY;
constexpr unsigned kBoxBytes = 3u * kBoxPlane * sizeof(float);
constexpr unsigned kIntBytes = 3u * kTileX * kTileY * sizeof(float);  // interior box (no halo) of u or r
constexpr int kBoxStride = ((kBoxBytes + 127) / 128) * 128 / sizeof(float);  // floats between box buffers
constexpr size_t kCgTmaSmem = 6 * (size_t)kBoxStride * sizeof(float) + 128;   // 2 stages x 3 slots + alignment

// Operator of updateAlpha on a box in shared memory: f(i) is the value at box index i, ROW floats per box row.
template <int ROW = kBoxX, class F>
__device__ __forceinline__ float box_op(F f, int i, int x, int y, int W, int H, float lambda) {
    const float c = f(i);
    float lx, ly;
    if (x == 0) lx = c - f(i + 1);
    else if (x < W - 1) lx = 2.f * c - f(i - 1) - f(i + 1);
    else lx = c - f(i - 1);
    if (y == 0) ly = c - f(i + ROW);
    else if (y < H - 1) ly = 2.f * c - f(i - ROW) - f(i + ROW);
    else ly = c - f(i - ROW);
    return lambda * c + lx + ly;
}

// Thread 0 waits (bounded) for the stage's box; the block learns the outcome through shared memory, then every
// other thread observes the completed phase itself (it returns at once) so the box contents are visible to it.
__device__ __forceinline__ bool block_wait_box(uint64_t *bar, unsigned parity, int *s_flag) {
    if (threadIdx.x == 0) *s_flag = mbar_wait(bar, parity, kSpinLimit) ? 1 : 0;
    __syncthreads();
    const bool ok = *s_flag != 0;
    if (ok && threadIdx.x != 0) mbar_wait(bar, parity, kSpinLimit);
    return ok;
}

// Corrected CG of the IBR_gradient normal equations, all iterations in one launch. State layout (doubles):
// [0..2] delta, [3] E, [4] gap, [5] iterations, [6] status (0 ok, 1 barrier timeout).
// TMA = true reads the operator phases' tiles through the tensor maps of r, dA and dB (W a multiple of 4).
template <bool TMA>
__global__ void __launch_bounds__(kPersistThreads) k_cg_persistent(int W, int H, const float *__restrict__ gX,
                                                                   const float *__restrict__ gY, float *U,
                                                                   const float *U0, float *r,
                                                                   float *dA, float *dB, double *partA,
                                                                   double *partB, GridBarrier gb, int max_iter,
                                                                   double gap_tol, double *state,
                                                                   double *trace, int trace_cap,
                                                                   const __grid_constant__ CUtensorMap mapR,
                                                                   const __grid_constant__ CUtensorMap mapA,
                                                                   const __grid_constant__ CUtensorMap mapB,
                                                                   const __grid_constant__ CUtensorMap mapUi,
                                                                   const __grid_constant__ CUtensorMap mapRi) {
    __shared__ double sh[8];
    const size_t N = (size_t)W * H;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nthr = (size_t)gridDim.x * blockDim.x;
    __shared__ float tile[TMA ? 1 : 3][TMA ? 1 : kHaloY][TMA ? 1 : kHaloX];
    extern __shared__ __align__(128) float dyn_smem[];
    // TMA destinations: [stage][slot][kBoxStride], 128-byte aligned explicitly
    float *boxes = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(dyn_smem) + 127) & ~uintptr_t(127));
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int s_flag;
    unsigned par[2] = {0u, 0u};
    const int tiles_x = (W + kTileX - 1) / kTileX, ntiles = tiles_x * ((H + kTileY - 1) / kTileY);
    const int nk = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const float lambda = 1.0f;
    unsigned int gen = 0;
    if (TMA && threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_proxy_async_smem();
    }
    __syncthreads();
    // thread 0 starts the loads of this block's k-th tile into stage k & 1. Phase A: halo boxes of r and d_old
    // (slots 0, 1). Phase B: halo box of d_new (slot 0) and the interior boxes of u and r (slots 1, 2).
    auto slot = [&](int st, int j) { return boxes + (size_t)(3 * st + j) * kBoxStride; };
    auto issue = [&](int k, bool phase_b, const CUtensorMap *halo1) {
        if (threadIdx.x != 0) return;
        const int t = (int)blockIdx.x + k * (int)gridDim.x, st = k & 1;
        const int x0 = (t % tiles_x) * kTileX, y0 = (t / tiles_x) * kTileY;
        fence_proxy_async_smem();
        if (!phase_b) {
            mbar_arrive_expect_tx(&bars[st], 2 * kBoxBytes);
            tma_load_3d(slot(st, 0), &mapR, x0 - 4, y0 - 1, 0, &bars[st]);
            tma_load_3d(slot(st, 1), halo1, x0 - 4, y0 - 1, 0, &bars[st]);
        } else {
            mbar_arrive_expect_tx(&bars[st], kBoxBytes + 2 * kIntBytes);
            tma_load_3d(slot(st, 0), halo1, x0 - 4, y0 - 1, 0, &bars[st]);
            tma_load_3d(slot(st, 1), &mapUi, x0, y0, 0, &bars[st]);
            tma_load_3d(slot(st, 2), &mapRi, x0, y0, 0, &bars[st]);
        }
    };
    // on a box that never arrived: flag the error, give the other stage's load a bounded wait, leave
    auto abandon = [&](int k) {
        if (threadIdx.x == 0) {
            atomicExch(gb.err, 1);
            if (k + 1 < nk) mbar_wait(&bars[(k + 1) & 1], par[(k + 1) & 1], kSpinLimit);
        }
    };
    // ---- phase 0: r = b - A x (initConjGrad, solver.cu:383-467) and the energy F(x)
    {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (size_t o = tid; o < N; o += nthr) {
            cg_start_pixel(W, H, N, o, gX, gY, U, U0, r, lambda, acc);
        }
        block_partials_f(acc, 4, partB, gridDim.x);
    }
    if (TMA) fence_proxy_async_global();
    if (!grid_sync(gb, gen)) return;
    block_reduce_partials(partB, gridDim.x, 4, sh);
    // The FP64 scalars (delta, E, gap) live in thread 0 of each block, which derives the float coefficients
    // and the stop decision and hands them to the block through shared memory (every block computes the same
    // values from the same partials, so the grid agrees).
    __shared__ float s_coef[3];
    __shared__ int s_stop;
    double delta[3] = {sh[0], sh[1], sh[2]};
    double E = sh[3];
    float beta[3] = {0.f, 0.f, 0.f};
    const float *dold = r;  // d_0 = r_0 (beta = 0)
    float *dnew = dA;
    double gap = 1e300;
    int it = 0;
    for (;; ++it) {
        if (threadIdx.x == 0) {
            const double bound = (delta[0] + delta[1] + delta[2]) / (2.0 * (double)lambda);
            gap = (E - bound) > 0 ? bound / (E - bound) : 1e300;
            s_stop = (it >= max_iter || (gap_tol > 0 && gap <= gap_tol)) ? 1 : 0;
        }
        __syncthreads();
        if (s_stop) break;
        // ---- phase A: d = r + beta d_old on each tile + halo in shared memory, q = A d, d . q
        float accA[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (TMA) {
            const CUtensorMap *mdold = (dold == r) ? &mapR : (dold == dA ? &mapA : &mapB);
            if (nk > 0) issue(0, false, mdold);
            for (int k = 0; k < nk; ++k) {
                if (k + 1 < nk) issue(k + 1, false, mdold);
                const int st = k & 1;
                if (!block_wait_box(&bars[st], par[st], &s_flag)) {
                    abandon(k);
                    return;
                }
                par[st] ^= 1u;
                const int t = (int)blockIdx.x + k * (int)gridDim.x;
                const int x0 = (t % tiles_x) * kTileX, y0 = (t / tiles_x) * kTileY;
                const float *R = slot(st, 0), *D = slot(st, 1);
                for (int p = threadIdx.x; p < kTileX * kTileY; p += blockDim.x) {
                    const int lx = p % kTileX, ly = p / kTileX, x = x0 + lx, y = y0 + ly;
                    if (x >= W || y >= H) continue;
                    const size_t o = (size_t)y * W + x;
                    const int bi = (ly + 1) * kBoxX + (lx + 4);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float *Rc = R + c * kBoxPlane, *Dc = D + c * kBoxPlane;
                        const float b = beta[c];
                        auto v = [&](int i) { return Rc[i] + b * Dc[i]; };
                        const float qv = box_op(v, bi, x, y, W, H, lambda);
                        const float dcv = v(bi);
                        dnew[c * N + o] = dcv;
                        accA[c] += dcv * qv;
                    }
                }
                __syncthreads();
            }
        } else {
            float *acc = accA;
            for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
                const int x0 = (t % tiles_x) * kTileX, y0 = (t / tiles_x) * kTileY;
                for (int k = threadIdx.x; k < 3 * kHaloY * kHaloX; k += blockDim.x) {
                    const int c = k / (kHaloY * kHaloX), rem = k % (kHaloY * kHaloX);
                    const int gx = x0 - 1 + rem % kHaloX, gy = y0 - 1 + rem / kHaloX;
                    float v = 0.f;
                    if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
                        const size_t o = c * N + (size_t)gy * W + gx;
                        v = __ldcg(r + o) + beta[c] * __ldcg(dold + o);
                    }
                    tile[c][rem / kHaloX][rem % kHaloX] = v;
                }
                __syncthreads();
                for (int p = threadIdx.x; p < kTileX * kTileY; p += blockDim.x) {
                    const int lx = p % kTileX, ly = p / kTileX, x = x0 + lx, y = y0 + ly;
                    if (x >= W || y >= H) continue;
                    const size_t o = (size_t)y * W + x;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float qv = tile_op(tile[c], lx + 1, ly + 1, x, y, W, H, lambda);
                        const float dcv = tile[c][ly + 1][lx + 1];
                        dnew[c * N + o] = dcv;
                        acc[c] += dcv * qv;
                    }
                }
                __syncthreads();
            }
        }
        block_partials_f(accA, 3, partA, gridDim.x);
        if (TMA) fence_proxy_async_global();
        if (!grid_sync(gb, gen)) return;
        block_reduce_partials(partA, gridDim.x, 3, sh);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double alpha_d = (sh[c] > 0) ? delta[c] / sh[c] : 0.0;
                s_coef[c] = (float)alpha_d;
                E -= 0.5 * alpha_d * delta[c];
            }
            if (blockIdx.x == 0 && trace && it < trace_cap) trace[it] = E;
        }
        __syncthreads();
        const float alpha[3] = {s_coef[0], s_coef[1], s_coef[2]};
        // ---- phase B: x += alpha d, r -= alpha A d, r . r (d tile + halo in shared memory)
        float accB[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (TMA) {
            const CUtensorMap *mdnew = (dnew == dA) ? &mapA : &mapB;
            if (nk > 0) issue(0, true, mdnew);
            for (int k = 0; k < nk; ++k) {
                if (k + 1 < nk) issue(k + 1, true, mdnew);
                const int st = k & 1;
                if (!block_wait_box(&bars[st], par[st], &s_flag)) {
                    abandon(k);
                    return;
                }
                par[st] ^= 1u;
                const int t = (int)blockIdx.x + k * (int)gridDim.x;
                const int x0 = (t % tiles_x) * kTileX, y0 = (t / tiles_x) * kTileY;
                const float *Dn = slot(st, 0), *Ui = slot(st, 1), *Ri = slot(st, 2);
                for (int p = threadIdx.x; p < kTileX * kTileY; p += blockDim.x) {
                    const int lx = p % kTileX, ly = p / kTileX, x = x0 + lx, y = y0 + ly;
                    if (x >= W || y >= H) continue;
                    const size_t o = (size_t)y * W + x;
                    const int bi = (ly + 1) * kBoxX + (lx + 4);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float *Dc = Dn + c * kBoxPlane;
                        auto v = [&](int i) { return Dc[i]; };
                        const float qv = box_op(v, bi, x, y, W, H, lambda);
                        const float dv = Dc[bi];
                        U[c * N + o] = Ui[c * kTileX * kTileY + p] + alpha[c] * dv;
                        const float rv = Ri[c * kTileX * kTileY + p] - alpha[c] * qv;
                        r[c * N + o] = rv;
                        accB[c] += rv * rv;
                    }
                }
                __syncthreads();
            }
        } else {
            float *acc = accB;
            for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
                const int x0 = (t % tiles_x) * kTileX, y0 = (t / tiles_x) * kTileY;
                for (int k = threadIdx.x; k < 3 * kHaloY * kHaloX; k += blockDim.x) {
                    const int c = k / (kHaloY * kHaloX), rem = k % (kHaloY * kHaloX);
                    const int gx = x0 - 1 + rem % kHaloX, gy = y0 - 1 + rem / kHaloX;
                    tile[c][rem / kHaloX][rem % kHaloX] =
                        (gx >= 0 && gx < W && gy >= 0 && gy < H) ? __ldcg(dnew + c * N + (size_t)gy * W + gx) : 0.f;
                }
                __syncthreads();
                for (int p = threadIdx.x; p < kTileX * kTileY; p += blockDim.x) {
                    const int lx = p % kTileX, ly = p / kTileX, x = x0 + lx, y = y0 + ly;
                    if (x >= W || y >= H) continue;
                    const size_t o = (size_t)y * W + x;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float qv = tile_op(tile[c], lx + 1, ly + 1, x, y, W, H, lambda);
                        const float dv = tile[c][ly + 1][lx + 1];
                        U[c * N + o] = __ldcg(U + c * N + o) + alpha[c] * dv;
                        const float rv = __ldcg(r + c * N + o) - alpha[c] * qv;
                        r[c * N + o] = rv;
                        acc[c] += rv * rv;
                    }
                }
                __syncthreads();
            }
        }
        block_partials_f(accB, 3, partB, gridDim.x);
        if (TMA) fence_proxy_async_global();
        if (!grid_sync(gb, gen)) return;
        block_reduce_partials(partB, gridDim.x, 3, sh);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s_coef[c] = (delta[c] > 0) ? (float)(sh[c] / delta[c]) : 0.f;
                delta[c] = sh[c];
            }
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 3; ++c) beta[c] = s_coef[c];
        dold = dnew;
        dnew = (dnew == dA) ? dB : dA;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        state[0] = delta[0];
        state[1] = delta[1];
        state[2] = delta[2];
        state[3] = E;
        state[4] = gap;
        state[5] = (double)it;
    }
}

// On-chip strip form of the corrected CG (units of 64 x R pixels and one channel, kStripUnits spatial units per SM,
// R <= 28).
//
// One warp owns one unit: lane l holds columns 2l and 2l + 1 of its rows. r (with a ring of ghost cells) and s = A d
// stay in shared memory, x and d in registers (they meet no neighbour), so an iteration touches no global memory
// beyond the units' borders. A ghost cell inside the image is a copy of the neighbour unit's pixel; one outside it
// repeats the border pixel, which is the operator's one-sided difference there, so the stencil has no border cases.
//
// One barrier per iteration (Chronopoulos and Gear's form of CG): with w = A r, gamma = r . r and delta = r . w,
//   beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old),
//   s = w + beta s, d = r + beta d, x += alpha d, r -= alpha s,
// which are CG's iterates with both dot products of an iteration in one reduction. A unit publishes the border of
// its w (not of r) before the barrier; afterwards the neighbours apply the same recurrence to their copies of its
// border (s_h = w_h + beta s_h, r_h -= alpha s_h), so their halo of r equals the owner's r bit for bit without a
// second exchange. Borders and block partials are double-buffered by iteration parity: a block that has passed the
// barrier writes the next set while a slower one still reads this one. A step whose denominator is not positive
// (rounding at FP32's floor, long after the certified gap) restarts from the residual (beta = 0).
// Dot products: FP32 over four rows (eight where a unit has no more) of two columns that a lane adds, pairs of floats (CgSum,
// some 42 bits) across those chunks and a warp's lanes, FP64 across warps and blocks. The streamed form adds fewer pixels a lane, but the lanes of a
// warp in FP32; with FP32 up to the warp here too, 1792 products would be added before FP64.
//
// Measured against the shared-memory form with two barriers an iteration that stood here before, 25 iterations: 64^2 249 ->
// 103 us, 384^2 275 -> 143, 512^2 322 -> 151, 768^2 422 -> 217, 1024^2 (152 blocks, R = 28) 547 -> 315. Bound at 1024^2 by
// the walks (about 160 cycles a row of a warp, three warps a scheduler), below 512^2 by the reduction, the barrier and the
// FP64 scalars between two iterations.
constexpr int kStripWarps = kStripUnits * 3, kStripThreads = kStripWarps * 32;
constexpr int kStripSlots = 7;                               // gamma x 3, delta x 3, the starting energy
constexpr int kStripChunk = 4;                               // rows that a lane adds in FP32 (the walk's unrolling)

constexpr int kStripRow = kStripCols + 4;                    // a row of r: 2 words (ghost in the second), 64 columns, ghost

// per warp: r with its ghost rows (and one row read ahead of need), s
__host__ __device__ constexpr int strip_warp_floats(int R) { return (R + 3) * kStripRow + R * kStripCols; }
constexpr size_t strip_smem(int R) { return sizeof(float) * kStripWarps * (size_t)strip_warp_floats(R); }

// a / b in FP64 for the solver's scalars: an FP32 reciprocal refined by Newton steps in FP64 (a few dependent
// FMAs instead of the full division sequence, whose latency sits on the path every block waits for). The
// result is within a few units in the last place of the rounded quotient; b outside the FP32 range takes
// the division.
__device__ __forceinline__ double res_div(double a, double b) {
    const double ab = fabs(b);
    if (!(ab > 1e-30 && ab < 1e30)) return a / b;
    double r = (double)__frcp_rn((float)b);
    r = fma(r, fma(-b, r, 1.0), r);  // ~46 bits
    r = fma(r, fma(-b, r, 1.0), r);  // full precision
    const double q = a * r;
    return fma(r, fma(-b, q, a), q);
}

// cg_start_values for one channel at (x, y): the initial residual; e receives the pixel's energy. Branch-free (a
// neighbour outside the image is the pixel itself, a gradient across the border 0), so that the loads of several
// pixels are in flight together.
__device__ __forceinline__ float strip_start(int W, int H, int x, int y, const float *gX, const float *gY,
                                             const float *u, const float *u0, float &e) {
    const size_t o = (size_t)y * W + x;
    const float uc = u[o];
    const float ul = u[x > 0 ? o - 1 : o], ur = u[x < W - 1 ? o + 1 : o];
    const float uu = u[y > 0 ? o - W : o], ud = u[y < H - 1 ? o + W : o];
    const float gxo = x < W - 1 ? __ldg(gX + o) : 0.f, gyo = y < H - 1 ? __ldg(gY + o) : 0.f;
    const float gxl = x > 0 ? __ldg(gX + o - 1) : 0.f, gyu = y > 0 ? __ldg(gY + o - W) : 0.f;
    const float dv = u0 ? u0[o] - uc : 0.f;
    const float ex = ur - uc - gxo, ey = ud - uc - gyo;
    e = 0.5f * (dv * dv + ex * ex + ey * ey);
    const float lx = 2.f * uc - ul - ur + gxo - gxl, ly = 2.f * uc - uu - ud + gyo - gyu;
    return dv - (lx + ly);
}

// Sums of nslots slots (slot s: count FP64 values at p + s * stride) into out[s]: warp s, a fixed order. The loads of
// a lane are in flight together; the tree is only as deep as the lanes that hold values (FP64 latency is on the path
// of every iteration).
__device__ __forceinline__ void strip_reduce(const double *p, int count, size_t stride, int nslots, double *out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (wid < nslots) {
        const double *q = p + (size_t)wid * stride;
        double t = 0.0;
        for (int base = 0; base < count; base += 128) {
            double v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = base + lane + 32 * j < count ? __ldcg(q + base + lane + 32 * j) : 0.0;
            if (count > 32) v[0] = (v[0] + v[1]) + (v[2] + v[3]);
            t = base ? t + v[0] : v[0];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            if (count > o) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) out[wid] = t;
    }
    __syncthreads();
}

// probs == nullptr: one problem (`one`) on the whole grid; else block b works on problem block_prob[b]. Every
// problem has its own barrier words (gb.count + 8 * problem) and its own columns of the partial arrays.
template <int R>
__global__ void __launch_bounds__(kStripThreads, 1) k_cg_strip(const CgProblem one, const CgProblem *__restrict__ probs,
                                                               const int *__restrict__ block_prob, double *partA,
                                                               double *partB, GridBarrier gb, int cluster) {
    constexpr int NB = strip_border(R);
    static_assert(R <= 32, "a ghost column is one value per lane");
    extern __shared__ __align__(16) float strip_mem[];
    __shared__ double sh[8], s_dE[3], s_den[3], s_ig[3], s_ia[3];
    __shared__ float s_coef[6];
    __shared__ CgSum red[kStripWarps][3];
    __shared__ int s_stop;
    const int pid = probs ? block_prob[blockIdx.x] : 0;
    const CgProblem P = probs ? probs[pid] : one;
    const int W = P.W, H = P.H, lb = (int)blockIdx.x - P.b0, G = (int)gridDim.x;
    const size_t N = (size_t)W * H;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = warp % 3;
    const int cols = (W + kStripCols - 1) / kStripCols, rows = (H + R - 1) / R;
    const int u = lb * kStripUnits + warp / 3;
    const bool active = u < cols * rows;
    const int ry = u / cols, cx = u - ry * cols;
    const int x = cx * kStripCols + 2 * lane, y0 = ry * R;
    const int nrows = active ? min(R, H - y0) : 0;
    const bool ina = active && x < W, inb = active && x + 1 < W;
    const bool top = ry == 0, bottom = y0 + nrows == H;
    const bool left = cx > 0, right = cx + 1 < cols;  // a unit on that side
    const bool edgeL = lane == 0, edge = lane == 0 || lane == 31;
    const bool borderL = x == 0, borderA = x == W - 1, borderB = x + 1 == W - 1;  // image columns 0 and W - 1
    float *Rw = strip_mem + (size_t)warp * strip_warp_floats(R) + kStripRow + 2;  // row 0, column 0
    float *Rl = Rw + 2 * lane;                                                   // this lane's pair in row 0
    float2 *Ss = reinterpret_cast<float2 *>(Rw - 2 + (R + 2) * kStripRow) + lane;
    float *U = P.U + (size_t)c * N;
    const float *U0 = P.U0 ? P.U0 + (size_t)c * N : nullptr;
    GridBarrier bar = gb;
    bar.count = gb.count + 8 * pid;
    unsigned int gen = 0;
    auto border = [&](int set, int unit) { return (set ? P.dB : P.dA) + ((size_t)unit * 3 + c) * NB; };
    auto pair = [](float *p) -> float2 & { return *reinterpret_cast<float2 *>(p); };
    float2 X[R], D[R];
    float2 st = {}, sb = {};     // s on the ghost rows
    float sl = 0.f, sr = 0.f;    // s on the ghost columns (row = lane)
    CgSum e = {0.f, 0.f};
    // ---- start: r = b - A x on the unit and its ghost ring (outside the image: the border pixel), F(x)
    if (active) {
        auto start = [&](int px, int py, float &en) {
            return strip_start(W, H, min(max(px, 0), W - 1), min(max(py, 0), H - 1), P.gx, P.gy, U, U0, en);
        };
        float e0, e1, none;
        {
            // the ghost ring
            const float2 gt = make_float2(start(x, y0 - 1, none), start(x + 1, y0 - 1, none));
            const float2 gb2 = make_float2(start(x, y0 + nrows, none), start(x + 1, y0 + nrows, none));
            const float gl = start(cx * kStripCols - 1, y0 + min(lane, nrows - 1), none);
            const float gr = start((cx + 1) * kStripCols, y0 + min(lane, nrows - 1), none);
            pair(Rl - kStripRow) = gt;
            pair(Rl + nrows * kStripRow) = gb2;
            if (lane < nrows) {
                Rw[lane * kStripRow - 1] = gl;
                Rw[lane * kStripRow + kStripCols] = gr;
            }
        }
#pragma unroll 4
        for (int j = 0; j < nrows; ++j) {
            pair(Rl + j * kStripRow) = make_float2(start(x, y0 + j, e0), start(x + 1, y0 + j, e1));
            e = cg_add(e, {(ina ? e0 : 0.f) + (inb ? e1 : 0.f), 0.f});
            Ss[j * 32] = make_float2(0.f, 0.f);
        }
        __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
        X[j] = D[j] = make_float2(0.f, 0.f);
        if (j < nrows) {
            if (ina) X[j].x = __ldcg(U + (size_t)(y0 + j) * W + x);
            if (inb) X[j].y = __ldcg(U + (size_t)(y0 + j) * W + x + 1);
        }
    }
    // walks the rows: f(j, r of row j, w = A r of row j); the next row is read before f may overwrite row j
    auto walk = [&](auto f) {
        float2 up = pair(Rl - kStripRow), cur = pair(Rl), nxt = pair(Rl + kStripRow);
        float l = Rl[-1], q = Rl[2];
        float *row = Rl + kStripRow;
#pragma unroll 4
        for (int j = 0; j < nrows; ++j, row += kStripRow) {
            float2 w;
            w.x = cur.x + (2.f * cur.x - l - cur.y) + (2.f * cur.x - up.x - nxt.x);
            w.y = cur.y + (2.f * cur.y - cur.x - q) + (2.f * cur.y - up.y - nxt.y);
            const float2 after = pair(row + kStripRow);
            l = row[-1];
            q = row[2];
            f(j, cur, w);
            up = cur;
            cur = nxt;
            nxt = after;
        }
    };
    // dot products of the current r, w's border into set `set`, block partials into part
    auto dots = [&](int set, double *part, bool energy) {
        float g0 = 0.f, g1 = 0.f, d0 = 0.f, d1 = 0.f;
        CgSum g = {0.f, 0.f}, d = {0.f, 0.f};
        float *B = border(set, active ? u : 0);
        float2 *Brow = reinterpret_cast<float2 *>(B) + lane;
        float *col = edgeL ? B + 2 * kStripCols : B + 2 * kStripCols + R;
        auto fold = [&]() {
            g = cg_add(g, {(ina ? g0 : 0.f) + (inb ? g1 : 0.f), 0.f});
            d = cg_add(d, {(ina ? d0 : 0.f) + (inb ? d1 : 0.f), 0.f});
            g0 = g1 = d0 = d1 = 0.f;
        };
        if (active) {
            walk([&](int j, float2 v, float2 w) {
                if (j == 0) Brow[0] = w;
                if (j == nrows - 1) Brow[32] = w;
                if (edge) *col = edgeL ? w.x : w.y;
                ++col;
                g0 = fmaf(v.x, v.x, g0);
                g1 = fmaf(v.y, v.y, g1);
                d0 = fmaf(v.x, w.x, d0);
                d1 = fmaf(v.y, w.y, d1);
                if (R > 2 * kStripChunk && (j & (kStripChunk - 1)) == kStripChunk - 1) fold();
            });
            fold();
        }
        // lanes 0 to 15 go on with g, the others with d
        auto from = [&](CgSum v, int o) {
            return CgSum{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        };
        const bool upper = lane >= 16;
        CgSum h = cg_add(upper ? d : g, from(upper ? g : d, 16));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) h = cg_add(h, from(h, o));
        if (energy) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e = cg_add(e, from(e, o));
            if (lane == 0) red[warp][2] = cg_result(e);
        }
        if ((lane & 15) == 0) red[warp][lane >> 4] = cg_result(h);
        __syncthreads();
        if (threadIdx.x < 6) {
            const CgSum *v = &red[threadIdx.x % 3][threadIdx.x / 3];
            static_assert(kStripUnits == 4, "four units per channel");
            const double hi = ((double)v[0].hi + (double)v[9].hi) + ((double)v[18].hi + (double)v[27].hi);
            part[(size_t)threadIdx.x * G + blockIdx.x] = hi + (double)((v[0].lo + v[9].lo) + (v[18].lo + v[27].lo));
        } else if (threadIdx.x == 6 && energy) {
            double t = 0.0;
#pragma unroll
            for (int k = 0; k < kStripWarps; ++k) t += (double)red[k][2].hi + (double)red[k][2].lo;
            part[(size_t)6 * G + blockIdx.x] = t;
        }
    };
    auto sync_all = [&]() {
        if (cluster) {
            asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
            return true;
        }
        if (P.nb == 1) {
            __syncthreads();
            return true;
        }
        return grid_sync(bar, gen, (unsigned int)P.nb);
    };
    dots(0, partA, true);
    // The FP64 scalars. An FP64 operation has a latency of some dozens of cycles, so the path every warp waits for
    // holds only beta, the denominator and the step length (warp 0, one channel per lane; cg_quotient) beside the stop test
    // (warp 1); the quotients that the next iteration needs (1 / gamma, 1 / alpha, the energy's decrease) follow on nine
    // lanes of the last warp while the others go on (an FP64 instruction holds the SM's pipe as long for one lane as
    // for 32).
    double E = 0.0;  // warp 1's copy is the one in use
    if (threadIdx.x < 3) s_ig[threadIdx.x] = s_ia[threadIdx.x] = 0.0;
    for (int it = 0;; ++it) {
        if (!sync_all()) return;
        const int set = it & 1;
        // the neighbours' borders, in flight while the partials are summed
        float2 wt = {}, wb = {};
        float wl = 0.f, wr = 0.f;
        if (active && !top) wt = __ldcg(reinterpret_cast<const float2 *>(border(set, u - cols)) + 32 + lane);
        if (active && !bottom) wb = __ldcg(reinterpret_cast<const float2 *>(border(set, u + cols)) + lane);
        if (lane < nrows && left) wl = __ldcg(border(set, u - 1) + 2 * kStripCols + R + lane);
        if (lane < nrows && right) wr = __ldcg(border(set, u + 1) + 2 * kStripCols + lane);
        strip_reduce((set ? partB : partA) + P.b0, P.nb, (size_t)G, it == 0 ? kStripSlots : 6, sh);
        if (threadIdx.x < 3) {
            const double gam = sh[threadIdx.x], del = sh[3 + threadIdx.x];
            double beta = gam * s_ig[threadIdx.x], den = fma(-beta, gam * s_ia[threadIdx.x], del);
            if (!(den > 0.0)) {
                // (a residual whose square is infinite does not restart: infinity by infinity, the channel shows it)
                beta = gam > 1e300 ? (double)NAN : 0.0;
                den = del;
            }
            s_coef[threadIdx.x] = den > 0.0 ? cg_quotient(gam, den) : 0.f;
            s_coef[3 + threadIdx.x] = (float)beta;
            s_den[threadIdx.x] = den;
        }
        if (threadIdx.x == 32) {
            if (it == 0) E = sh[6];
            else {
                E = E - s_dE[0] - s_dE[1] - s_dE[2];
                if (lb == 0 && P.trace && it <= P.trace_cap) P.trace[it - 1] = E;
            }
            // gap = bound / (E - bound) <= gap_tol, tested without the division
            const double bound = 0.5 * (sh[0] + sh[1] + sh[2]), room = E - bound;
            s_stop = (it >= P.max_iter || (P.gap_tol > 0 && room > 0 && bound <= P.gap_tol * room)) ? 1 : 0;
            if (s_stop && lb == 0) {
                P.state[0] = sh[0];
                P.state[1] = sh[1];
                P.state[2] = sh[2];
                P.state[3] = E;
                P.state[4] = room > 0 ? bound / room : 1e300;
                P.state[5] = (double)it;
            }
        }
        __syncthreads();
        if (s_stop) break;
        if (warp == kStripWarps - 1 && lane < 9) {
            const int k = lane % 3, what = lane / 3;
            const double gam = sh[k], den = s_den[k];
            const bool step = gam > 0.0 && den > 0.0;
            const double q = step ? res_div(what == 0 ? 1.0 : (what == 1 ? den : gam), what == 2 ? den : gam) : 0.0;
            if (what == 0) s_ig[k] = q;
            else if (what == 1) s_ia[k] = q;
            else s_dE[k] = 0.5 * gam * q;
        }
        const float alpha = s_coef[c], beta = s_coef[3 + c];
        // (rows past the unit hold nothing that is read later)
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const float2 v = pair(Rl + j * kStripRow);
            D[j].x = fmaf(beta, D[j].x, v.x);
            D[j].y = fmaf(beta, D[j].y, v.y);
            X[j].x = fmaf(alpha, D[j].x, X[j].x);
            X[j].y = fmaf(alpha, D[j].y, X[j].y);
        }
        if (active) {
            __syncwarp();
            walk([&](int j, float2 v, float2 w) {
                float2 q = Ss[j * 32];
                q.x = fmaf(beta, q.x, w.x);
                q.y = fmaf(beta, q.y, w.y);
                Ss[j * 32] = q;
                float2 n = make_float2(fmaf(-alpha, q.x, v.x), fmaf(-alpha, q.y, v.y));
                __syncwarp();  // every lane has read row j and its neighbours
                float *cell = Rl + j * kStripRow;
                if (borderA) n.y = n.x;
                if (ina) pair(cell) = n;
                if (borderL) cell[-1] = n.x;
                if (borderB) cell[2] = n.y;
                if (top && j == 0) pair(cell - kStripRow) = n;
                if (bottom && j == nrows - 1) pair(cell + kStripRow) = n;
            });
            auto ghost = [&](float &sv, float &rv, float wv) {
                sv = fmaf(beta, sv, wv);
                rv = fmaf(-alpha, sv, rv);
            };
            if (!top) {
                float2 &g = pair(Rl - kStripRow);
                ghost(st.x, g.x, wt.x);
                ghost(st.y, g.y, wt.y);
            }
            if (!bottom) {
                float2 &g = pair(Rl + nrows * kStripRow);
                ghost(sb.x, g.x, wb.x);
                ghost(sb.y, g.y, wb.y);
            }
            if (lane < nrows && left) ghost(sl, Rw[lane * kStripRow - 1], wl);
            if (lane < nrows && right) ghost(sr, Rw[lane * kStripRow + kStripCols], wr);
            __syncwarp();
        }
        dots(set ^ 1, set ? partA : partB, false);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (j < nrows) {
            if (ina) U[(size_t)(y0 + j) * W + x] = X[j].x;
            if (inb) U[(size_t)(y0 + j) * W + x + 1] = X[j].y;
        }
    }
}

// Hole filling in shared memory, without a grid barrier: one block (C = 1) for at most kSmallHoles holes, or one
// cluster of C blocks for at most C * kSmallHoles, each block holding a contiguous share of the sorted hole list.
// The visible pixels never change, so every hole keeps, per direction (left, up, right, down: the summation order
// of compute_laplacian), either a reference to the neighbouring hole (block rank << 11 | index in that block's
// share) or the neighbour's fixed value; the iterations then touch shared memory only, a cluster's blocks reading
// each other's shares through distributed shared memory, with one cluster barrier per iteration. Each update
// gives k_hole_fill_persistent's value bit for bit (its division by the neighbour count is a corrected
// reciprocal product). holes must be in ascending pixel order with the row starts behind them (launch_hole_list).
constexpr int kSmallHoles = 2048, kSmallThreads = 1024, kHoleCluster = 8;
static_assert(kSmallHoles == 1 << 11 && kHoleCluster * kSmallHoles <= 32767, "hole references are 16-bit");
constexpr size_t kSmallHoleSmem = (size_t)kSmallHoles * (6 * 4 + 12 * 4 + 4 * 2 + 4);

// Shared arrays of a block besides the dynamic ones.
struct HoleShared {
    float rws[kSmallHoles];  // 1 / wts
    float wsum[2][kSmallThreads / 32];
    int holes[kSmallHoles];
};

template <int C>
__device__ __forceinline__ void hole_fill_small(int W, int H, const int *__restrict__ holes, int nh, float *A, int max_iter,
                                                double *state, float *hsm, HoleShared &sh) {
    float *cur = hsm, *nxt = hsm + 3 * kSmallHoles;            // [3][kSmallHoles] each
    float *fixedv = hsm + 6 * kSmallHoles;                      // [4 dirs][3][kSmallHoles]
    float *wts = hsm + 18 * kSmallHoles;                        // [kSmallHoles]
    short *nb = reinterpret_cast<short *>(hsm + 19 * kSmallHoles);  // [4][kSmallHoles]: reference, -1 fixed, -2 none
    float *rws = sh.rws;
    float(&wsum)[2][kSmallThreads / 32] = sh.wsum;
    int *s_holes = sh.holes;
    const int rank = C > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int chunk = (nh + C - 1) / C, h0 = rank * chunk, nloc = max(0, min(nh - h0, chunk));
    const size_t N = (size_t)W * H;
    for (int h = threadIdx.x; h < nloc; h += kSmallThreads) s_holes[h] = __ldg(holes + h0 + h);
    __syncthreads();
    // row starts of the hole list (launch_hole_list keeps them in holes[N .. N + H)): a vertical neighbour is
    // searched in its row's few holes only, a horizontal one is the adjacent entry of the sorted list
    const int *row_start = holes + N;
    for (int h = threadIdx.x; h < nloc; h += kSmallThreads) {
        const int g = h0 + h, o = s_holes[h];
        const int ox = o % W, oy = o / W;
        const bool has[4] = {ox > 0, oy > 0, ox < W - 1, oy < H - 1};
        const int q[4] = {o - 1, o - W, o + 1, o + W};
        int lo[4] = {g - 1, 0, g + 1, 0}, hi[4] = {g - 1, -1, min(g + 1, nh - 1), -1};
        if (has[1]) {
            lo[1] = __ldg(row_start + oy - 1);
            hi[1] = __ldg(row_start + oy) - 1;
        }
        if (has[3]) {
            lo[3] = __ldg(row_start + oy + 1);
            hi[3] = (oy + 2 < H ? __ldg(row_start + oy + 2) : nh) - 1;
        }
        float wt = 0.f;
        short idx4[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            short idx = -2;
            if (has[d]) {
                wt += 1.f;
                idx = -1;
                int l = max(lo[d], 0), r = hi[d];
                while (l <= r) {
                    const int mid = (l + r) >> 1, v = __ldg(holes + mid);
                    if (v == q[d]) {
                        const int rr = mid / chunk;
                        idx = (short)((rr << 11) | (mid - rr * chunk));
                        break;
                    }
                    if (v < q[d]) l = mid + 1;
                    else r = mid - 1;
                }
            }
            idx4[d] = idx;
            nb[d * kSmallHoles + h] = idx;
        }
        wts[h] = wt;
        rws[h] = 1.0f / wt;
        // the fixed neighbours' values and the hole's own, all loads issued together
#pragma unroll
        for (int d = 0; d < 4; ++d)
            if (idx4[d] == -1)
                for (int c = 0; c < 3; ++c) fixedv[(d * 3 + c) * kSmallHoles + h] = A[c * N + q[d]];
        for (int c = 0; c < 3; ++c) cur[c * kSmallHoles + h] = A[c * N + o];
    }
    // a cluster: every block's share is in place before any block reads another's
    if constexpr (C > 1) cg::this_cluster().sync();
    else __syncthreads();
    // one block: only the warps that hold holes iterate (at least one, so that an empty hole set reports its one
    // iteration as the reference does); the others leave, and the iterations synchronise on named barrier 1 with
    // the iterating threads' count. A cluster: every thread takes part in the cluster barriers.
    const int active = C > 1 ? kSmallThreads : max(32, min(kSmallThreads, (nloc + 31) & ~31));
    if ((int)threadIdx.x >= active) return;
    float energy = 0.0f, previous = 0.0f;
    int k;
    for (k = 0; k < max_iter; ++k) {
        previous = energy;
        // the energy in FP32 (a handful of terms per thread, fixed shuffle trees): the FP64 pipe of this part is
        // narrow, and the stop test compares single-precision energies
        float acc = 0.f;
        for (int h = threadIdx.x; h < nloc; h += kSmallThreads) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float v = 0.f;
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const short idx = nb[d * kSmallHoles + h];
                    if (idx == -2) continue;
                    if (idx == -1) {
                        v += fixedv[(d * 3 + c) * kSmallHoles + h];
                    } else {
                        const int rr = idx >> 11, l = idx & (kSmallHoles - 1);
                        const float *src = cur + c * kSmallHoles + l;
                        if constexpr (C > 1)
                            if (rr != rank) src = cg::this_cluster().map_shared_rank(src, rr);
                        v += *src;
                    }
                }
                // v / wt as the reciprocal product with one residual correction (Markstein): with rw the
                // rounded reciprocal and q within an ulp of the quotient, q + rw (v - wt q) is the correctly
                // rounded quotient, i.e. the division's result bit for bit (no underflow at these magnitudes)
                {
                    const float wt = wts[h], rw = rws[h];
                    const float q = v * rw;
                    v = fmaf(fmaf(-q, wt, v), rw, q);
                }
                const float uc = cur[c * kSmallHoles + h];
                const float lap = v - uc;
                const float un = uc + lap;
                nxt[c * kSmallHoles + h] = un;
                if (c == 2) acc += lap * un;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        // one barrier per iteration: the warp sums alternate between two slots, and every warp sums the 32 of
        // this iteration (of each block in rank order) with the same fixed tree, so all agree
        const int lane = threadIdx.x & 31;
        if (lane == 0) wsum[k & 1][threadIdx.x >> 5] = acc;
        float tot;
        if constexpr (C > 1) {
            cg::this_cluster().sync();
            tot = 0.f;
            for (int rr = 0; rr < C; ++rr) {
                const float *ws = cg::this_cluster().map_shared_rank(&wsum[k & 1][0], rr);
                float t = ws[lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
                tot += __shfl_sync(0xffffffffu, t, 0);
            }
        } else {
            asm volatile("bar.sync 1, %0;" ::"r"(active) : "memory");
            tot = (lane < active / 32) ? wsum[k & 1][lane] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(0xffffffffu, tot, o);
        }
        energy = __shfl_sync(0xffffffffu, tot, 0);
        float *t = cur;
        cur = nxt;
        nxt = t;
        if (fabsf(previous - energy) < 1e-3f) {
            ++k;
            break;
        }
    }
    for (int h = threadIdx.x; h < nloc; h += kSmallThreads) {
        const int o = s_holes[h];
#pragma unroll
        for (int c = 0; c < 3; ++c) A[c * N + o] = cur[c * kSmallHoles + h];
    }
    if (rank == 0 && threadIdx.x == 0) state[0] = (double)k;
    // no block leaves while another may still read its shared memory
    if constexpr (C > 1) cg::this_cluster().sync();
}

// C = 1: at most kSmallHoles holes. C > 1: at most C times as many; the first block alone fills what one block holds (its
// barrier is the cheaper one), so that one launch serves both ranges: a second one that finds nothing to do took 2 to 5 us
// of a render (64^2 137 -> 135 us, 24 views of 301 x 203 241 -> 236).
template <int C>
__global__ void __launch_bounds__(kSmallThreads) k_hole_fill_small(int W, int H, const int *__restrict__ holes,
                                                                   const int *__restrict__ count, float *A,
                                                                   int max_iter, double *state) {
    extern __shared__ __align__(16) float hsm[];
    __shared__ HoleShared sh;
    const int nh = *count;
    // every block of a cluster returns together, before any cluster barrier
    if (nh > C * kSmallHoles) return;
    if (C > 1 && nh > kSmallHoles) hole_fill_small<C>(W, H, holes, nh, A, max_iter, state, hsm, sh);
    else if (blockIdx.x == 0) hole_fill_small<1>(W, H, holes, nh, A, max_iter, state, hsm, sh);
}

// Hole filling with the whole iteration loop in one launch (hole_filling, sources/gradientIBR.cu:87-152).
// count: device pointer to the number of holes. A holds the initial image (and the result); B is scratch, into
// which the kernel first copies every hole's value and its neighbours' (the pixels the iterations read).
// state: [0] iterations.
// Only as many blocks as the hole count needs take part (kHoleFillPerBlock holes each; the others return at
// once), so the grid barrier of each iteration spans few blocks, and none is needed when one block suffices. The energy partials alternate between two
// slots by iteration parity: a block overwrites slot k & 1 in iteration k + 2 only after every block passed
// the barrier of iteration k + 1, i.e. after all of them read it, so one barrier per iteration suffices.
constexpr int kHoleFillPerBlock = 4 * kPersistThreads;

__global__ void __launch_bounds__(kPersistThreads) k_hole_fill_persistent(int W, int H, const int *__restrict__ holes,
                                                                          const int *__restrict__ count, float *A,
                                                                          float *B, double *part, GridBarrier gb,
                                                                          int max_iter, double *state, int handled) {
    __shared__ double sh[8];
    const size_t N = (size_t)W * H;
    const int nh = *count;
    if (nh <= handled) return;  // k_hole_fill_small (one block or one cluster) has done it
    const int active = min((int)gridDim.x, max(1, (nh + kHoleFillPerBlock - 1) / kHoleFillPerBlock));
    if ((int)blockIdx.x >= active) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = active * blockDim.x;
    unsigned int gen = 0;
    // B = A at the holes and their neighbours; every copy of one pixel writes the same value
    for (int h = tid; h < nh; h += nthr) {
        const int o = __ldg(holes + h);
        const int ox = o % W, oy = o / W;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t p = (size_t)c * N + o;
            B[p] = __ldcg(A + p);
            if (ox > 0) B[p - 1] = __ldcg(A + p - 1);
            if (oy > 0) B[p - W] = __ldcg(A + p - W);
            if (ox < W - 1) B[p + 1] = __ldcg(A + p + 1);
            if (oy < H - 1) B[p + W] = __ldcg(A + p + W);
        }
    }
    if (active > 1) {
        if (!grid_sync(gb, gen, active)) return;
    } else {
        __syncthreads();
    }
    float *src = A, *dst = B;
    float energy = 0.0f, previous = 0.0f;
    int k;
    for (k = 0; k < max_iter; ++k) {
        previous = energy;
        double acc[4] = {0, 0, 0, 0};
        for (int h = tid; h < nh; h += nthr) {
            const int o = __ldg(holes + h);
            const int ox = o % W, oy = o / W;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float *u = src + c * N;
                float v = 0.f, wt = 0.f;
                if (ox > 0) { v += __ldcg(u + o - 1); wt += 1.f; }
                if (oy > 0) { v += __ldcg(u + o - W); wt += 1.f; }
                if (ox < W - 1) { v += __ldcg(u + o + 1); wt += 1.f; }
                if (oy < H - 1) { v += __ldcg(u + o + W); wt += 1.f; }
                v /= wt;
                const float uc = __ldcg(u + o);
                const float lap = v - uc;
                const float un = uc + lap;
                dst[c * N + o] = un;
                if (c == 2) acc[0] += (double)(lap * un);
            }
        }
        double *slot = part + (size_t)(k & 1) * active;
        block_partials(acc, 1, slot, active);
        if (active > 1) {
            if (!grid_sync(gb, gen, active)) return;
        } else {
            __syncthreads();  // one block: its own global writes are visible to it after the block barrier
        }
        block_reduce_partials(slot, active, 1, sh);
        energy = (float)sh[0];
        float *t = src;
        src = dst;
        dst = t;
        if (fabsf(previous - energy) < 1e-3f) {
            ++k;
            break;
        }
    }
    if (src != A) {  // copy the holes of the result back into A
        for (int h = tid; h < nh; h += nthr) {
            const int o = __ldg(holes + h);
#pragma unroll
            for (int c = 0; c < 3; ++c) A[c * N + o] = __ldcg(src + c * N + o);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) state[0] = (double)k;
}

// ------------------------------------------------------------------ Jacobi Poisson integration
// poisson_jacobi (sources/gradientIBR.cu:923-1013): z = (m u0 - div g) / (4 + m) per channel (compute_divergence,
// jacobi_z, sources/gradientIBR_kernels.cuh:553-598), then sweeps x <- (x_l + x_u + x_r + x_d) / (4 + m) + z with the
// border pixel standing in for a missing neighbour (jacobi_B :600-643). The reference launches 2 kernels per channel
// and sweep; here one cooperative launch runs every sweep of all three channels, kJacK sweeps per grid barrier: a
// block stages its tile with a halo of kJacK pixels in shared memory (each sweep's stencil reaches one pixel) and
// ping-pongs there. Every operation is the reference's float expression in its order, without contraction.
constexpr int kJacTX = 32, kJacTY = 16, kJacK = 4, kJacThreads = 512;
constexpr int kJacRX = kJacTX + 2 * kJacK, kJacRY = kJacTY + 2 * kJacK, kJacRN = kJacRX * kJacRY;
constexpr size_t kJacSmem = (size_t)10 * kJacRN * sizeof(float);  // x (3 channels x 2 buffers), z (3), 4 + m

__global__ void k_jacobi_setup(int W, int H, const float *__restrict__ gX, const float *__restrict__ gY,
                               const float *__restrict__ mask, const float *__restrict__ U, float *__restrict__ z,
                               float *__restrict__ den) {
    const int ox = blockIdx.x * blockDim.x + threadIdx.x, oy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ox >= W || oy >= H) return;
    const size_t o = (size_t)oy * W + ox, N = (size_t)W * H;
    float dv = 0.0f;
    if (ox != 0 && ox != W - 1) dv = __fadd_rn(dv, __fsub_rn(gX[o + 1], gX[o - 1]) / 2);
    if (oy != 0 && oy != H - 1) dv = __fadd_rn(dv, __fsub_rn(gY[o + W], gY[o - W]) / 2);
    const float data_w = __fmul_rn(1.0f, mask[o]);
    const float d = __fadd_rn(4.0f, data_w);
    den[o] = d;
#pragma unroll
    for (int c = 0; c < 3; ++c) z[c * N + o] = __fsub_rn(__fmul_rn(data_w, U[c * N + o]), dv) / d;
}

__global__ void __launch_bounds__(kJacThreads) k_jacobi_persistent(int W, int H, int iters,
                                                                   const float *__restrict__ z,
                                                                   const float *__restrict__ den, float *U0, float *U1,
                                                                   GridBarrier gb) {
    extern __shared__ float jsm[];
    float *sX = jsm, *sZ = jsm + 6 * kJacRN, *sD = jsm + 9 * kJacRN;  // sX: [buffer][channel][kJacRN]
    const int tiles_x = (W + kJacTX - 1) / kJacTX, ntiles = tiles_x * ((H + kJacTY - 1) / kJacTY);
    const size_t N = (size_t)W * H;
    unsigned int gen = 0;
    int step = 0;
    for (int done = 0; done < iters; done += kJacK, ++step) {
        const int n_it = min(kJacK, iters - done);
        const float *Ui = (step & 1) ? U1 : U0;
        float *Uo = (step & 1) ? U0 : U1;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int rx0 = (t % tiles_x) * kJacTX - kJacK, ry0 = (t / tiles_x) * kJacTY - kJacK;
            for (int i = threadIdx.x; i < kJacRN; i += kJacThreads) {
                const int gx = rx0 + i % kJacRX, gy = ry0 + i / kJacRX;
                const bool in = gx >= 0 && gx < W && gy >= 0 && gy < H;
                const size_t o = in ? (size_t)gy * W + gx : 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    sX[c * kJacRN + i] = in ? __ldcg(Ui + c * N + o) : 0.f;
                    sZ[c * kJacRN + i] = in ? __ldg(z + c * N + o) : 0.f;
                }
                sD[i] = in ? __ldg(den + o) : 1.f;
            }
            __syncthreads();
            for (int it = 0; it < n_it; ++it) {
                const float *src = sX + (it & 1) * 3 * kJacRN;
                float *dst = sX + ((it + 1) & 1) * 3 * kJacRN;
                for (int i = threadIdx.x; i < kJacRN; i += kJacThreads) {
                    const int lx = i % kJacRX, ly = i / kJacRX, gx = rx0 + lx, gy = ry0 + ly;
                    if (gx < 0 || gx >= W || gy < 0 || gy >= H) continue;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float *x = src + c * kJacRN;
                        const float xc = x[i];
                        // neighbours outside the staged region are stale only where the tile does not look
                        const float xl = gx == 0 ? xc : (lx > 0 ? x[i - 1] : 0.f);
                        const float xu = gy == 0 ? xc : (ly > 0 ? x[i - kJacRX] : 0.f);
                        const float xr = gx == W - 1 ? xc : (lx + 1 < kJacRX ? x[i + 1] : 0.f);
                        const float xd = gy == H - 1 ? xc : (ly + 1 < kJacRY ? x[i + kJacRX] : 0.f);
                        float v = 0.0f;
                        v = __fadd_rn(v, xl);
                        v = __fadd_rn(v, xu);
                        v = __fadd_rn(v, xr);
                        v = __fadd_rn(v, xd);
                        v = v / sD[i];
                        dst[c * kJacRN + i] = __fadd_rn(v, sZ[c * kJacRN + i]);
                    }
                }
                __syncthreads();
            }
            const float *res = sX + (n_it & 1) * 3 * kJacRN;
            for (int i = threadIdx.x; i < kJacTX * kJacTY; i += kJacThreads) {
                const int lx = kJacK + i % kJacTX, ly = kJacK + i / kJacTX, gx = rx0 + lx, gy = ry0 + ly;
                if (gx >= W || gy >= H) continue;
                const size_t o = (size_t)gy * W + gx;
                const int r = ly * kJacRX + lx;
#pragma unroll
                for (int c = 0; c < 3; ++c) Uo[c * N + o] = res[c * kJacRN + r];
            }
            __syncthreads();  // the next tile overwrites the staged region
        }
        if (!grid_sync(gb, gen)) return;
    }
}

// ------------------------------------------------------------------ launchers
static inline dim3 cg_grid(int W, int H) { return dim3((W + kCgBX - 1) / kCgBX, (H + kCgBY - 1) / kCgBY); }
int cg_partials(int W, int H) {
    const dim3 g = cg_grid(W, H);
    return (int)(g.x * g.y);
}

void launch_hole_list(int W, int H, const uint8_t *vis, int *holes, int *count, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "hole_list", st);
    // row starts are kept in holes[N .. N + H) scratch supplied by the caller (holes has N + H entries)
    int *row = holes + (size_t)W * H;
    const int rows_per_block = 256 / 32;
    // programmatic launches: each kernel's launch overlaps the tail of the one before it
    const dim3 rows_grid((H + rows_per_block - 1) / rows_per_block);
    launch_pdl(k_hole_rows, rows_grid, dim3(256), 0, st, W, H, vis, row);
    launch_pdl(k_hole_scan, dim3(1), dim3(1024), 0, st, H, row, count);
    launch_pdl(k_hole_write, rows_grid, dim3(256), 0, st, W, H, vis, row, holes);
    lc.add(3);
}

// Blocks of a cooperative launch: every block must be resident at once (the grid barrier waits for all).
static int coop_blocks(const void *kernel, int want, size_t smem = 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPersistThreads, smem);
    per_sm = per_sm < 2 ? per_sm : 2;
    const int resident = sms * per_sm;
    return want < resident ? (want > 0 ? want : 1) : resident;
}

int persistent_partials() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return 2 * sms;
}

cudaError_t launch_poisson_jacobi(int W, int H, int iters, const float *gx, const float *gy, const float *mask,
                                  float *U, float *U1, float *z, float *den, GridBarrier gb, cudaStream_t st,
                                  LaunchCounter &lc) {
    ProfScope _ps(lc, "poisson_jacobi", st);
    const dim3 b(32, 8), g((W + 31) / 32, (H + 7) / 8);
    k_jacobi_setup<<<g, b, 0, st>>>(W, H, gx, gy, mask, U, z, den);
    lc.add(1);
    if (iters <= 0) return cudaGetLastError();
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jacobi_persistent, kJacThreads, kJacSmem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int ntiles = ((W + kJacTX - 1) / kJacTX) * ((H + kJacTY - 1) / kJacTY);
    const int resident = sms * per_sm;
    const int per_block = (ntiles + resident - 1) / resident;
    const int blocks = std::max(1, (ntiles + per_block - 1) / per_block);
    void *args[] = {&W, &H, &iters, (void *)&z, (void *)&den, &U, &U1, &gb};
    e = cudaLaunchCooperativeKernel((const void *)k_jacobi_persistent, dim3(blocks), dim3(kJacThreads), args, kJacSmem,
                                    st);
    lc.add(1);
    if (e != cudaSuccess) return e;
    // an odd number of super-steps leaves the result in U1
    const int steps = (iters + kJacK - 1) / kJacK;
    if (steps & 1) return cudaMemcpyAsync(U, U1, sizeof(float) * 3 * (size_t)W * H, cudaMemcpyDeviceToDevice, st);
    return cudaSuccess;
}

// ------------------------------------------------------------------ strip CG: rule and launch
// Whether a block of k_cg_strip<R> fits an SM of the current device. The attribute belongs to the device's context, which
// a program may reset, so it is set every time, as the other launchers do, and the occupancy asked with it.
template <int R>
static bool strip_ready() {
    const void *kern = (const void *)k_cg_strip<R>;
    int per_sm = 0;
    const bool ok =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strip_smem(R)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kStripThreads, strip_smem(R)) == cudaSuccess &&
        per_sm >= 1;
    if (!ok) cudaGetLastError();  // a refused query leaves no error behind
    return ok;
}

// Blocks of a strip launch that can be resident at once: one per SM, 0 (every image runs the streamed form) where the
// largest does not fit.
static int strip_capacity() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return strip_ready<kCgBatchMaxRows>() ? sms : 0;
}

template <int R>
static cudaError_t launch_strip_r(int blocks, const CgProblem &one, const CgProblem *probs, const int *block_prob,
                                  double *partA, double *partB, GridBarrier gb, cudaStream_t st) {
    const void *kern = (const void *)k_cg_strip<R>;
    const size_t smem = strip_smem(R);
    if (!strip_ready<R>()) return cudaErrorInvalidConfiguration;
    int dev = 0;
    cudaGetDevice(&dev);
    // per device: whether one cluster of kStripClusterBlocks can be placed
    static std::mutex mu;
    static int placed[64] = {};  // 0 unknown, 1 yes, -1 no
    bool fits = false;
    if (R <= kStripClusterR && dev >= 0 && dev < 64) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            std::lock_guard<std::mutex> lock(mu);
            if (placed[dev] == 0) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(kStripClusterBlocks);
                cfg.blockDim = dim3(kStripThreads);
                cfg.dynamicSmemBytes = smem;
                cudaLaunchAttribute at[1];
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim = {kStripClusterBlocks, 1, 1};
                cfg.attrs = at;
                cfg.numAttrs = 1;
                int n = 0;
                placed[dev] = cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1 ? 1 : -1;
            }
            fits = placed[dev] > 0;
        }
        if (!fits) cudaGetLastError();
    }
    int cluster = (!probs && blocks > 1 && blocks <= kStripClusterBlocks && fits) ? 1 : 0;
    void *args[] = {(void *)&one, (void *)&probs, (void *)&block_prob, &partA, &partB, &gb, &cluster};
    if (cluster) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(kStripThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {(unsigned)blocks, 1, 1};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelExC(&cfg, kern, args);
    }
    return cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kStripThreads), args, smem, st);
}

static cudaError_t launch_strip(int R, int blocks, const CgProblem &one, const CgProblem *probs, const int *block_prob,
                                double *partA, double *partB, GridBarrier gb, cudaStream_t st) {
    switch (R) {
        case 4: return launch_strip_r<4>(blocks, one, probs, block_prob, partA, partB, gb, st);
        case 8: return launch_strip_r<8>(blocks, one, probs, block_prob, partA, partB, gb, st);
        case 16: return launch_strip_r<16>(blocks, one, probs, block_prob, partA, partB, gb, st);
        case kCgBatchMaxRows: return launch_strip_r<kCgBatchMaxRows>(blocks, one, probs, block_prob, partA, partB, gb, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_cg_persistent(int W, int H, const float *gx, const float *gy, float *U, float *r, float *dA,
                                 float *dB, double *partA, double *partB, GridBarrier gb, int max_iter, double gap_tol,
                                 double *state, cudaStream_t st, LaunchCounter &lc, const float *U0,
                                 double *trace, int trace_cap) {
    ProfScope _ps(lc, "cg_persistent", st);
    const int ntiles = ((W + kTileX - 1) / kTileX) * ((H + kTileY - 1) / kTileY);
    {
        CgProblem one = {};
        one.W = W;
        one.H = H;
        one.max_iter = max_iter;
        one.gap_tol = gap_tol;
        one.gx = gx;
        one.gy = gy;
        one.U = U;
        one.dA = dA;
        one.dB = dB;
        one.state = state;
        one.U0 = U0;
        one.trace = trace;
        one.trace_cap = trace_cap;
        const int R = strip_rows(W, H, strip_capacity());
        if (R > 0) {
            if (!cg_borders_aligned(dA, dB)) return cudaErrorMisalignedAddress;
            one.nb = strip_blocks(W, H, R);
            lc.add(1);
            return launch_strip(R, one.nb, one, nullptr, nullptr, partA, partB, gb, st);
        }
    }
    // the TMA form needs row pitches of a multiple of 16 bytes (W % 4 == 0) and the driver's encoder
    CUtensorMap maps[5];
    const bool tma = encode_tensor_map_3d(&maps[0], r, W, H, 3, kBoxX, kBoxY, 3) &&
                     encode_tensor_map_3d(&maps[1], dA, W, H, 3, kBoxX, kBoxY, 3) &&
                     encode_tensor_map_3d(&maps[2], dB, W, H, 3, kBoxX, kBoxY, 3) &&
                     encode_tensor_map_3d(&maps[3], U, W, H, 3, kTileX, kTileY, 3) &&
                     encode_tensor_map_3d(&maps[4], r, W, H, 3, kTileX, kTileY, 3);
    if (!tma) std::memset(maps, 0, sizeof(maps));
    const void *kern = tma ? (const void *)k_cg_persistent<true> : (const void *)k_cg_persistent<false>;
    const size_t smem = tma ? kCgTmaSmem : 0;
    if (tma) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    // as many blocks as can be resident, then as few as keep the per-block tile count at its minimum (equal
    // tile counts: no block waits at the grid barrier for a straggler with one tile more)
    const int resident = coop_blocks(kern, 1 << 30, smem);
    const int per_block = (ntiles + resident - 1) / resident;
    const int blocks = std::max(1, (ntiles + per_block - 1) / per_block);
    void *args[] = {&W,     &H,       (void *)&gx, (void *)&gy, &U,       (void *)&U0, &r,        &dA,
                    &dB,    &partA,   &partB,      &gb,         &max_iter, &gap_tol,   &state,    &trace,
                    &trace_cap, &maps[0], &maps[1], &maps[2], &maps[3], &maps[4]};
    lc.add(1);
    return cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kPersistThreads), args, smem, st);
}

cudaError_t launch_cg_faithful(int W, int H, const float *gx, const float *gy, float *U, float *r, float *d, float *q,
                               double *partA, double *partB, GridBarrier gb, int first, int count, double *state,
                               cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "cg_faithful", st);
    const size_t N = (size_t)W * H;
    const int want = (int)std::min<size_t>((N + kPersistThreads - 1) / kPersistThreads, 1 << 20);
    const int blocks = coop_blocks((const void *)k_cg_faithful, want);
    void *args[] = {&W, &H, (void *)&gx, (void *)&gy, &U, &r, &d, &q, &partA, &partB, &gb, &first, &count, &state};
    lc.add(1);
    return cudaLaunchCooperativeKernel((const void *)k_cg_faithful, dim3(blocks), dim3(kPersistThreads), args, 0, st);
}

int cg_batch_resident_blocks() { return strip_capacity(); }

int cg_batch_blocks(int W, int H, int R) { return strip_fits(W, H, R) ? strip_blocks(W, H, R) : 0; }

// The smallest R whose blocks of all the images fit the GPU together (as strip_rows for one image); 0: none.
int cg_batch_rows(const CgProblem *probs, int count) {
    const int capacity = strip_capacity();
    for (int R : kStripRows) {
        long long blocks = 0;
        for (int i = 0; i < count && blocks <= capacity; ++i) {
            const int b = cg_batch_blocks(probs[i].W, probs[i].H, R);
            blocks += b > 0 ? b : capacity + 1;
        }
        if (blocks <= capacity) return R;
    }
    return 0;
}

cudaError_t launch_cg_batch(const CgProblem *probs, int count, const CgProblem *d_probs, const int *d_block_prob, int R,
                            int blocks, double *partA, double *partB, GridBarrier gb, cudaStream_t st,
                            LaunchCounter &lc) {
    for (int i = 0; i < count; ++i)
        if (!cg_borders_aligned(probs[i].dA, probs[i].dB)) return cudaErrorMisalignedAddress;
    ProfScope _ps(lc, "cg_batch", st);
    lc.add(1);
    return launch_strip(R, blocks, CgProblem{}, d_probs, d_block_prob, partA, partB, gb, st);
}

void *tensor_map_encoder() {
    static void *encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = fn;
        cudaGetLastError();
    });
    return encode;
}

bool encode_tensor_map_3d(CUtensorMap *map, const float *base, int cols, int rows, int planes, int box_x, int box_y,
                          int box_z) {
    const auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encoder());
    if (!encode || !base || cols <= 0 || rows <= 0 || planes <= 0) return false;
    if (((size_t)cols * sizeof(float)) % 16 != 0 || reinterpret_cast<uintptr_t>(base) % 16 != 0) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * sizeof(float), (cuuint64_t)cols * rows * sizeof(float)};
    const cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_y, (cuuint32_t)box_z};
    const cuuint32_t estride[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(base), dims, strides, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_hole_fill_persistent(int W, int H, const int *holes, const int *count, float *A, float *B,
                                        double *part, GridBarrier gb, int max_iter, double *state, cudaStream_t st,
                                        LaunchCounter &lc) {
    // The hole count is on the device: the shared-memory form (one cluster of kHoleCluster blocks, where the device can
    // place one, whose first block alone fills what one block holds; else one block) and the grid-wide kernel are both
    // queued, and each returns at once unless the count is in its range.
    int handled = kSmallHoles;
    {
        ProfScope _ps(lc, "hole_fill_small", st);
        int dev = 0;
        cudaGetDevice(&dev);
        // per device: the shared-memory attributes, and whether a cluster of kHoleCluster such blocks fits
        static std::mutex mu;
        static int cluster_ok[64] = {};  // 0 unknown, 1 yes, -1 no
        const int slot = (dev >= 0 && dev < 64) ? dev : 0;
        int use_cluster = 0;
        {
            std::lock_guard<std::mutex> lock(mu);
            if (cluster_ok[slot] == 0) {
                cudaError_t e = cudaFuncSetAttribute(k_hole_fill_small<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)kSmallHoleSmem);
                if (e != cudaSuccess) return e;
                int ok = -1;
                if (cudaFuncSetAttribute(k_hole_fill_small<kHoleCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmallHoleSmem) == cudaSuccess) {
                    cudaLaunchConfig_t q = {};
                    cudaLaunchAttribute at[1];
                    at[0].id = cudaLaunchAttributeClusterDimension;
                    at[0].val.clusterDim.x = kHoleCluster;
                    at[0].val.clusterDim.y = 1;
                    at[0].val.clusterDim.z = 1;
                    q.gridDim = dim3(kHoleCluster);
                    q.blockDim = dim3(kSmallThreads);
                    q.dynamicSmemBytes = kSmallHoleSmem;
                    q.attrs = at;
                    q.numAttrs = 1;
                    int nclusters = 0;
                    if (cudaOccupancyMaxActiveClusters(&nclusters, (const void *)k_hole_fill_small<kHoleCluster>, &q) ==
                            cudaSuccess &&
                        nclusters >= 1)
                        ok = 1;
                }
                cudaGetLastError();  // a refused query leaves no error behind
                cluster_ok[slot] = ok;
            }
            use_cluster = cluster_ok[slot] > 0;
        }
        cudaError_t e;
        if (use_cluster) {
            cudaLaunchConfig_t q = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = kHoleCluster;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            q.gridDim = dim3(kHoleCluster);
            q.blockDim = dim3(kSmallThreads);
            q.dynamicSmemBytes = kSmallHoleSmem;
            q.stream = st;
            q.attrs = at;
            q.numAttrs = 1;
            e = cudaLaunchKernelEx(&q, k_hole_fill_small<kHoleCluster>, W, H, holes, count, A, max_iter, state);
            handled = kHoleCluster * kSmallHoles;
        } else {
            k_hole_fill_small<1><<<1, kSmallThreads, kSmallHoleSmem, st>>>(W, H, holes, count, A, max_iter, state);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) return e;
        lc.add(1);
    }
    ProfScope _ps(lc, "hole_fill", st);
    const size_t N = (size_t)W * H;
    const int blocks =
        coop_blocks((const void *)k_hole_fill_persistent, (int)((N + kPersistThreads - 1) / kPersistThreads));
    void *args[] = {&W, &H, (void *)&holes, (void *)&count, &A, &B, &part, &gb, &max_iter, &state, &handled};
    lc.add(1);
    return cudaLaunchCooperativeKernel((const void *)k_hole_fill_persistent, dim3(blocks), dim3(kPersistThreads), args,
                                       0, st);
}

void launch_cg_energy(int W, int H, const float *U, const float *U0, const float *gx, const float *gy, double *partial,
                      cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "cg_energy", st);
    k_cg_energy<<<cg_grid(W, H), dim3(kCgBX, kCgBY), 0, st>>>(W, H, U, U0, gx, gy, partial);
    lc.add(1);
}

}  // namespace lfrv

// ====================================================================== allocation-free CG entry point
// lfrv_cg_solve_static runs the corrected CG (k_cg_strip, or k_cg_persistent for images too thin for it) with all of its
// scratch in one file-scope device array instead of context buffers: r and the two buffers of directions or borders (3
// planes of kStaticPixels floats each), two arrays of FP64 block partials (7 doubles per block of k_cg_strip, one block per
// SM; 4 per block of k_cg_persistent, at most two per SM), 16 doubles of solver state, 64 bytes of barrier words.
namespace {

constexpr size_t kStaticPixels = LFRV_CG_STATIC_MAX_PIXELS;
constexpr int kStaticBlocks = 1024;  // blocks of k_cg_persistent the partial slots hold (2 per SM for <= 512 SMs)
static_assert(lfrv::kStripSlots <= 2 * 4, "a block of k_cg_strip per SM needs no more than two of k_cg_persistent");
constexpr size_t kStaticVecBytes = 9 * kStaticPixels * sizeof(float);
constexpr size_t kStaticPartBytes = 2 * 4 * (size_t)kStaticBlocks * sizeof(double);
constexpr size_t kStaticStateBytes = 16 * sizeof(double);
constexpr size_t kStaticBarrierBytes = 64;
constexpr size_t kStaticBytes = kStaticVecBytes + kStaticPartBytes + kStaticStateBytes + kStaticBarrierBytes;
static_assert(kStaticVecBytes % 256 == 0 && kStaticPartBytes % 64 == 0, "scratch sections stay aligned");
constexpr int kMaxDevices = 64;

__device__ __align__(256) unsigned char g_cg_scratch[kStaticBytes];

std::mutex g_scratch_mu;
unsigned char *g_scratch_addr[kMaxDevices] = {};
void *g_scratch_ctx[kMaxDevices] = {};  // the driver context the cached address belongs to

// The calling thread's current driver context (cuCtxGetCurrent through the runtime's entry-point query, so the
// library does not link the driver library directly); nullptr when it cannot be asked.
void *current_driver_context() {
    using Fn = int (*)(void **);
    static Fn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<Fn>(f);
        cudaGetLastError();
    });
    void *ctx = nullptr;
    if (!fn || fn(&ctx) != 0) return nullptr;
    return ctx;
}

// Address of this device's copy of g_cg_scratch, looked up with that device current the first time a driver
// context of the device calls here. Keyed by the context: after a cudaDeviceReset, or under another context of the
// same ordinal, the module is loaded again and the array moves, so the address is looked up again.
unsigned char *static_scratch(int dev) {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    void *ctx = current_driver_context();
    if (!g_scratch_addr[dev] || !ctx || ctx != g_scratch_ctx[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_cg_scratch);
        if (e != cudaSuccess || !p)
            lfrv::raise(LFRV_E_CUDA, "cudaGetSymbolAddress(g_cg_scratch): %s", cudaGetErrorString(e));
        g_scratch_addr[dev] = static_cast<unsigned char *>(p);
        g_scratch_ctx[dev] = current_driver_context();  // the runtime has made the primary context current by now
    }
    return g_scratch_addr[dev];
}

}  // namespace

extern "C" int lfrv_cg_solve_static(void *stream, int W, int H, int max_iter, double gap_tol, const float *gx,
                                    const float *gy, float *U, int *iterations, double *gap) {
    using namespace lfrv;
    LFRV_API_BEGIN
    if (W < 2 || H < 2 || !gx || !gy || !U || max_iter < 0) return fail(LFRV_E_ARG, "bad arguments");
    if ((size_t)W * H > kStaticPixels)
        return fail(LFRV_E_ARG, "%d x %d pixels exceed LFRV_CG_STATIC_MAX_PIXELS (%zu)", W, H, kStaticPixels);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(LFRV_E_NODEVICE, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(LFRV_E_ARG, "device %d out of range", dev);
    if (persistent_partials() > kStaticBlocks)
        return fail(LFRV_E_ARG, "this device needs more than %d cooperative blocks", kStaticBlocks);
    unsigned char *base = static_scratch(dev);
    float *r = reinterpret_cast<float *>(base);
    float *dA = r + 3 * kStaticPixels, *dB = dA + 3 * kStaticPixels;
    double *partA = reinterpret_cast<double *>(base + kStaticVecBytes), *partB = partA + 4 * kStaticBlocks;
    double *state = partB + 4 * kStaticBlocks;
    unsigned int *bar = reinterpret_cast<unsigned int *>(state + 16);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    e = cudaMemsetAsync(bar, 0, kStaticBarrierBytes, st);  // arrival count and error flag start at zero
    if (e != cudaSuccess) return fail(LFRV_E_CUDA, "clearing the barrier words: %s", cudaGetErrorString(e));
    GridBarrier gb;
    gb.count = bar;
    gb.err = reinterpret_cast<int *>(bar + 4);
    LaunchCounter lc;
    e = launch_cg_persistent(W, H, gx, gy, U, r, dA, dB, partA, partB, gb, max_iter, gap_tol, state, st, lc);
    if (e != cudaSuccess) return fail(LFRV_E_CUDA, "CG launch: %s", cudaGetErrorString(e));
    if (iterations || gap) {
        double hs[16];
        int hb[8];
        e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaMemcpy(hs, state, sizeof(hs), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(hb, bar, sizeof(hb), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return fail(LFRV_E_CUDA, "reading the solver state: %s", cudaGetErrorString(e));
        if (hb[4] != 0) return fail(LFRV_E_TIMEOUT, "a device-side grid barrier gave up waiting");
        if (iterations) *iterations = (int)hs[5];
        if (gap) *gap = hs[4];
    }
    LFRV_API_END
}

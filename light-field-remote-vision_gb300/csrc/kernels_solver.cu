// kernels_solver.cu -- solver-stage kernels of the IBR_color / IBR_gradient path (sm_103a).
//
// Layout in HBM (all planar float32, row-major, top-left origin):
//   per view v (V views, n = w*h source pixels): img[v][3][n], tau[v][2][n] (tau_x, tau_y),
//     dp[v][2][n] (sigma_z * dtau/dz), wgt[v][n] (omega_i), res[v][3][n] (weighted residual scratch)
//   target (N = W*H pixels): U[3][N], P[6][N] duals (px0,py0,px1,py1,px2,py2), F[3][N], g[N], masks.
//
// The reference splats A_i^T r with one launch per host-computed non-overlapping cell segment
// (sources/optimization.cu:882-1025, 1921-1951). Here the scatter becomes a deterministic gather: source
// pixels of all views are bucketed by the anchor of their footprint (counting sort, buckets sorted by
// (view, pixel)), and every target pixel reads the ks x ks anchor buckets that can reach it, recomputing
// the footprint weights from tau instead of storing A (the reference stores ks^2 floats per source pixel).
#include <algorithm>
#include <mutex>
#include <type_traits>

#include <cuda_bf16.h>

#include "device_common.cuh"
#include "kernels.h"

namespace lfrv {

// Storage of the per-view stacks: FP32, or BF16 when the configuration asks for it (loads widen to FP32, and
// every accumulation stays FP32).
__device__ __forceinline__ float ldv(const float *p) { return __ldg(p); }
__device__ __forceinline__ float ldv(const __nv_bfloat16 *p) { return __bfloat162float(__ldg(p)); }
__device__ __forceinline__ void stv(float *p, float v) { *p = v; }
__device__ __forceinline__ void stv(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }


// ====================================================================== inverse footprint map
// Count and fill take kBucketPer source pixels per thread (m, m + blockDim.x, ...): each stage's loads and atomics
// for all of them are issued before any result is used, so their round trips to L2 overlap. Bucket of a
// splatted source pixel: its footprint anchor, offset by ks - 1 (-1: not splatted).
// The count also sets bit v of its bucket's view mask (ceil(V / 64) 64-bit words per bucket, word-major). A bucket
// whose count equals the mask's population holds one entry per view, and the entry of view v goes to slot
// popc(mask & (2^v - 1)): already in (view, pixel) order, with no atomic in the fill and nothing for the sort to
// do. Only buckets with two entries of one view take slots from the cursor (in arrival order) and need the sort.
constexpr int kBucketPer = 4;


__global__ void k_bucket_count(int V, int n, int W, int H, int dsf, int BW, const float *__restrict__ tau,
                               unsigned int *__restrict__ cnt, unsigned long long *__restrict__ mask, int nb) {
    const int v = (int)(blockIdx.x % (unsigned)V);
    const int m0 = (int)(blockIdx.x / (unsigned)V) * blockDim.x * kBucketPer + threadIdx.x;
    const float *tv = tau + (size_t)v * 2 * n;
    float tx[kBucketPer], ty[kBucketPer];
#pragma unroll
    for (int j = 0; j < kBucketPer; ++j) {
        const int m = min(m0 + j * (int)blockDim.x, n - 1);
        tx[j] = tv[m];
        ty[j] = tv[n + m];
    }
#pragma unroll
    for (int j = 0; j < kBucketPer; ++j) {
        const int b = bucket_of(tx[j], ty[j], W, H, dsf, BW);
        if (m0 + j * (int)blockDim.x < n && b >= 0) {
            atomicAdd(&cnt[b], 1u);
            atomicOr(&mask[(size_t)(v >> 6) * nb + b], 1ull << (v & 63));
        }
    }
}

// Views in bucket b's mask (mw words).
__device__ __forceinline__ unsigned int mask_pop(const unsigned long long *mask, int mw, int nb, long long b) {
    unsigned int c = 0;
    for (int w = 0; w < mw; ++w) c += (unsigned int)__popcll(mask[(size_t)w * nb + b]);
    return c;
}

// Whether bucket b's entries must come from the cursor and be sorted (see above).
__device__ __forceinline__ bool bucket_dup(const unsigned int *start, const unsigned long long *mask, int mw, int nb,
                                           long long b) {
    return start[b + 1] - start[b] != mask_pop(mask, mw, nb, b);
}

// MW: the mask words (0: more than two). With their number known, a pixel's words are loaded together with its bucket's
// start, not one after the other (24 views of 512^2: 36 -> 31 us; 80
// views of 1024^2: 653 -> 634, bound by the scattered stores, 32 lines a warp).
template <int MW>
__global__ void __launch_bounds__(256) k_bucket_fill(int V, int n, int W, int H, int dsf, int BW,
                                                     const float *__restrict__ tau,
                                                     const unsigned int *__restrict__ start,
                                                     unsigned int *__restrict__ cursor,
                                                     const unsigned long long *__restrict__ mask, int mw, int nb,
                                                     unsigned int *__restrict__ entries) {
    pdl_wait();
    pdl_trigger();
    const int v = (int)(blockIdx.x % (unsigned)V);
    const int m0 = (int)(blockIdx.x / (unsigned)V) * blockDim.x * kBucketPer + threadIdx.x;
    const float *tv = tau + (size_t)v * 2 * n;
    const int vw = v >> 6;
    const unsigned long long before = (1ull << (v & 63)) - 1ull;  // the views before v in its word
    float tx[kBucketPer], ty[kBucketPer];
#pragma unroll
    for (int j = 0; j < kBucketPer; ++j) {
        const int m = min(m0 + j * (int)blockDim.x, n - 1);
        tx[j] = tv[m];
        ty[j] = tv[n + m];
    }
    int b[kBucketPer];
    unsigned int base[kBucketPer], end[kBucketPer], pop[kBucketPer], below[kBucketPer];
#pragma unroll
    for (int j = 0; j < kBucketPer; ++j) {
        b[j] = m0 + j * (int)blockDim.x < n ? bucket_of(tx[j], ty[j], W, H, dsf, BW) : -1;
        const int q = max(b[j], 0);
        base[j] = start[q];
        end[j] = start[q + 1];
        pop[j] = below[j] = 0;
        auto word = [&](int w) {
            const unsigned long long k = mask[(size_t)w * nb + q];
            pop[j] += (unsigned int)__popcll(k);
            below[j] += w < vw ? (unsigned int)__popcll(k) : (w == vw ? (unsigned int)__popcll(k & before) : 0u);
        };
        if constexpr (MW > 0) {
#pragma unroll
            for (int w = 0; w < MW; ++w) word(w);
        } else {
            for (int w = 0; w < mw; ++w) word(w);
        }
    }
#pragma unroll
    for (int j = 0; j < kBucketPer; ++j) {
        if (b[j] < 0) continue;
        const unsigned int slot = end[j] - base[j] != pop[j] ? atomicAdd(&cursor[b[j]], 1u) : below[j];
        entries[base[j] + slot] = ((unsigned int)v << 24) | (unsigned int)(m0 + j * (int)blockDim.x);
    }
}

// Orders the buckets that hold two entries of one view (the only ones filled out of order) by (view, pixel), so that
// the gathers sum in a fixed order. With dsf 1 they are common (a surface a little farther from the target camera than
// from a view's puts two of its pixels into one bucket) and hold an entry of nearly every view, so eight lanes sort each
// such bucket: its entries in shared memory, every lane counts the entries smaller than its own (they are distinct, so
// the count is the entry's place). One thread's insertion sort per bucket, which stood here before, made this pass 5.2
// of the 6.3 ms of a 384^2 target of 80 views. It remains for buckets beyond kSortCap entries (80 views with four pixels
// each in a bucket fit; 320 entries a bucket are 40 KB of shared memory a block), one such bucket per lane, so that a warp
// sorts 32 of them beside each other and not one per group of eight lanes.
constexpr int kSortBuckets = 256, kSortLanes = 8, kSortCap = 320;

__device__ __forceinline__ void insertion_sort(unsigned int *a, unsigned int s, unsigned int e) {
    for (unsigned int i = s + 1; i < e; ++i) {
        const unsigned int key = a[i];
        unsigned int j = i;
        while (j > s && a[j - 1] > key) {
            a[j] = a[j - 1];
            --j;
        }
        a[j] = key;
    }
}

__global__ void __launch_bounds__(kSortBuckets) k_bucket_sort(int nb, const unsigned int *__restrict__ start,
                                                              const unsigned long long *__restrict__ mask, int mw,
                                                              unsigned int *entries) {
    pdl_wait();
    __shared__ __align__(16) unsigned int buf[kSortBuckets / kSortLanes][kSortCap];
    const int lane = threadIdx.x & 31, sub = lane % kSortLanes, b = blockIdx.x * kSortBuckets + (int)threadIdx.x;
    unsigned int *own = buf[threadIdx.x / kSortLanes];
    const bool dup = b < nb && bucket_dup(start, mask, mw, nb, b);
    const unsigned int s0 = dup ? start[b] : 0u, n0 = dup ? start[b + 1] - s0 : 0u;
    if (n0 > (unsigned int)kSortCap) insertion_sort(entries, s0, s0 + n0);
    unsigned int todo = __ballot_sync(0xffffffffu, dup && n0 <= (unsigned int)kSortCap);
    while (todo) {
        // the next buckets, one per group of lanes
        unsigned int rest = todo;
        for (int g = lane / kSortLanes; g > 0; --g) rest &= rest - 1;
        const int l = rest ? __ffs(rest) - 1 : 0;
        const unsigned int s = __shfl_sync(0xffffffffu, s0, l), have = __shfl_sync(0xffffffffu, n0, l);
        const unsigned int m = rest ? have : 0u;
        for (int g = 0; g < 32 / kSortLanes; ++g) todo &= todo - 1;
        const unsigned int padded = (m + 3u) & ~3u;  // the last group of four is filled with the largest key
        for (unsigned int i = sub; i < padded; i += kSortLanes) own[i] = i < m ? entries[s + i] : 0xFFFFFFFFu;
        __syncwarp();
        for (unsigned int i = sub; i < m; i += kSortLanes) {
            const unsigned int key = own[i];
            unsigned int rank = 0;
            for (unsigned int q = 0; q < padded; q += 4) {
                const uint4 k = *reinterpret_cast<const uint4 *>(own + q);
                rank += (k.x < key) + (k.y < key) + (k.z < key) + (k.w < key);
            }
            entries[s + rank] = key;
        }
        __syncwarp();
    }
}

// Exclusive scan of unsigned counts: each block scans kScanPer * kScanBlock counts (kScanPer per thread: a
// thread's own prefix, then warp shuffles over the thread totals and one warp over the warp totals) and writes its
// total; k_scan_finish then adds to every block the totals of the blocks before it. Integer sums: the result does
// not depend on the order.
constexpr int kScanBlock = 1024, kScanPer = 4, kScanSpan = kScanBlock * kScanPer;

__global__ void __launch_bounds__(kScanBlock) k_scan_blocks(int nb, const unsigned int *__restrict__ in,
                                                            unsigned int *__restrict__ out,
                                                            unsigned int *__restrict__ block_sums) {
    pdl_wait();
    pdl_trigger();
    __shared__ unsigned int warp_tot[kScanBlock / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i0 = blockIdx.x * kScanSpan + threadIdx.x * kScanPer;
    unsigned int v[kScanPer];
#pragma unroll
    for (int j = 0; j < kScanPer; ++j) v[j] = (i0 + j < nb) ? in[i0 + j] : 0u;
    unsigned int t = 0;
#pragma unroll
    for (int j = 0; j < kScanPer; ++j) t += v[j];
    unsigned int incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        unsigned int w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        warp_tot[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    unsigned int run = (wid > 0 ? warp_tot[wid - 1] : 0u) + incl - t;  // exclusive prefix of this thread
#pragma unroll
    for (int j = 0; j < kScanPer; ++j) {
        if (i0 + j < nb) out[i0 + j] = run;
        run += v[j];
    }
    if (threadIdx.x == kScanBlock - 1) block_sums[blockIdx.x] = warp_tot[31];
}

// Adds to block b's exclusive scan the sum of the totals of blocks 0 .. b - 1; out[nb] = the grand total.
// zero (optional): the scanned counts, cleared here for their next use as cursors (k_scan_blocks has read them)
__global__ void __launch_bounds__(kScanBlock) k_scan_finish(int nb, unsigned int *__restrict__ out,
                                                            const unsigned int *__restrict__ block_sums,
                                                            unsigned int *__restrict__ zero) {
    pdl_wait();
    pdl_trigger();
    __shared__ unsigned int red[kScanBlock / 32];
    unsigned int s = 0;
    for (int j = threadIdx.x; j < (int)blockIdx.x; j += kScanBlock) s += block_sums[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned int t = (threadIdx.x < kScanBlock / 32) ? red[threadIdx.x] : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) red[0] = t;
    }
    __syncthreads();
    const unsigned int off = red[0];
    const int i0 = blockIdx.x * kScanSpan + threadIdx.x * kScanPer;
#pragma unroll
    for (int j = 0; j < kScanPer; ++j)
        if (i0 + j < nb) {
            out[i0 + j] += off;
            if (zero) zero[i0 + j] = 0u;
        }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[nb] = off + block_sums[blockIdx.x];
}

// ====================================================================== per-source gathers (v = A u)
// Weighted residual e = w * (A_i U - v_i) over the gather set, and the intensity energy
// sum sigma^2 w (A_i U - v_i)^2 (vtv_sr_dataterm_intensities sources/optimization.cu:1871-1903 and
// coco_vtv_sr_primal_energy_unstructured :1560-1608). Outside the gather set A_i U = 0.
// splat_set: the residual over the splat set instead, zero elsewhere (the corrected IBR_color objective, whose
// gradient splats over the same set).
// ENERGY: the energy's FP64 terms and their block sum, for the callers that read it (half of the kernel's time at 256^2:
// some ten FP64 operations per pixel on a pipe that takes 16 cycles a warp).
template <int KS, bool ENERGY>
__global__ void __launch_bounds__(256) k_residual(int V, int n, int W, int H, int dsf, const float *__restrict__ U,
                                                  const float *__restrict__ img, const float *__restrict__ tau,
                                                  const float *__restrict__ wgt, float s2,
                                                  float *__restrict__ res, double *__restrict__ partial,
                                                  int splat_set) {
    __shared__ double red[8];
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    const size_t N = (size_t)W * H;
    double e = 0.0;
    if (m < n) {
        const float tx = tau[(size_t)v * 2 * n + m], ty = tau[(size_t)v * 2 * n + n + m];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        if (in_gather(tx, ty, W, H)) {
            Footprint fp;
            footprint<KS>(tx, ty, dsf, W, H, fp);
#pragma unroll
            for (int j = 0; j < KS; ++j)
#pragma unroll
                for (int i = 0; i < KS; ++i) {
                    const int x = fp.x0 + j, y = fp.y0 + i;
                    if (0 <= x && x <= W - 1 && 0 <= y && y <= H - 1) {
                        const float A = fp.A[KS * i + j];
                        const size_t o = (size_t)y * W + x;
                        a0 += A * __ldg(U + o);
                        a1 += A * __ldg(U + N + o);
                        a2 += A * __ldg(U + 2 * N + o);
                    }
                }
        }
        const float *iv = img + (size_t)v * 3 * n;
        const float w = (splat_set && !in_splat(tx, ty, W, H)) ? 0.f : wgt[(size_t)v * n + m];
        const float d0 = a0 - iv[m], d1 = a1 - iv[n + m], d2 = a2 - iv[2 * n + m];
        float *rv = res + (size_t)v * 3 * n;
        rv[m] = d0 * w;
        rv[n + m] = d1 * w;
        rv[2 * n + m] = d2 * w;
        if (ENERGY) e = (double)s2 * (double)w * ((double)d0 * d0 + (double)d1 * d1 + (double)d2 * d2);
    }
    if (!ENERGY) return;
    const double s = block_sum<256>(e, red);
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

// Angular and deformation weights of every source pixel (coco_vtv_sr_compute_weights_unstructured,
// sources/optimization.cu:1094-1163; vtv_sr_angular_weights_device and vtv_sr_gold_deform_weights_device,
// vtv_sr_kernels_unstructured.cu:174-266): w = 1/(sg^2 + sigma^2) * deform with sg = clamp(A_i grad) . dpart.
// GATHER = false: the target gradient is identically zero (gx == nullptr), so the gather through A is skipped
// at compile time and the kernel keeps few registers.
template <int KS, typename TW, bool GATHER>
__global__ void __launch_bounds__(256, GATHER ? 1 : 8) k_weights(int V, int n, int w, int h, int W, int H, int dsf,
                                                 const float *__restrict__ gx, const float *__restrict__ gy,
                                                 const float *__restrict__ tau, const float *__restrict__ dp,
                                                 float sigma, float thr, TW *__restrict__ wgt) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    if (m >= n) return;
    const float *tx = tau + (size_t)v * 2 * n, *ty = tx + n;
    // every load the pixel can need, issued together (neighbour indices clamped to the view; the clamped values
    // are read only where the neighbour exists)
    int mx, my;
    pixel_of(m, w, n, __frcp_rn((float)w), mx, my);
    const int ml = mx > 0 ? m - 1 : m, mr = mx < w - 1 ? m + 1 : m;
    const int mu = my > 0 ? m - w : m, md = my < h - 1 ? m + w : m;
    const float txm = __ldg(tx + m), tym = __ldg(ty + m);
    const float txl = __ldg(tx + ml), tyl = __ldg(ty + ml), txr = __ldg(tx + mr), tyr = __ldg(ty + mr);
    const float txu = __ldg(tx + mu), tyu = __ldg(ty + mu), txd = __ldg(tx + md), tyd = __ldg(ty + md);
    // (no dp: dtau/dz taken as 0, for callers whose gathered gradient is 0 anyway)
    const float dpx = dp ? __ldg(dp + (size_t)v * 2 * n + m) : 0.f;
    const float dpy = dp ? __ldg(dp + (size_t)v * 2 * n + n + m) : 0.f;
    float ax = 0.f, ay = 0.f;
    if (GATHER && in_gather(txm, tym, W, H)) {
        Footprint fp;
        footprint<KS>(txm, tym, dsf, W, H, fp);
#pragma unroll
        for (int j = 0; j < KS; ++j)
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                const int x = fp.x0 + j, y = fp.y0 + i;
                if (0 <= x && x <= W - 1 && 0 <= y && y <= H - 1) {
                    const float A = fp.A[KS * i + j];
                    const size_t o = (size_t)y * W + x;
                    ax += A * __ldg(gx + o);
                    ay += A * __ldg(gy + o);
                }
            }
    }
    // angular weight
    const float norm = sqrtf(ax * ax + ay * ay);
    if (norm > thr) {
        ax = ax / norm * thr;
        ay = ay / norm * thr;
    }
    float sg = ax * dpx + ay * dpy;
    if (sg > 0.5f) sg = 0.5f;
    const float ang = 1.0f / (sg * sg + sigma * sigma);
    // deformation weight
    auto out = [&](float x, float y) { return x < 0.f || x > (float)W || y < 0.f || y > (float)H; };
    float def;
    if (out(txm, tym)) def = 0.0f;
    else if (mx == 0 || my == 0 || mx == w - 1 || my == h - 1) def = 1.0f;
    else if (out(txl, tyl) || out(txr, tyr) || out(txu, tyu) || out(txd, tyd)) def = 1.0f;
    else {
        const float Dxx = 0.5f * (txr - txl);
        const float Dyx = 0.5f * (tyr - tyl);
        const float Dxy = 0.5f * (txd - txu);
        const float Dyy = 0.5f * (tyd - tyu);
        const float N = fabsf(Dxx * Dyy - Dxy * Dyx);
        def = (N > 1.0f) ? 1.0f / N : 1.0f;
    }
    stv(wgt + (size_t)v * n + m, ang * def);
}

// k_weights without a target gradient (GATHER = false) and without dtau/dz, four pixels of a row per thread: the angular
// weight is then one constant (ang = 1 / sigma^2), and the four pixels share their neighbours' loads (six 16-byte loads
// and four words instead of 40 words). For view widths of a multiple of four, so that a thread's pixels share a row and
// every 16-byte load is aligned. 80 views of 1024^2: 468 -> 230 us, 4.4 TB/s of its
// 12 B a pixel.
template <typename TW>
__global__ void __launch_bounds__(256) k_weights_flat(int n, int w, int h, int W, int H, const float *__restrict__ tau,
                                                      float ang, TW *__restrict__ wgt) {
    const int m = (blockIdx.x * blockDim.x + threadIdx.x) * 4, v = blockIdx.y;
    if (m >= n) return;
    const float *tx = tau + (size_t)v * 2 * n, *ty = tx + n;
    int mx, my;
    pixel_of(m, w, n, __frcp_rn((float)w), mx, my);
    const int mu = my > 0 ? m - w : m, md = my < h - 1 ? m + w : m;
    auto ld4 = [](const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); };
    const float4 xc = ld4(tx + m), yc = ld4(ty + m), xu = ld4(tx + mu), yu = ld4(ty + mu), xd = ld4(tx + md),
                 yd = ld4(ty + md);
    const int ml = mx > 0 ? m - 1 : m, mr = mx + 4 < w ? m + 4 : m + 3;
    const float X[6] = {__ldg(tx + ml), xc.x, xc.y, xc.z, xc.w, __ldg(tx + mr)};
    const float Y[6] = {__ldg(ty + ml), yc.x, yc.y, yc.z, yc.w, __ldg(ty + mr)};
    const float XU[4] = {xu.x, xu.y, xu.z, xu.w}, YU[4] = {yu.x, yu.y, yu.z, yu.w};
    const float XD[4] = {xd.x, xd.y, xd.z, xd.w}, YD[4] = {yd.x, yd.y, yd.z, yd.w};
    auto out = [&](float x, float y) { return x < 0.f || x > (float)W || y < 0.f || y > (float)H; };
    bool oc[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) oc[i] = out(X[i], Y[i]);
    const bool row = my == 0 || my == h - 1;
    float r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float def = 1.0f;
        if (oc[i + 1]) def = 0.0f;
        else if (!(row || mx + i == 0 || mx + i == w - 1) &&
                 !(oc[i] || oc[i + 2] || out(XU[i], YU[i]) || out(XD[i], YD[i]))) {
            const float Dxx = 0.5f * (X[i + 2] - X[i]);
            const float Dyx = 0.5f * (Y[i + 2] - Y[i]);
            const float Dxy = 0.5f * (XD[i] - XU[i]);
            const float Dyy = 0.5f * (YD[i] - YU[i]);
            const float N = fabsf(Dxx * Dyy - Dxy * Dyx);
            def = (N > 1.0f) ? 1.0f / N : 1.0f;
        }
        r[i] = ang * def;
    }
    TW *o = wgt + (size_t)v * n + m;
    if constexpr (sizeof(TW) == 4) {
        *reinterpret_cast<float4 *>(o) = make_float4(r[0], r[1], r[2], r[3]);
    } else {
        __nv_bfloat162 b[2] = {__floats2bfloat162_rn(r[0], r[1]), __floats2bfloat162_rn(r[2], r[3])};
        *reinterpret_cast<uint2 *>(o) = *reinterpret_cast<const uint2 *>(b);
    }
}

// ====================================================================== A^T gathers (per target pixel)
// (SplatSrc and splat_accumulate live in device_common.cuh)

// Coverage and visibility (coco_vtv_setup_visibility_mask sources/optimization.cu:33-135):
// cov = sum A, vis = cov >= 1.
template <int KS>
__global__ void k_coverage(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                           const unsigned int *__restrict__ entries, const float *__restrict__ tau,
                           float *__restrict__ cov, uint8_t *__restrict__ vis) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    SplatSrc src{{nullptr, nullptr, nullptr}, {0, 0, 0}, nullptr};
    float acc[3], norm;
    splat_accumulate<KS, 0>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x;
    cov[o] = norm;
    vis[o] = (norm < 1.0f) ? 0 : 1;
}

// Visibility of IBR_gradient (setup_target_visibility, sources/gradientIBR.cu:40-83): some splatted tap
// with a non-zero raw overlap.
template <int KS>
__global__ void k_vis_any(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                          const unsigned int *__restrict__ entries, const float *__restrict__ tau,
                          uint8_t *__restrict__ vis) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    bool any = false;
#pragma unroll
    for (int i = 0; i < KS; ++i)
#pragma unroll
        for (int j = 0; j < KS; ++j) {
            const int ax = x - j, ay = y - i;
            const size_t b = (size_t)(ay + KS - 1) * BW + (ax + KS - 1);
            const unsigned int s = start[b], e = start[b + 1];
            for (unsigned int k = s; k < e && !any; ++k) {
                const unsigned int ent = entries[k];
                const int v = (int)(ent >> 24), m = (int)(ent & 0xFFFFFFu);
                const float tx = tau[(size_t)v * 2 * n + m], ty = tau[(size_t)v * 2 * n + n + m];
                if (footprint_raw<KS>(tx, ty, dsf, j, i, ax, ay) != 0.0f) any = true;
            }
        }
    vis[(size_t)y * W + x] = any ? 1 : 0;
}

// IBR_gradient set-up in one traversal of the inverse map (per target pixel):
//   visibility   setup_target_visibility (sources/gradientIBR.cu:40-83): some splatted raw overlap != 0;
//   weighted average of compute_initial_image (:724-808): U = sum w A v / sum w A;
//   gradient splat of init_u_gradient (:833-920): (gx, gy, mask) = sum A (Sobel_x, Sobel_y, w) / sum A,
//   mask scaled by sigma^2.
// img: per view [3][n]; vgrad: per view [2][n] (Sobel of the view luminance); wgt: per view [n].
struct SetupAcc {
    float u0 = 0.f, u1 = 0.f, u2 = 0.f, wn = 0.f;  // weighted average
    float g0 = 0.f, g1 = 0.f, g2 = 0.f, nrm = 0.f;  // gradient splat
    bool any = false;
    __device__ __forceinline__ void add(float A, float raw, float w, float c0, float c1, float c2, float s0, float s1) {
        any |= (raw != 0.0f);
        const float wA = w * A;
        wn += wA;
        u0 += wA * c0;
        u1 += wA * c1;
        u2 += wA * c2;
        nrm += A;
        g0 += A * s0;
        g1 += A * s1;
        g2 += A * w;
    }
    __device__ __forceinline__ void store(size_t o, size_t N, float s2, uint8_t *vis, float *U, float *gx, float *gy,
                                          float *mask) {
        vis[o] = any ? 1 : 0;
        if (wn != 0.f) {
            u0 /= wn;
            u1 /= wn;
            u2 /= wn;
        }
        U[o] = u0;
        U[N + o] = u1;
        U[2 * N + o] = u2;
        if (nrm != 0.f) {
            g0 /= nrm;
            g1 /= nrm;
            g2 /= nrm;
        }
        gx[o] = g0;
        gy[o] = g1;
        mask[o] = g2 * s2;
    }
};

// The set-up of one target pixel reading every entry straight from global memory.
template <int KS, typename TS>
__device__ __forceinline__ void gradient_setup_global(int x, int y, int W, int H, int n, int dsf, int BW,
                                                      const unsigned int *__restrict__ start,
                                                      const unsigned int *__restrict__ entries,
                                                      const float *__restrict__ tau, const TS *__restrict__ img,
                                                      const TS *__restrict__ vgrad, const TS *__restrict__ wgt,
                                                      SetupAcc &acc) {
#pragma unroll
    for (int i = 0; i < KS; ++i) {
#pragma unroll
        for (int j = 0; j < KS; ++j) {
            const int ax = x - j, ay = y - i;
            const size_t b = (size_t)(ay + KS - 1) * BW + (ax + KS - 1);
            const unsigned int s = __ldg(start + b), e = __ldg(start + b + 1);
            for (unsigned int k = s; k < e; ++k) {
                const unsigned int ent = __ldg(entries + k);
                const int v = (int)(ent >> 24), m = (int)(ent & 0xFFFFFFu);
                const float tx = __ldg(tau + (size_t)v * 2 * n + m), ty = __ldg(tau + (size_t)v * 2 * n + n + m);
                float raw;
                const float A = footprint_tap<KS>(tx, ty, dsf, W, H, ax, ay, j, i, raw);
                const TS *iv = img + (size_t)v * 3 * n;
                const TS *gv = vgrad + (size_t)v * 2 * n;
                acc.add(A, raw, ldv(wgt + (size_t)v * n + m), ldv(iv + m), ldv(iv + n + m), ldv(iv + 2 * n + m),
                        ldv(gv + m), ldv(gv + n + m));
            }
        }
    }
}

// Anchor-row form (KS <= 3). The entries of one anchor bucket reach a KS x KS block of target pixels, so
// instead of every target pixel re-reading the entries of its KS^2 buckets, a lane reads each entry of its
// buckets once and accumulates its taps in registers.
// A source pixel's overlaps along one axis are (1 - a, a) for KS 2 and (1 - a, 1, a) for KS 3, so two sums per axis
// carry all of them: Q0 = sum (1 - a) v, Q1 = sum a v, and the middle tap is Q0 + Q1 (terms of one sign, nothing
// cancels). Four sums per field instead of KS^2: 28 accumulators and 28 multiply-adds per entry, not 63 and 72.
// A warp owns 64 consecutive anchors of one anchor row, starting at an even column: lane l takes anchor 2l in
// pass 0 and anchor 2l + 1 in pass 1, and owns pixel columns 2l and 2l + 1. With dsf 2 most source pixels of a
// box-decimated view land on even anchors, so one pass per parity makes a warp wait for its longest even bucket
// plus its longest odd bucket, not twice the longest of both. Pixel x of tap row i sums tap j of anchor x - j:
//   column 2l:      (P0[0] of 2l + P0[2] of 2l - 2) + P1[1] of 2l - 1
//   column 2l + 1:   P0[1] of 2l + (P1[0] of 2l + 1 + P1[2] of 2l - 1)
// (P0 / P1: the pass-0 / pass-1 tap sums; the left terms come from lane l - 1 by shuffle). The block then adds
// the KS tap rows of each pixel from shared memory. Every sum has a fixed order, so results are deterministic.
// Lane 0's columns lack their left anchors, so a warp outputs 62 pixels. The footprint norm is the product of
// the row and column overlap sums (the KS^2 taps are an outer product). Fields: 0 w A, 1-3 w A v, 4 A, 5-6 A Sobel; a
// pixel is visible when its sum of A is not 0 (no A is negative). The mask sum (A w) is field 0.
// RPW: anchor rows per warp; one where two would leave SMs without a block (the rows shared between blocks cost less
// than that). The gathers in flight live in L1, so shared memory is kept small (with 73 KB a block, three blocks took
// 2.2 ms where two took 1.0 at 2048^2). Measured, two rows and three blocks per SM: 24 views of 512^2 -> 1024^2 119 ->
// 80 us, 80 views of 1024^2 -> 2048^2 1278 -> 977 us (3.1 TB/s of compulsory reads); one row and two blocks: 80 BF16
// views of 384^2, dsf 1, 373 -> 223 us. Bound by the latency of the gathers.
constexpr int kGrWarps = 8;
constexpr int kGrTXO = 62;  // output pixels per warp row
constexpr int kGrNF = 7;    // fields per tap-row partial

// Sums a pixel row is kept in until they are added, one per warp that contributes: its tap rows come from KS
// consecutive anchor rows, so from KS warps at one row each and from two (its own and the one before) at two.
template <int KS, int RPW>
__host__ __device__ constexpr int gradient_rows_slots() {
    return RPW == 1 ? KS : 2;
}
template <int KS, int RPW>
constexpr size_t gradient_rows_smem() {
    return sizeof(float) * (kGrWarps * RPW - (KS - 1)) * gradient_rows_slots<KS, RPW>() * kGrNF * kGrTXO;
}

template <int KS, typename TS, int RPW>
__global__ void __launch_bounds__(kGrWarps * 32, RPW == 2 ? 3 : 2) k_gradient_setup_rows(int W, int H, int n, int dsf, int BW,
                                                                       const unsigned int *__restrict__ start,
                                                                       const unsigned int *__restrict__ entries,
                                                                       const float *__restrict__ tau,
                                                                       const TS *__restrict__ img,
                                                                       const TS *__restrict__ vgrad,
                                                                       const TS *__restrict__ wgt, float s2,
                                                                       uint8_t *__restrict__ vis,
                                                                       float *__restrict__ U, float *__restrict__ gx,
                                                                       float *__restrict__ gy,
                                                                       float *__restrict__ mask) {
    constexpr int TY = kGrWarps * RPW - (KS - 1);  // output pixel rows per block
    constexpr int NF = kGrNF, NS = gradient_rows_slots<KS, RPW>();
    extern __shared__ float gr_part[];  // [TY][NS][NF][kGrTXO]: (pixel row, contributing warp, field, pixel)
    pdl_trigger();                      // the hole list, launched next, waits for this grid's completion
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = blockIdx.x * kGrTXO, y0 = blockIdx.y * TY;
    const int BH = H + KS - 1;
    const int lx = 2 * lane - 2;  // this lane's first pixel column inside the tile
    // warp w takes the consecutive anchor rows RPW w, RPW w + 1, ...: with two, one of each parity (with dsf = 2 the
    // populated anchors mostly sit on even rows, so rows w and w + 8 would leave half the warps idle)
#pragma unroll 1
    for (int q = 0; q < RPW; ++q) {
        const int rr = RPW * warp + q;
        const int ay = y0 - (KS - 1) + rr, by = ay + KS - 1;
        // overlaps of the in-image taps: the first and last tap count when inside, the middle one always is unless
        // the whole row lies outside
        const bool y_first = 0 <= ay && ay <= H - 1, y_last = 0 <= ay + KS - 1 && ay + KS - 1 <= H - 1;
        const float y_mid = (KS == 3 && 0 <= ay + 1 && ay + 1 <= H - 1) ? 1.f : 0.f;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            const int ax = x0 - 2 + 2 * lane + pass, bx = ax + KS - 1;
            const bool x_first = 0 <= ax && ax <= W - 1, x_last = 0 <= ax + KS - 1 && ax + KS - 1 <= W - 1;
            const float x_mid = (KS == 3 && 0 <= ax + 1 && ax + 1 <= W - 1) ? 1.f : 0.f;
            float Q[2][2][NF];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int f = 0; f < NF; ++f) Q[i][j][f] = 0.f;
            if (bx >= 0 && bx < BW && by < BH) {
                const size_t b = (size_t)by * BW + bx;
                const unsigned int s = __ldg(start + b), e = __ldg(start + b + 1);
                struct Src {
                    float tx, ty, w, c0, c1, c2, s0, s1;
                };
                auto fetch = [&](unsigned int ent, Src &d) {
                    const size_t vn = (size_t)(ent >> 24) * (size_t)n, m = ent & 0xFFFFFFu;
                    const float *tv = tau + 2 * vn + m;
                    const TS *iv = img + 3 * vn + m, *gv = vgrad + 2 * vn + m;
                    d.tx = __ldg(tv);
                    d.ty = __ldg(tv + n);
                    d.w = ldv(wgt + vn + m);
                    d.c0 = ldv(iv);
                    d.c1 = ldv(iv + n);
                    d.c2 = ldv(iv + 2 * (size_t)n);
                    d.s0 = ldv(gv);
                    d.s1 = ldv(gv + n);
                };
                auto add = [&](const Src &d) {
                    const float px = d.tx - 0.5f, py = d.ty - 0.5f;
                    const float dx[2] = {fp_overlap(0, KS, ax, px, dsf), fp_overlap(KS - 1, KS, ax + KS - 1, px, dsf)};
                    const float dy[2] = {fp_overlap(0, KS, ay, py, dsf), fp_overlap(KS - 1, KS, ay + KS - 1, py, dsf)};
                    const float sx = (x_first ? dx[0] : 0.f) + x_mid + (x_last ? dx[1] : 0.f);
                    const float sy = (y_first ? dy[0] : 0.f) + y_mid + (y_last ? dy[1] : 0.f);
                    // one reciprocal per entry; A = (dx * (1 / norm)) * dy is within a few ulps of dx dy / norm
                    const float norm = __fmul_rn(sx, sy);
                    const float inv = (norm != 0.0f) ? __frcp_rn(norm) : 1.0f;
                    const float v[NF] = {d.w, d.w * d.c0, d.w * d.c1, d.w * d.c2, 1.f, d.s0, d.s1};
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float yi = __fmul_rn(dy[i], inv);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const float A = __fmul_rn(dx[j], yi);
#pragma unroll
                            for (int f = 0; f < NF; ++f) Q[i][j][f] = f == 4 ? Q[i][j][f] + A : fmaf(A, v[f], Q[i][j][f]);
                        }
                    }
                };
                // two entries in flight while two are added, and the indices of the two after those
                Src a = {}, c = {};
                unsigned int ea = 0, ec = 0;
                if (s < e) fetch(__ldg(entries + s), a);
                if (s + 1 < e) fetch(__ldg(entries + s + 1), c);
                if (s + 2 < e) ea = __ldg(entries + s + 2);
                if (s + 3 < e) ec = __ldg(entries + s + 3);
                for (unsigned int k = s; k < e; k += 2) {
                    add(a);
                    if (k + 2 < e) fetch(ea, a);
                    if (k + 4 < e) ea = __ldg(entries + k + 4);
                    if (k + 1 < e) add(c);
                    if (k + 3 < e) fetch(ec, c);
                    if (k + 5 < e) ec = __ldg(entries + k + 5);
                }
            }
            // tap rows of this pass into shared memory: the warp's first contribution to a slot stores, the others add
            // (same lane, same slots)
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                const int py = ay + i - y0;  // output pixel row inside the tile
                const bool store = lane >= 1 && py >= 0 && py < TY;
                const bool first = pass == 0 && (RPW == 1 || q == 0 || i == KS - 1);
                float *row = gr_part + (size_t)(py * NS + (q + i) / RPW) * NF * kGrTXO + lx;
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    // taps 0 and KS - 1 of tap row i
                    const float t0 = i == 0 ? Q[0][0][f] : (i == KS - 1 ? Q[1][0][f] : Q[0][0][f] + Q[1][0][f]);
                    const float t1 = i == 0 ? Q[0][1][f] : (i == KS - 1 ? Q[1][1][f] : Q[0][1][f] + Q[1][1][f]);
                    float c0, c1;
                    const float last = __shfl_up_sync(0xffffffffu, t1, 1);  // the last tap of lane l - 1
                    if (KS == 3) {
                        const float mid = t0 + t1;
                        if (pass == 0) {
                            c0 = t0 + last;
                            c1 = mid;
                        } else {
                            c0 = __shfl_up_sync(0xffffffffu, mid, 1);
                            c1 = t0 + last;
                        }
                    } else if (pass == 0) {
                        c0 = t0;
                        c1 = t1;
                    } else {
                        c0 = last;
                        c1 = t0;
                    }
                    if (store) {
                        float2 *d = reinterpret_cast<float2 *>(row + f * kGrTXO);
                        if (first) {
                            *d = make_float2(c0, c1);
                        } else {
                            const float2 o = *d;
                            *d = make_float2(o.x + c0, o.y + c1);
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    // add the slots of every pixel in order and normalise (as SetupAcc::store)
    const size_t N = (size_t)W * H;
    for (int p = threadIdx.x; p < TY * kGrTXO; p += kGrWarps * 32) {
        const int px = p % kGrTXO, ly = p / kGrTXO, x = x0 + px, y = y0 + ly;
        if (x >= W || y >= H) continue;
        SetupAcc acc;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            // (KS 2, two rows per warp: a warp's second row gets both tap rows from that warp)
            if (KS == 2 && RPW == 2 && i == 1 && ((ly + 1) & 1)) continue;
            const float *c = gr_part + (size_t)(ly * NS + i) * NF * kGrTXO + px;
            acc.wn += c[0 * kGrTXO];
            acc.u0 += c[1 * kGrTXO];
            acc.u1 += c[2 * kGrTXO];
            acc.u2 += c[3 * kGrTXO];
            acc.nrm += c[4 * kGrTXO];
            acc.g0 += c[5 * kGrTXO];
            acc.g1 += c[6 * kGrTXO];
        }
        acc.g2 = acc.wn;
        acc.any = acc.nrm != 0.f;
        acc.store((size_t)y * W + x, N, s2, vis, U, gx, gy, mask);
    }
}

// Per-pixel form for KS > 3 (too many register partials for the anchor-row form).
template <int KS, typename TS>
__global__ void __launch_bounds__(256) k_gradient_setup_px(int W, int H, int n, int dsf, int BW,
                                                           const unsigned int *__restrict__ start,
                                                           const unsigned int *__restrict__ entries,
                                                           const float *__restrict__ tau, const TS *__restrict__ img,
                                                           const TS *__restrict__ vgrad,
                                                           const TS *__restrict__ wgt, float s2,
                                                           uint8_t *__restrict__ vis, float *__restrict__ U,
                                                           float *__restrict__ gx, float *__restrict__ gy,
                                                           float *__restrict__ mask) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    SetupAcc acc;
    gradient_setup_global<KS, TS>(x, y, W, H, n, dsf, BW, start, entries, tau, img, vgrad, wgt, acc);
    acc.store((size_t)y * W + x, (size_t)W * H, s2, vis, U, gx, gy, mask);
}

// Weighted average (coco_vtv_sr_compute_initial_image sources/optimization.cu:1300-1344):
// U = sum w A v / sum w A where the weight sum is non-zero.
template <int KS>
__global__ void k_initial_image(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                                const unsigned int *__restrict__ entries, const float *__restrict__ tau,
                                SplatSrc src, float *__restrict__ U, float *__restrict__ norm_out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    float acc[3], norm;
    splat_accumulate<KS, 3>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x, N = (size_t)W * H;
#pragma unroll
    for (int c = 0; c < 3; ++c) U[c * N + o] = (norm != 0.f) ? acc[c] / norm : acc[c];
    if (norm_out) norm_out[o] = norm;
}

// Input of the learned warm start, NHWC BF16 with kLearnChannels (48) channels per target pixel:
// [0..2] the anchor u0 (hole-filled weighted average), [3] gx, [4] gy (the splatted luminance gradient, one plane
// each; zero in the last column / row, which the normal equations never read, and clamped to [-1, 1], the range
// of finite differences of [0, 1] images), [5] visibility, [6 + 3 v .. 8 + 3 v] view v splatted alone
// (sum A w v / sum A w over its own footprints), [30 + v] view v's share of the total splat weight, for the first
// kLearnViews views; [38..40] the CG's initial residual at u0 per channel, r0 = grad^T g + Delta u0 (FP32, the
// operator's boundary rules, clamped to [-4, 4]); [41..47] zero. Per-view accumulators live in shared memory (one
// column per thread), so the view index of an entry needs no register indexing.
// Each entry's tap is computed alone, not through footprint_tap's KS^2 products: the footprint is an outer product,
// so its norm is the product of the in-image row and column overlap sums, and the tap (j, i) is
// dx_j * (dy_i / norm) with one reciprocal (within a few ulps of footprint_tap's quotient, as in the set-up's
// anchor-row form). The gather is a chain of dependent loads (bucket bounds, entry, the view's data), so all KS x KS
// buckets' bounds and first entries are loaded up front (a row's KS buckets are contiguous) and each bucket's loop
// keeps the entry two ahead and the next entry's data in flight.
template <int KS, typename TS>
__global__ void __launch_bounds__(256, 4) k_learn_input(int W, int H, int n, int dsf, int BW,
                                                     const unsigned int *__restrict__ start,
                                                     const unsigned int *__restrict__ entries,
                                                     const float *__restrict__ tau, const TS *__restrict__ img,
                                                     const TS *__restrict__ wgt, const float *__restrict__ U,
                                                     const float *__restrict__ gx, const float *__restrict__ gy,
                                                     const uint8_t *__restrict__ vis, __nv_bfloat16 *__restrict__ out) {
    __shared__ float acc[kLearnViews * 4][256];
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    // a block covers 64 x 4 pixels; warp w takes the columns of parity w & 1 of row w >> 1, so that the lanes of a
    // warp scan buckets of one anchor parity (with dsf 2 most entries sit on even anchors)
    const int x = blockIdx.x * 64 + 2 * threadIdx.x + (threadIdx.y & 1), y = blockIdx.y * 4 + (threadIdx.y >> 1);
#pragma unroll
    for (int i = 0; i < kLearnViews * 4; ++i) acc[i][t] = 0.f;
    if (x >= W || y >= H) return;
    // row i's anchors x - KS + 1 .. x are buckets r .. r + KS - 1 of that row: column j's bucket is r + KS - 1 - j
    unsigned int bs[KS][KS + 1];
#pragma unroll
    for (int i = 0; i < KS; ++i) {
        const size_t r = (size_t)(y - i + KS - 1) * BW + x;
#pragma unroll
        for (int q = 0; q <= KS; ++q) bs[i][q] = __ldg(start + r + q);
    }
    constexpr unsigned int kNone = 0xFFFFFFFFu;  // view 255: past the first views
    auto ok = [](unsigned int ent) { return (int)(ent >> 24) < kLearnViews; };
    // every bucket's first entry, loaded together
    unsigned int first[KS][KS];
#pragma unroll
    for (int i = 0; i < KS; ++i)
#pragma unroll
        for (int j = 0; j < KS; ++j)
            first[i][j] = bs[i][KS - 1 - j] < bs[i][KS - j] ? __ldg(entries + bs[i][KS - 1 - j]) : kNone;
    struct Src {
        float px, py, w, c0, c1, c2;
    };
    auto fetch = [&](unsigned int ent) {
        const size_t v = ent >> 24, m = ent & 0xFFFFFFu;
        Src d;
        d.px = __ldg(tau + v * 2 * n + m) - 0.5f;
        d.py = __ldg(tau + v * 2 * n + n + m) - 0.5f;
        d.w = ldv(wgt + v * n + m);
        d.c0 = ldv(img + (v * 3 + 0) * n + m);
        d.c1 = ldv(img + (v * 3 + 1) * n + m);
        d.c2 = ldv(img + (v * 3 + 2) * n + m);
        return d;
    };
#pragma unroll
    for (int i = 0; i < KS; ++i) {
        const int ay = y - i;
        bool iny[KS];
#pragma unroll
        for (int q = 0; q < KS; ++q) iny[q] = (0 <= ay + q && ay + q <= H - 1);
#pragma unroll
        for (int j = 0; j < KS; ++j) {
            const int ax = x - j;
            bool inx[KS];
#pragma unroll
            for (int q = 0; q < KS; ++q) inx[q] = (0 <= ax + q && ax + q <= W - 1);
            // software pipeline: the entry two ahead and the view data of the next entry are in flight while the
            // current entry is added
            const unsigned int s0 = bs[i][KS - 1 - j], e0 = bs[i][KS - j];
            unsigned int cur = first[i][j];
            if (!ok(cur)) continue;
            unsigned int nxt = s0 + 1 < e0 ? __ldg(entries + s0 + 1) : kNone;
            Src d = fetch(cur);
            for (unsigned int k = s0;; ++k) {
                const unsigned int n2 = (ok(nxt) && k + 2 < e0) ? __ldg(entries + k + 2) : kNone;
                Src dn = {};
                if (ok(nxt)) dn = fetch(nxt);
                const int v = (int)(cur >> 24);
                float sx = 0.f, sy = 0.f, dxj = 0.f, dyi = 0.f;
#pragma unroll
                for (int q = 0; q < KS; ++q) {
                    const float dx = inx[q] ? fp_overlap(q, KS, ax + q, d.px, dsf) : 0.f;
                    const float dy = iny[q] ? fp_overlap(q, KS, ay + q, d.py, dsf) : 0.f;
                    sx = __fadd_rn(sx, dx);
                    sy = __fadd_rn(sy, dy);
                    if (q == j) dxj = dx;
                    if (q == i) dyi = dy;
                }
                const float norm = __fmul_rn(sx, sy);
                const float inv = (norm != 0.0f) ? __frcp_rn(norm) : 1.0f;
                const float A = __fmul_rn(dxj, __fmul_rn(dyi, inv)) * d.w;
                acc[v * 4 + 3][t] += A;
                acc[v * 4 + 0][t] += A * d.c0;
                acc[v * 4 + 1][t] += A * d.c1;
                acc[v * 4 + 2][t] += A * d.c2;
                if (!ok(nxt)) break;  // entries ascend by view: the rest of the bucket are later views
                cur = nxt;
                nxt = n2;
                d = dn;
            }
        }
    }
    const size_t o = (size_t)y * W + x, N = (size_t)W * H;
    float f[kLearnChannels];
#pragma unroll
    for (int c = 0; c < kLearnChannels; ++c) f[c] = 0.f;
    const float gxo = gx[o], gyo = gy[o];
    const float gxl = x > 0 ? gx[o - 1] : 0.f, gyu = y > 0 ? gy[o - W] : 0.f;
    f[3] = x < W - 1 ? fminf(fmaxf(gxo, -1.f), 1.f) : 0.f;
    f[4] = y < H - 1 ? fminf(fmaxf(gyo, -1.f), 1.f) : 0.f;
    f[5] = vis[o] ? 1.f : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float *u = U + c * N;
        const float uc = u[o];
        float lx, ly;
        if (x == 0) lx = uc - u[o + 1] + gxo;
        else if (x < W - 1) lx = 2.f * uc - u[o - 1] - u[o + 1] + gxo - gxl;
        else lx = uc - u[o - 1] - gxl;
        if (y == 0) ly = uc - u[o + W] + gyo;
        else if (y < H - 1) ly = 2.f * uc - u[o - W] - u[o + W] + gyo - gyu;
        else ly = uc - u[o - W] - gyu;
        f[c] = uc;
        f[38 + c] = fminf(fmaxf(-(lx + ly), -4.f), 4.f);
    }
    // quotients as products with one reciprocal each (within an ulp or two of the division; stored as BF16); a
    // divisor below 1e-30, whose reciprocal could overflow, divides
    auto quot = [](float num, float den, float rden) {
        return den >= 1e-30f ? num * rden : (den > 0.f ? num / den : 0.f);
    };
    float total = 0.f;
#pragma unroll
    for (int v = 0; v < kLearnViews; ++v) total += acc[v * 4 + 3][t];
    const float rtotal = total >= 1e-30f ? __frcp_rn(total) : 0.f;
#pragma unroll
    for (int v = 0; v < kLearnViews; ++v) {
        const float a = acc[v * 4 + 3][t];
        const float ra = a >= 1e-30f ? __frcp_rn(a) : 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) f[6 + 3 * v + c] = quot(acc[v * 4 + c][t], a, ra);
        f[6 + 3 * kLearnViews + v] = quot(a, total, rtotal);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(out + o * kLearnChannels);
#pragma unroll
    for (int q = 0; q < kLearnChannels / 8; ++q) {
        uint4 u;
        __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[8 * q + 2 * i], f[8 * q + 2 * i + 1]);
        dst[q] = u;
    }
}

// Data-term gradient and the proximal data F (vtv_sr_dataterm_intensities :1953-1963 and
// vtv_sr_ista_step_unstructured :1785-1812): G = alpha sigma^2 sum A e / sum A, F = clamp(U + fs clamp(G)).
// With a gradient term (gt.resg set, vtv_sr_dataterm_gradients sources/optimization.cu:1969-2116) the
// residuals of the gradients are splatted too (same entries, same coverage) and
// G += beta * (-step) * [sigma^2 if gw_type] * sum A resg / sum A.
template <int KS>
__global__ void k_dataterm_F(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                             const unsigned int *__restrict__ entries, const float *__restrict__ tau, SplatSrc src,
                             float s2, float alpha, float fscale, const float *__restrict__ U,
                             float *__restrict__ F, float *__restrict__ G_out, GradTerm gt) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    float acc[3], norm;
    splat_accumulate<KS, 3>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    float accg[3] = {0.f, 0.f, 0.f}, normg = 0.f;
    if (gt.resg) {
        const size_t s3 = (size_t)3 * n;
        const SplatSrc sg{{gt.resg, gt.resg + n, gt.resg + 2 * (size_t)n}, {s3, s3, s3}, nullptr};
        splat_accumulate<KS, 3>(x, y, W, H, n, dsf, BW, start, entries, tau, sg, accg, normg);
    }
    const size_t o = (size_t)y * W + x, N = (size_t)W * H;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float gi = (norm != 0.f) ? acc[c] / norm : acc[c];
        gi *= s2;
        float G = 0.f + alpha * gi;
        if (gt.resg) {
            float gg = (normg != 0.f) ? accg[c] / normg : accg[c];
            if (gt.gw) gg *= s2;
            gg *= -gt.step;
            G += gt.beta * gg;
        }
        if (G_out) G_out[c * N + o] = G;
        G = fminf(1.0f, fmaxf(-1.0f, G));
        G *= fscale;
        G += U[c * N + o];
        F[c * N + o] = fminf(1.0f, fmaxf(0.0f, G));
    }
}

// Regulariser weight before the blur (coco_vtv_sr_init_regularizer_weight_unstructured
// sources/optimization.cu:2262-2319, vtv_sr_init_regularizer_weight_device vtv_sr_kernels.cu:1172-1195).
// norm_prior is the coverage accumulator's content before the call (never cleared upstream).
template <int KS>
__global__ void k_regweight(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                            const unsigned int *__restrict__ entries, const float *__restrict__ tau, SplatSrc src,
                            const float *__restrict__ norm_prior, float s2, float lmax, float lmin, float mmax,
                            float *__restrict__ g0, float *__restrict__ norm_out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    float acc[3], norm;
    splat_accumulate<KS, 1>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x;
    const float nm = (norm_prior ? norm_prior[o] : 0.f) + norm;
    float m = (nm != 0.f) ? acc[0] / nm : acc[0];
    m *= s2;
    g0[o] = (m == 0.0f) ? lmax : fmaxf(lmin, lmax - m / mmax);
    if (norm_out) norm_out[o] = nm;
}

// Gradient splatting of IBR_gradient (init_u_gradient sources/gradientIBR.cu:856-916): payload
// (Sobel_x, Sobel_y, weight) of every source pixel, normalised by the coverage; mask scaled by sigma^2.
template <int KS>
__global__ void k_u_gradient(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                             const unsigned int *__restrict__ entries, const float *__restrict__ tau, SplatSrc src,
                             float s2, float *__restrict__ gx, float *__restrict__ gy, float *__restrict__ mask) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    float acc[3], norm;
    splat_accumulate<KS, 3>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x;
    if (norm != 0.f) {
        acc[0] /= norm;
        acc[1] /= norm;
        acc[2] /= norm;
    }
    gx[o] = acc[0];
    gy[o] = acc[1];
    mask[o] = acc[2] * s2;
}

// ====================================================================== stencils on the target
// Sobel of the luminance (vtv_sr_compute_gradient_device, vtv_sr_kernels_unstructured.cu:96-148); with a
// mask, interior pixels without a fully visible 3x3 neighbourhood keep the old content of gx/gy.
// Also used on source views (sources/gradientIBR_kernels.cuh:57-100, no mask); views are addressed with a
// per-blockIdx.z plane stride.
__global__ void k_sobel(int W, int H, const float *__restrict__ rgb, size_t in_stride, size_t ch_stride,
                        float *__restrict__ gx, float *__restrict__ gy, size_t out_stride,
                        const uint8_t *__restrict__ vis, double *__restrict__ abs_partial) {
    __shared__ double red[8];
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    const float *r = rgb + (size_t)z * in_stride, *g = r + ch_stride, *b = g + ch_stride;
    float *ox = gx + (size_t)z * out_stride, *oy = gy + (size_t)z * out_stride;
    double a = 0.0;
    if (x < W && y < H) {
        const size_t o = (size_t)y * W + x;
        float gX = 0.f, gY = 0.f;
        bool write = true;
        if (0 < x && x < W - 1 && 0 < y && y < H - 1) {
            if (vis) {
                for (int dy = -1; dy <= 1 && write; ++dy)
                    for (int dx = -1; dx <= 1; ++dx)
                        if (!vis[o + (ptrdiff_t)dy * W + dx]) {
                            write = false;
                            break;
                        }
            }
            if (write) {
                // The reference evaluates the luminance as a double expression rounded to float; the
                // masked (target) Sobel does the same because the angular weights amplify its rounding.
                auto L = [&](int dx, int dy) {
                    const size_t q = o + (ptrdiff_t)dy * W + dx;
                    if (!vis) return lum(r[q], g[q], b[q]);
                    return (float)__dadd_rn(__dadd_rn(__dmul_rn(0.2126, (double)r[q]), __dmul_rn(0.7152, (double)g[q])),
                                            __dmul_rn(0.0722, (double)b[q]));
                };
                const float Ypp = L(-1, -1), Ypc = L(0, -1), Ypn = L(1, -1);
                const float Ycp = L(-1, 0), Ycn = L(1, 0);
                const float Ynp = L(-1, 1), Ync = L(0, 1), Ynn = L(1, 1);
                gX = (Ypn + 2.f * Ycn + Ynn - Ypp - 2.f * Ycp - Ynp) / 8.f;
                gY = (Ynp + 2.f * Ync + Ynn - Ypp - 2.f * Ypc - Ypn) / 8.f;
            }
        }
        if (write) {
            ox[o] = gX;
            oy[o] = gY;
        }
        if (abs_partial) a = fabs((double)ox[o]) + fabs((double)oy[o]);
    }
    if (abs_partial) {
        // block of 32x8 threads
        const int tid = threadIdx.y * blockDim.x + threadIdx.x;
        double v = a;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if ((tid & 31) == 0) red[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            double s = 0;
            for (int i = 0; i < (int)(blockDim.x * blockDim.y) / 32; ++i) s += red[i];
            abs_partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
        }
    }
}

// Inner ROF iterations, temporally blocked. One iteration is the dual step p += sigma grad_fwd(U) (vtv_rof.cu:118-147),
// the reprojection of the 6 duals onto the ball of radius g (vtv_rof.cu:280-320) and the primal prox
// U = (tau F + lambda (U + tau div_bwd p)) / (tau + lambda) (cuda_kernels.cu:504-532). All niter of them run in one
// cooperative launch: each super-step runs up to K iterations on a (kRofTX + 2 K) x (TY + 2 K) region around a
// kRofTX x TY tile and writes back the tile, whose values depend only on the region (the halo absorbs one pixel of
// staleness per iteration from each side). Super-steps read one global (U, P) pair and write the other, with a bounded
// grid barrier between them; a block with one tile keeps it in registers and reads back only the halo.
//
// A thread owns V vertically adjacent pixels: their U, p, tau F and g stay in registers, the neighbours above and
// below come from registers too except at the ends, and shared memory carries U and the x duals (which the left and
// right neighbours read) and the y duals of each thread's last pixel. The code of a pixel has no branch for the image:
//   - a dual whose forward difference does not exist (the last column / row, pixels outside the image) has step 0 and
//     keeps its value; outside the image it starts at 0, which is what the divergence of the first column / row subtracts;
//   - what other pixels outside the image hold is in no difference.
// Infinite, not-a-number and overflowing values spread as in the reference's loop: a dual whose squared norm is not finite
// is worked out again, leaving out differences that do not exist (the step of 0 gives 0 times infinity) and scaling by
// r / inf = 0, off the common path; an infinite numerator of the prox stays infinite.
// Threads whose pixels the tile no longer depends on skip the iteration; what the rest computes beyond that is stale
// and stays outside the tile.
// The projection scales by g / |p| only beyond the ball, as g times a reciprocal square root with one Newton step; the
// prox divides by tau + lambda as a reciprocal product with its remainder corrected.
//
// Bound by the chain of an iteration (two block barriers, shared-memory loads, the projection) and by the super-steps'
// grid barriers, about 3 us each (waiting for the eight neighbouring blocks alone, with a flag each, took longer). 256^2,
// 300 iterations (K = 8, TY = 16, V = 2, 128 blocks): 537 -> 325 us a launch against the form before it with two scattered
// pixels per thread, border branches, and IEEE square roots and divisions; V = 4 saves instructions but leaves half the
// warps (398). K, TY and V are picked per image size by the host's autotuner; all give the same values.
constexpr int kRofTX = 32;
template <int K, int TY, int V>
__host__ __device__ constexpr int rof_threads() {
    return ((kRofTX + 2 * K) * ((TY + 2 * K) / V) + 31) / 32 * 32;
}
// U and the x duals (3 planes each, one row more than the region and a cell on either side), the segments' last y duals
template <int K, int TY, int V>
__host__ __device__ constexpr int rof_plane() {
    return (kRofTX + 2 * K) * (TY + 2 * K + 1) + 2;
}
template <int K, int TY, int V>
__host__ __device__ constexpr int rof_plane_y() {
    return (kRofTX + 2 * K) * ((TY + 2 * K) / V + 1);
}
template <int K, int TY, int V>
constexpr size_t rof_smem() {
    return sizeof(float) * (size_t)(6 * rof_plane<K, TY, V>() + 3 * rof_plane_y<K, TY, V>());
}

template <int K, int TY, int V>
__global__ void __launch_bounds__((rof_threads<K, TY, V>())) k_rof_persistent(int W, int H, int niter, float tau,
                                                                           float sigma, float lam, float *U0,
                                                                           float *P0, float *U1, float *P1,
                                                                           const float *__restrict__ F,
                                                                           const float *__restrict__ g, GridBarrier gb) {
    constexpr int RX = kRofTX + 2 * K, RY = TY + 2 * K;
    static_assert(RY % V == 0, "whole segments");
    constexpr int PL = rof_plane<K, TY, V>(), PY = rof_plane_y<K, TY, V>();
    constexpr float kInf = INFINITY;
    extern __shared__ float sm[];
    const int seg = threadIdx.x / RX, lx = threadIdx.x - seg * RX, ly0 = seg * V;
    const bool mine = seg < RY / V;
    float *sU = sm + 1 + ly0 * RX + lx, *sPx = sU + 3 * PL;         // this thread's first pixel, plane 0
    float *sPy = sm + 6 * PL + (seg + 1) * RX + lx;                 // its last pixel's y dual; - RX: the segment above
    const int tiles_x = (W + kRofTX - 1) / kRofTX, ntiles = tiles_x * ((H + TY - 1) / TY);
    const bool resident = ntiles <= (int)gridDim.x;  // one tile per block
    const size_t N = (size_t)W * H;
    const float denom = tau + lam, rden = __frcp_rn(denom);
    // distance of the segment's column and of its nearest row from the tile
    const int dx = max(max(K - lx, lx - (K + kRofTX - 1)), 0);
    const int dist = max(dx, max(max(K - (ly0 + V - 1), ly0 - (K + TY - 1)), 0));
    const bool tile_x = mine && lx >= K && lx < K + kRofTX;
    unsigned int gen = 0;
    int step = 0;
    // shared memory that no thread writes (pads) is read too: finite from here on
    for (int i = threadIdx.x; i < 6 * PL + 3 * PY; i += blockDim.x) sm[i] = 0.f;
    __syncthreads();
    float u[V][3], p[V][6], tf[V][3], r[V], sy[V], sx = 0.f;
    for (int done = 0; done < niter; done += K, ++step) {
        const int iters = min(K, niter - done);
        const float *Ui = (step & 1) ? U1 : U0, *Pi = (step & 1) ? P1 : P0;
        float *Uo = (step & 1) ? U0 : U1, *Po = (step & 1) ? P0 : P1;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int gx = (t % tiles_x) * kRofTX - K + lx, gy0 = (t / tiles_x) * TY - K + ly0;
            const bool inx = mine && gx >= 0 && gx < W;
            sx = inx && gx < W - 1 ? sigma : 0.f;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int gy = gy0 + k;
                const bool in = inx && gy >= 0 && gy < H;
                const bool own = tile_x && ly0 + k >= K && ly0 + k < K + TY;
                const size_t o = in ? (size_t)gy * W + gx : 0;
                sy[k] = gy >= 0 && gy < H - 1 ? sigma : 0.f;
                if (step == 0 || !resident) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) tf[k][c] = in ? tau * __ldg(F + c * N + o) : 0.f;
                    r[k] = in ? __ldg(g + o) : 0.f;
                }
                if (step == 0 || !resident || !own) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) u[k][c] = in ? __ldcg(Ui + c * N + o) : 0.f;
#pragma unroll
                    for (int c = 0; c < 6; ++c) p[k][c] = in ? __ldcg(Pi + c * N + o) : 0.f;
                }
                if (mine) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        sU[c * PL + k * RX] = u[k][c];
                        sPx[c * PL + k * RX] = p[k][2 * c];
                    }
                }
            }
            if (mine) {
#pragma unroll
                for (int c = 0; c < 3; ++c) sPy[c * PY] = p[V - 1][2 * c + 1];
            }
            __syncthreads();
            for (int it = 0; it < iters; ++it) {
                // after iteration it the tile needs U within distance iters - it - 1 of it, and that prox reads the
                // duals one pixel further out
                if (mine && dist <= iters - it) {
                    float below[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) below[c] = sU[c * PL + V * RX];
#pragma unroll
                    for (int k = 0; k < V; ++k) {
                        float n2 = 0.f, v[6], scale = 1.f;
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float uc = u[k][c];
                            const float ur = sU[c * PL + k * RX + 1];
                            const float ud = k + 1 < V ? u[k + 1 < V ? k + 1 : k][c] : below[c];
                            v[2 * c] = fmaf(sx, ur - uc, p[k][2 * c]);
                            v[2 * c + 1] = fmaf(sy[k], ud - uc, p[k][2 * c + 1]);
                            n2 = fmaf(v[2 * c + 1], v[2 * c + 1], fmaf(v[2 * c], v[2 * c], n2));
                        }
                        // beyond the ball: p *= g / |p| (a negative radius scales always, as |p| > g does)
                        const float r2 = r[k] < 0.f ? -1.f : r[k] * r[k];
                        if (!(n2 <= r2)) {
                            if (n2 > r2 && n2 < kInf) {
                                const float e = rsqrtf(n2);
                                scale = r[k] * fmaf(e * 0.5f, fmaf(-n2 * e, e, 1.f), e);
                            } else {
                                n2 = 0.f;
#pragma unroll
                                for (int c = 0; c < 3; ++c) {
                                    if (!(inx && gx < W - 1)) v[2 * c] = p[k][2 * c];
                                    if (!(gy0 + k >= 0 && gy0 + k < H - 1)) v[2 * c + 1] = p[k][2 * c + 1];
                                    n2 = fmaf(v[2 * c + 1], v[2 * c + 1], fmaf(v[2 * c], v[2 * c], n2));
                                }
                                if (n2 > r2) scale = n2 < kInf ? r[k] / sqrtf(n2) : 0.f;
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 6; ++c) p[k][c] = v[c] * scale;
#pragma unroll
                        for (int c = 0; c < 3; ++c) sPx[c * PL + k * RX] = p[k][2 * c];
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) sPy[c * PY] = p[V - 1][2 * c + 1];
                }
                __syncthreads();
                if (mine && dist <= iters - it - 1) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        float above = sPy[c * PY - RX];
#pragma unroll
                        for (int k = 0; k < V; ++k) {
                            const float py = p[k][2 * c + 1];
                            const float st = p[k][2 * c] + py - sPx[c * PL + k * RX - 1] - above;
                            above = py;
                            const float x = fmaf(lam, fmaf(tau, st, u[k][c]), tf[k][c]), q = x * rden;
                            const float rest = fmaf(-denom, q, x);
                            u[k][c] = fabsf(rest) < kInf ? fmaf(rest, rden, q) : q;
                            sU[c * PL + k * RX] = u[k][c];
                        }
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int gy = gy0 + k;
                if (!(tile_x && inx && ly0 + k >= K && ly0 + k < K + TY && gy < H)) continue;
                const size_t o = (size_t)gy * W + gx;
#pragma unroll
                for (int c = 0; c < 3; ++c) Uo[c * N + o] = u[k][c];
#pragma unroll
                for (int c = 0; c < 6; ++c) Po[c * N + o] = p[k][c];
            }
        }
        if (done + K < niter && !grid_sync(gb, gen)) return;
    }
}

// Count of pixels whose largest channel change reaches thr (sr_compare_images,
// sources/super-resolution.cpp:16-51).
__global__ void k_moving(size_t N, const float *__restrict__ A, const float *__restrict__ B, float thr,
                         double *__restrict__ partial) {
    __shared__ double red[8];
    const size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    double c = 0.0;
    if (o < N) {
        float mx = 0.f;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) mx = fmaxf(mx, fabsf(A[ch * N + o] - B[ch * N + o]));
        c = (mx < thr) ? 0.0 : 1.0;
    }
    const double s = block_sum<256>(c, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Separable 11-tap Gaussian with clamp-to-edge (convolutionRowGPU / convolutionColumnGPU,
// cocolib/cocolib/cuda/cuda_convolutions.cu:110-238; kernel from gsl_kernel_gauss_1xn(11, 2.0)).
__constant__ float c_gauss[11];

// Both passes stage their block's rows (columns) with the 5-pixel halo in shared memory, clamped to the image as
// the taps are, and sum the 11 taps there in the order of the reference's loop.
constexpr int kBlurBX = 32, kBlurBY = 8, kBlurR = 5;

__global__ void __launch_bounds__(kBlurBX * kBlurBY) k_blur_rows(int W, int H, const float *__restrict__ in,
                                                                 float *__restrict__ out) {
    __shared__ float t[kBlurBY][kBlurBX + 2 * kBlurR];
    const int x0 = blockIdx.x * kBlurBX, y = min((int)(blockIdx.y * kBlurBY + threadIdx.y), H - 1);
    for (int i = threadIdx.x; i < kBlurBX + 2 * kBlurR; i += kBlurBX)
        t[threadIdx.y][i] = __ldg(in + (size_t)y * W + min(max(x0 - kBlurR + i, 0), W - 1));
    __syncthreads();
    const int x = x0 + threadIdx.x, yo = blockIdx.y * kBlurBY + threadIdx.y;
    if (x >= W || yo >= H) return;
    float s = 0.f;
#pragma unroll
    for (int k = -kBlurR; k <= kBlurR; ++k) s += t[threadIdx.y][threadIdx.x + kBlurR + k] * c_gauss[5 - k];
    out[(size_t)yo * W + x] = s;
}

__global__ void __launch_bounds__(kBlurBX * kBlurBY) k_blur_cols(int W, int H, const float *__restrict__ in,
                                                                 float *__restrict__ out) {
    __shared__ float t[kBlurBY + 2 * kBlurR][kBlurBX];
    const int x = min((int)(blockIdx.x * kBlurBX + threadIdx.x), W - 1), y0 = blockIdx.y * kBlurBY;
    for (int i = threadIdx.y; i < kBlurBY + 2 * kBlurR; i += kBlurBY)
        t[i][threadIdx.x] = __ldg(in + (size_t)min(max(y0 - kBlurR + i, 0), H - 1) * W + x);
    __syncthreads();
    const int xo = blockIdx.x * kBlurBX + threadIdx.x, y = y0 + threadIdx.y;
    if (xo >= W || y >= H) return;
    float s = 0.f;
#pragma unroll
    for (int k = -kBlurR; k <= kBlurR; ++k) s += t[threadIdx.y + kBlurR + k][threadIdx.x] * c_gauss[5 - k];
    out[(size_t)y * W + xo] = s;
}

// Deterministic final reduction of FP64 partials: block b sums list b.
__global__ void k_reduce_final(const ReduceLists lists) {
    __shared__ double red[32];
    const int count = lists.count[blockIdx.x];
    const double *partial = lists.partial[blockIdx.x];
    double s = 0.0;
    for (int i = threadIdx.x; i < count; i += blockDim.x) s += partial[i];
    const double t = block_sum<1024>(s, red);
    if (threadIdx.x == 0) *lists.out[blockIdx.x] = t;
}

// One energy-trace entry: the host's float expression lambda e_tv + alpha e_int (+ beta e_grad), without
// contraction (the host code is compiled with -ffp-contract=off).
__global__ void k_trace_energy(const double *__restrict__ sums, float lambda, float alpha, float beta, int grad,
                               double *__restrict__ dst) {
    float e = __fadd_rn(__fmul_rn(lambda, (float)sums[0]), __fmul_rn(alpha, (float)sums[1]));
    if (grad) e = __fadd_rn(e, __fmul_rn(beta, (float)sums[3]));
    *dst = (double)e;
}

__global__ void k_premultiply_dpart(int V, int n, const float *__restrict__ dpart3, int dpart_channels,
                                    float *__restrict__ dp) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    if (m >= n) return;
    const float *src = dpart3 + (size_t)v * dpart_channels * n;
    const float sz = src[m];
    dp[(size_t)v * 2 * n + m] = src[n + m] * sz;
    dp[(size_t)v * 2 * n + n + m] = src[2 * n + m] * sz;
}

__global__ void k_copy_tau(int V, int n, const float *__restrict__ tau_in, int tau_channels,
                           float *__restrict__ tau) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    if (m >= n) return;
    const float *src = tau_in + (size_t)v * tau_channels * n;
    tau[(size_t)v * 2 * n + m] = src[m];
    tau[(size_t)v * 2 * n + n + m] = src[n + m];
}

// ====================================================================== host launchers
static inline dim3 grid2(int W, int H, dim3 b) { return dim3((W + b.x - 1) / b.x, (H + b.y - 1) / b.y); }


void launch_bucket_build(const Geometry &G, const float *tau, Buckets &B, cudaStream_t st, LaunchCounter &lc,
                         bool counted) {
    ProfScope _ps(lc, "bucket_build", st);
    const int ks = G.dsf + 1;
    // one block per (view, chunk of 256 * kBucketPer source pixels), views varying fastest: the blocks in flight
    // cover one band of source rows in every view, so the buckets they count into and fill (whose entries
    // interleave the views) stay in one band of the target, in L2, until every view's entry of a sector is in
    const dim3 b1(256), gs((unsigned)((G.n + 256 * kBucketPer - 1) / (256 * kBucketPer)) * (unsigned)G.V);
    if (!counted) {  // else k_tau has counted while writing tau
        cudaMemsetAsync(B.count, 0, sizeof(unsigned int) * B.nb, st);
        cudaMemsetAsync(B.mask, 0, sizeof(unsigned long long) * B.nb * B.mask_words, st);
        k_bucket_count<<<gs, b1, 0, st>>>(G.V, G.n, G.W, G.H, G.dsf, B.BW, tau, B.count, B.mask, B.nb);
        lc.add(1);
    }
    // exclusive scan of the counts: block-local scans, then every block adds the sum of the block totals before
    // it (integer sums, so the result does not depend on the order) and the last block writes the total
    const int nblk = (B.nb + kScanSpan - 1) / kScanSpan;
    // programmatic launches: each kernel's launch overlaps the tail of the one before it; k_scan_finish clears
    // the counts for their use as k_bucket_fill's cursors
    launch_pdl(k_scan_blocks, dim3(nblk), dim3(kScanBlock), 0, st, B.nb, B.count, B.start, B.block_sums);
    launch_pdl(k_scan_finish, dim3(nblk), dim3(kScanBlock), 0, st, B.nb, B.start, B.block_sums, B.count);
    lc.add(2);
    launch_pdl(B.mask_words == 1   ? k_bucket_fill<1>
               : B.mask_words == 2 ? k_bucket_fill<2>
                                   : k_bucket_fill<0>,
               gs, b1, 0, st, G.V, G.n, G.W, G.H, G.dsf, B.BW, tau, B.start, B.count, B.mask, B.mask_words, B.nb,
               B.entries);
    launch_pdl(k_bucket_sort, dim3((B.nb + kSortBuckets - 1) / kSortBuckets), dim3(kSortBuckets), 0, st, B.nb,
               B.start, B.mask, B.mask_words, B.entries);
    lc.add(2);
    (void)ks;
}

void launch_residual(const Geometry &G, const float *U, const float *img, const float *tau, const float *wgt, float s2,
                     float *res, double *partial, cudaStream_t st, LaunchCounter &lc, bool splat_set) {
    ProfScope _ps(lc, "residual", st);
    const dim3 b(256), g((G.n + 255) / 256, G.V);
    auto run = [&](auto kernel) {
        kernel<<<g, b, 0, st>>>(G.V, G.n, G.W, G.H, G.dsf, U, img, tau, wgt, s2, res, partial, splat_set ? 1 : 0);
    };
    switch (G.dsf + 1) {
        case 2: run(partial ? k_residual<2, true> : k_residual<2, false>); break;
        case 3: run(partial ? k_residual<3, true> : k_residual<3, false>); break;
        case 4: run(partial ? k_residual<4, true> : k_residual<4, false>); break;
        case 5: run(partial ? k_residual<5, true> : k_residual<5, false>); break;
        default: break;
    }
    lc.add(1);
}
int residual_partials(const Geometry &G) { return ((G.n + 255) / 256) * G.V; }

template <typename TW>
static void weights_typed(const Geometry &G, const float *gx, const float *gy, const float *tau, const float *dp,
                          float sigma, float thr, TW *wgt, cudaStream_t st) {
    const dim3 b(256), g((G.n + 255) / 256, G.V);
    // (a negative threshold would clip the gradient 0 to 0 / 0: left to the general kernel)
    if (!gx && !dp && G.w % 4 == 0 && !(0.f > thr)) {
        const float s2 = sigma * sigma;
        k_weights_flat<TW><<<dim3((G.n / 4 + 255) / 256, G.V), b, 0, st>>>(G.n, G.w, G.h, G.W, G.H, tau, 1.0f / s2, wgt);
        return;
    }
#define LFRV_WEIGHTS(KS_)                                                                                          \
    if (gx)                                                                                                        \
        k_weights<KS_, TW, true><<<g, b, 0, st>>>(G.V, G.n, G.w, G.h, G.W, G.H, G.dsf, gx, gy, tau, dp, sigma, thr, wgt); \
    else                                                                                                           \
        k_weights<KS_, TW, false><<<g, b, 0, st>>>(G.V, G.n, G.w, G.h, G.W, G.H, G.dsf, gx, gy, tau, dp, sigma, thr, wgt);
    switch (G.dsf + 1) {
        case 2: LFRV_WEIGHTS(2) break;
        case 3: LFRV_WEIGHTS(3) break;
        case 4: LFRV_WEIGHTS(4) break;
        case 5: LFRV_WEIGHTS(5) break;
        default: break;
    }
#undef LFRV_WEIGHTS
}

void launch_weights(const Geometry &G, const float *gx, const float *gy, const float *tau, const float *dp, float sigma,
                    float thr, void *wgt, cudaStream_t st, LaunchCounter &lc, bool bf16) {
    ProfScope _ps(lc, "weights", st);
    if (bf16) weights_typed(G, gx, gy, tau, dp, sigma, thr, static_cast<__nv_bfloat16 *>(wgt), st);
    else weights_typed(G, gx, gy, tau, dp, sigma, thr, static_cast<float *>(wgt), st);
    lc.add(1);
}

static const dim3 kTile(32, 8);

void launch_coverage(const Geometry &G, const Buckets &B, const float *tau, float *cov, uint8_t *vis, cudaStream_t st,
                     LaunchCounter &lc) {
    LFRV_KS_DISPATCH(G.dsf + 1, k_coverage, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW, B.start,
                     B.entries, tau, cov, vis);
    lc.add(1);
}

void launch_vis_any(const Geometry &G, const Buckets &B, const float *tau, uint8_t *vis, cudaStream_t st,
                    LaunchCounter &lc) {
    LFRV_KS_DISPATCH(G.dsf + 1, k_vis_any, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW, B.start,
                     B.entries, tau, vis);
    lc.add(1);
}

void launch_initial_image(const Geometry &G, const Buckets &B, const float *tau, const float *img, const float *wgt,
                          float *U, float *norm, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "initial_image", st);
    const size_t s3 = (size_t)3 * G.n;
    SplatSrc src{{img, img + G.n, img + 2 * (size_t)G.n}, {s3, s3, s3}, wgt};
    LFRV_KS_DISPATCH(G.dsf + 1, k_initial_image, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW,
                     B.start, B.entries, tau, src, U, norm);
    lc.add(1);
}

template <typename TS>
static void learn_input_typed(const Geometry &G, const Buckets &B, const float *tau, const TS *img, const TS *wgt,
                              const float *U, const float *gx, const float *gy, const uint8_t *vis,
                              __nv_bfloat16 *out, cudaStream_t st) {
    const dim3 g((G.W + 63) / 64, (G.H + 3) / 4);  // 64 x 4 pixels per block of kTile (32 x 8) threads
    switch (G.dsf + 1) {
        case 2: k_learn_input<2, TS><<<g, kTile, 0, st>>>(G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, img, wgt, U, gx, gy, vis, out); break;
        case 3: k_learn_input<3, TS><<<g, kTile, 0, st>>>(G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, img, wgt, U, gx, gy, vis, out); break;
        case 4: k_learn_input<4, TS><<<g, kTile, 0, st>>>(G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, img, wgt, U, gx, gy, vis, out); break;
        case 5: k_learn_input<5, TS><<<g, kTile, 0, st>>>(G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, img, wgt, U, gx, gy, vis, out); break;
        default: break;
    }
}

void launch_learn_input(const Geometry &G, const Buckets &B, const float *tau, const void *img, const void *wgt,
                        const float *U, const float *gx, const float *gy, const uint8_t *vis, void *out,
                        cudaStream_t st, LaunchCounter &lc, bool bf16) {
    ProfScope _ps(lc, "learn_input", st);
    __nv_bfloat16 *o = static_cast<__nv_bfloat16 *>(out);
    if (bf16)
        learn_input_typed(G, B, tau, static_cast<const __nv_bfloat16 *>(img), static_cast<const __nv_bfloat16 *>(wgt),
                          U, gx, gy, vis, o, st);
    else
        learn_input_typed(G, B, tau, static_cast<const float *>(img), static_cast<const float *>(wgt), U, gx, gy, vis,
                          o, st);
    lc.add(1);
}

void launch_dataterm_F(const Geometry &G, const Buckets &B, const float *tau, const float *res, float s2, float alpha,
                       float fscale, const float *U, float *F, float *G_out, const GradTerm &gt, cudaStream_t st,
                       LaunchCounter &lc) {
    ProfScope _ps(lc, "dataterm", st);
    const size_t s3 = (size_t)3 * G.n;
    SplatSrc src{{res, res + G.n, res + 2 * (size_t)G.n}, {s3, s3, s3}, nullptr};
    LFRV_KS_DISPATCH(G.dsf + 1, k_dataterm_F, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW, B.start,
                     B.entries, tau, src, s2, alpha, fscale, U, F, G_out, gt);
    lc.add(1);
}

// cuda_laplacian_device (cocolib/cocolib/vtv/vtv_sr_kernels_unstructured.cu:720-760) without a visibility mask,
// on `planes` planes of W x H: mean of the in-image 4-neighbours (left, up, right, down) minus the centre.
__device__ __forceinline__ float laplacian_at(const float *u, int W, int H, int x, int y) {
    const size_t o = (size_t)y * W + x;
    float v = 0.f, wt = 0.f;
    if (x > 0) { v += u[o - 1]; wt += 1.f; }
    if (y > 0) { v += u[o - W]; wt += 1.f; }
    if (x < W - 1) { v += u[o + 1]; wt += 1.f; }
    if (y < H - 1) { v += u[o + W]; wt += 1.f; }
    v /= wt;
    v -= u[o];
    return v;
}

__global__ void k_laplacian(int W, int H, int planes, const float *__restrict__ in, float *__restrict__ out) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t N = (size_t)W * H, o = (size_t)y * W + x;
    for (int c = 0; c < planes; ++c) out[c * N + o] = laplacian_at(in + c * N, W, H, x, y);
}

// Residual of the gradient data term for every source pixel (vtv_sr_dataterm_gradients, optimization.cu:
// 2010-2069): dsf^2 A_i lap(U) - lap(v_i), times omega_i when gw_type != 0. lapU is 3 x N (k_laplacian).
template <int KS>
__global__ void __launch_bounds__(256) k_residual_grad(int V, int w, int h, int W, int H, int dsf,
                                                       const float *__restrict__ lapU, const float *__restrict__ img,
                                                       const float *__restrict__ tau, const float *__restrict__ wgt,
                                                       int gw, float *__restrict__ resg) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    const int n = w * h;
    if (m >= n) return;
    const size_t N = (size_t)W * H;
    const float tx = tau[(size_t)v * 2 * n + m], ty = tau[(size_t)v * 2 * n + n + m];
    float a[3] = {0.f, 0.f, 0.f};
    if (in_gather(tx, ty, W, H)) {
        Footprint fp;
        footprint<KS>(tx, ty, dsf, W, H, fp);
#pragma unroll
        for (int j = 0; j < KS; ++j)
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                const int x = fp.x0 + j, y = fp.y0 + i;
                if (0 <= x && x <= W - 1 && 0 <= y && y <= H - 1) {
                    const float A = fp.A[KS * i + j];
                    const size_t o = (size_t)y * W + x;
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[c] += A * __ldg(lapU + c * N + o);
                }
            }
    }
    const float dsf2 = (float)(dsf * dsf);
    int mx, my;
    pixel_of(m, w, n, __frcp_rn((float)w), mx, my);
    const float *iv = img + (size_t)v * 3 * n;
    float *rv = resg + (size_t)v * 3 * n;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float d = a[c] * dsf2;
        d -= laplacian_at(iv + (size_t)c * n, w, h, mx, my);
        if (gw) d *= wgt[(size_t)v * n + m];
        rv[(size_t)c * n + m] = d;
    }
}

// Gradient term of the reference energy (coco_vtv_sr_primal_energy_unstructured, optimization.cu:1610-1700):
// per source pixel (A_i Sobel_x lum U - Sobel_x lum v_i)^2 + (same for y), times omega_i sigma^2 when
// gw_type != 0. ugrad: 2 x N (Sobel of the luminance of U, no mask); vgrad: per view 2 x n.
template <int KS>
__global__ void __launch_bounds__(256) k_energy_grad(int V, int n, int W, int H, int dsf,
                                                     const float *__restrict__ ugrad, const float *__restrict__ vgrad,
                                                     const float *__restrict__ tau, const float *__restrict__ wgt,
                                                     float s2, int gw, double *__restrict__ partial) {
    __shared__ double red[8];
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    const size_t N = (size_t)W * H;
    double e = 0.0;
    if (m < n) {
        const float tx = tau[(size_t)v * 2 * n + m], ty = tau[(size_t)v * 2 * n + n + m];
        float ax = 0.f, ay = 0.f;
        if (in_gather(tx, ty, W, H)) {
            Footprint fp;
            footprint<KS>(tx, ty, dsf, W, H, fp);
#pragma unroll
            for (int j = 0; j < KS; ++j)
#pragma unroll
                for (int i = 0; i < KS; ++i) {
                    const int x = fp.x0 + j, y = fp.y0 + i;
                    if (0 <= x && x <= W - 1 && 0 <= y && y <= H - 1) {
                        const float A = fp.A[KS * i + j];
                        const size_t o = (size_t)y * W + x;
                        ax += A * __ldg(ugrad + o);
                        ay += A * __ldg(ugrad + N + o);
                    }
                }
        }
        const float *vg = vgrad + (size_t)v * 2 * n;
        float a = ax - vg[m], b = ay - vg[n + m];
        a = a * a;
        b = b * b;
        if (gw) {
            const float w = wgt[(size_t)v * n + m];
            a *= w;
            b *= w;
            a *= s2;
            b *= s2;
        }
        e = (double)a + (double)b;
    }
    const double s = block_sum<256>(e, red);
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

int energy_grad_partials(const Geometry &G) { return ((G.n + 255) / 256) * G.V; }

void launch_laplacian(int W, int H, int planes, const float *in, float *out, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "laplacian", st);
    k_laplacian<<<grid2(W, H, kTile), kTile, 0, st>>>(W, H, planes, in, out);
    lc.add(1);
}

void launch_residual_grad(const Geometry &G, const float *lapU, const float *img, const float *tau, const float *wgt,
                          int gw, float *resg, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "residual_grad", st);
    const dim3 b(256), g((G.n + 255) / 256, G.V);
    LFRV_KS_DISPATCH(G.dsf + 1, k_residual_grad, g, b, st, G.V, G.w, G.h, G.W, G.H, G.dsf, lapU, img, tau, wgt, gw,
                     resg);
    lc.add(1);
}

void launch_energy_grad(const Geometry &G, const float *ugrad, const float *vgrad, const float *tau, const float *wgt,
                        float s2, int gw, double *partial, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "energy_grad", st);
    const dim3 b(256), g((G.n + 255) / 256, G.V);
    LFRV_KS_DISPATCH(G.dsf + 1, k_energy_grad, g, b, st, G.V, G.n, G.W, G.H, G.dsf, ugrad, vgrad, tau, wgt, s2, gw,
                     partial);
    lc.add(1);
}

void launch_regweight(const Geometry &G, const Buckets &B, const float *tau, const float *wgt, const float *norm_prior,
                      float s2, float lmax, float lmin, float mmax, float *g0, float *norm_out, cudaStream_t st,
                      LaunchCounter &lc) {
    SplatSrc src{{wgt, nullptr, nullptr}, {(size_t)G.n, 0, 0}, nullptr};
    LFRV_KS_DISPATCH(G.dsf + 1, k_regweight, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW, B.start,
                     B.entries, tau, src, norm_prior, s2, lmax, lmin, mmax, g0, norm_out);
    lc.add(1);
}

void launch_u_gradient(const Geometry &G, const Buckets &B, const float *tau, const float *vgrad, const float *wgt,
                       float s2, float *gx, float *gy, float *mask, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "u_gradient", st);
    // vgrad: per view [2][n] (Sobel x, Sobel y); weights [V][n]
    SplatSrc src{{vgrad, vgrad + G.n, wgt}, {(size_t)2 * G.n, (size_t)2 * G.n, (size_t)G.n}, nullptr};
    LFRV_KS_DISPATCH(G.dsf + 1, k_u_gradient, grid2(G.W, G.H, kTile), kTile, st, G.W, G.H, G.n, G.dsf, B.BW, B.start,
                     B.entries, tau, src, s2, gx, gy, mask);
    lc.add(1);
}

template <int KS, typename TS>
static void gradient_setup_ks(const Geometry &G, const Buckets &B, const float *tau, const TS *img,
                              const TS *vgrad, const TS *wgt, float s2, uint8_t *vis, float *U, float *gx,
                              float *gy, float *mask, cudaStream_t st) {
    if constexpr (KS <= 3) {
        // two anchor rows per warp unless that gives the GPU fewer than two blocks per SM
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        auto launch = [&](auto rpw) {
            constexpr int RPW = decltype(rpw)::value, TY = kGrWarps * RPW - (KS - 1);
            constexpr size_t smem = gradient_rows_smem<KS, RPW>();
            static std::once_flag once;
            std::call_once(once, [] {
                cudaFuncSetAttribute(k_gradient_setup_rows<KS, TS, RPW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem);
            });
            const dim3 g((G.W + kGrTXO - 1) / kGrTXO, (G.H + TY - 1) / TY);
            k_gradient_setup_rows<KS, TS, RPW><<<g, kGrWarps * 32, smem, st>>>(
                G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, img, vgrad, wgt, s2, vis, U, gx, gy, mask);
        };
        constexpr int TY2 = kGrWarps * 2 - (KS - 1);
        if ((long long)((G.W + kGrTXO - 1) / kGrTXO) * ((G.H + TY2 - 1) / TY2) >= 2 * sms)
            launch(std::integral_constant<int, 2>{});
        else
            launch(std::integral_constant<int, 1>{});
    } else {
        k_gradient_setup_px<KS, TS><<<grid2(G.W, G.H, kTile), kTile, 0, st>>>(G.W, G.H, G.n, G.dsf, B.BW, B.start,
                                                                            B.entries, tau, img, vgrad, wgt, s2, vis,
                                                                            U, gx, gy, mask);
    }
}

template <typename TS>
static void gradient_setup_typed(const Geometry &G, const Buckets &B, const float *tau, const TS *img, const TS *vgrad,
                                 const TS *wgt, float s2, uint8_t *vis, float *U, float *gx, float *gy, float *mask,
                                 cudaStream_t st) {
    switch (G.dsf + 1) {
        case 2: gradient_setup_ks<2, TS>(G, B, tau, img, vgrad, wgt, s2, vis, U, gx, gy, mask, st); break;
        case 3: gradient_setup_ks<3, TS>(G, B, tau, img, vgrad, wgt, s2, vis, U, gx, gy, mask, st); break;
        case 4: gradient_setup_ks<4, TS>(G, B, tau, img, vgrad, wgt, s2, vis, U, gx, gy, mask, st); break;
        case 5: gradient_setup_ks<5, TS>(G, B, tau, img, vgrad, wgt, s2, vis, U, gx, gy, mask, st); break;
        default: break;
    }
}

void launch_gradient_setup(const Geometry &G, const Buckets &B, const float *tau, const void *img, const void *vgrad,
                           const void *wgt, float s2, uint8_t *vis, float *U, float *gx, float *gy, float *mask,
                           cudaStream_t st, LaunchCounter &lc, bool bf16) {
    ProfScope _ps(lc, "gradient_setup", st);
    if (bf16)
        gradient_setup_typed(G, B, tau, static_cast<const __nv_bfloat16 *>(img),
                             static_cast<const __nv_bfloat16 *>(vgrad), static_cast<const __nv_bfloat16 *>(wgt), s2,
                             vis, U, gx, gy, mask, st);
    else
        gradient_setup_typed(G, B, tau, static_cast<const float *>(img), static_cast<const float *>(vgrad),
                             static_cast<const float *>(wgt), s2, vis, U, gx, gy, mask, st);
    lc.add(1);
}

// Luminance Sobel of the views (the view path of k_sobel: no mask, zero on the border), FP32 or BF16 in and out.
// The luminance of a 32 x 32 tile and its one-pixel halo is computed once into shared memory (1.13 loads per
// pixel and plane instead of 9); each thread of a 32 x 8 block then takes four rows. The arithmetic is k_sobel's,
// so the results are the same bit for bit.
constexpr int kSobelTY = 32;

template <typename T>
__global__ void __launch_bounds__(256) k_view_sobel(int W, int H, const T *__restrict__ rgb, size_t in_stride,
                                                    size_t ch_stride, T *__restrict__ gx, T *__restrict__ gy,
                                                    size_t out_stride) {
    __shared__ float Ls[kSobelTY + 2][35];
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * kSobelTY, z = blockIdx.z;
    const T *r = rgb + (size_t)z * in_stride, *g = r + ch_stride, *b = g + ch_stride;
    const int t = threadIdx.y * 32 + threadIdx.x;
    for (int k = t; k < (kSobelTY + 2) * 34; k += 256) {
        const int ly = k / 34, lx = k - ly * 34, xx = x0 - 1 + lx, yy = y0 - 1 + ly;
        float L = 0.f;
        if (xx >= 0 && xx < W && yy >= 0 && yy < H) {
            const size_t q = (size_t)yy * W + xx;
            L = lum(ldv(r + q), ldv(g + q), ldv(b + q));
        }
        Ls[ly][lx] = L;
    }
    __syncthreads();
    const int x = x0 + threadIdx.x;
    if (x >= W) return;
#pragma unroll
    for (int j = 0; j < kSobelTY / 8; ++j) {
        const int ry = threadIdx.y + 8 * j, y = y0 + ry;
        if (y >= H) break;
        const int tx = threadIdx.x + 1, ty = ry + 1;
        float gX = 0.f, gY = 0.f;
        if (0 < x && x < W - 1 && 0 < y && y < H - 1) {
            const float Ypp = Ls[ty - 1][tx - 1], Ypc = Ls[ty - 1][tx], Ypn = Ls[ty - 1][tx + 1];
            const float Ycp = Ls[ty][tx - 1], Ycn = Ls[ty][tx + 1];
            const float Ynp = Ls[ty + 1][tx - 1], Ync = Ls[ty + 1][tx], Ynn = Ls[ty + 1][tx + 1];
            gX = (Ypn + 2.f * Ycn + Ynn - Ypp - 2.f * Ycp - Ynp) / 8.f;
            gY = (Ynp + 2.f * Ync + Ynn - Ypp - 2.f * Ypc - Ypn) / 8.f;
        }
        const size_t o = (size_t)y * W + x;
        stv(gx + (size_t)z * out_stride + o, gX);
        stv(gy + (size_t)z * out_stride + o, gY);
    }
}

void launch_view_sobel_bf16(int W, int H, int count, const void *rgb, size_t in_stride, size_t ch_stride, void *gx,
                            void *gy, size_t out_stride, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "sobel", st);
    const dim3 b(32, 8), g((W + 31) / 32, (H + kSobelTY - 1) / kSobelTY, count);
    k_view_sobel<__nv_bfloat16><<<g, b, 0, st>>>(W, H, static_cast<const __nv_bfloat16 *>(rgb), in_stride, ch_stride,
                                                 static_cast<__nv_bfloat16 *>(gx), static_cast<__nv_bfloat16 *>(gy),
                                                 out_stride);
    lc.add(1);
}

void launch_sobel(int W, int H, int count, const float *rgb, size_t in_stride, size_t ch_stride, float *gx, float *gy,
                  size_t out_stride, const uint8_t *vis, double *abs_partial, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "sobel", st);
    const dim3 b(32, 8), g((W + 31) / 32, (H + 7) / 8, count);
    if (!vis && !abs_partial) {
        const dim3 gv((W + 31) / 32, (H + kSobelTY - 1) / kSobelTY, count);
        k_view_sobel<float><<<gv, b, 0, st>>>(W, H, rgb, in_stride, ch_stride, gx, gy, out_stride);
    } else {
        k_sobel<<<g, b, 0, st>>>(W, H, rgb, in_stride, ch_stride, gx, gy, out_stride, vis, abs_partial);
    }
    lc.add(1);
}
int sobel_partials(int W, int H) { return ((W + 31) / 32) * ((H + 7) / 8); }

// Instantiations the autotuner chooses from: (iterations per super-step, threads per block).
struct RofVariant {
    int K, TY, threads;
    const void *kernel;
    size_t smem;
};
#define LFRV_ROF(K, TY, V) {K, TY, rof_threads<K, TY, V>(), (const void *)k_rof_persistent<K, TY, V>, rof_smem<K, TY, V>()}
static const RofVariant kRofVariants[] = {LFRV_ROF(4, 16, 2), LFRV_ROF(4, 16, 4),  LFRV_ROF(6, 16, 2),
                                          LFRV_ROF(8, 16, 2), LFRV_ROF(8, 32, 4),  LFRV_ROF(10, 16, 2),
                                          LFRV_ROF(6, 8, 2),  LFRV_ROF(8, 8, 2),   LFRV_ROF(4, 32, 2)};
#undef LFRV_ROF
int rof_variant_count() { return (int)(sizeof(kRofVariants) / sizeof(kRofVariants[0])); }
int rof_default_variant() { return 3; }  // K = 8, tiles of 32 x 16, two pixels per thread

// Number of super-steps of variant v for niter iterations: the result is in (U1, P1) when it is odd.
int rof_persistent_steps(int niter, int v) { return (niter + kRofVariants[v].K - 1) / kRofVariants[v].K; }

cudaError_t launch_rof_persistent(int W, int H, int niter, float tau, float sigma, float lam, float *U0, float *P0,
                                  float *U1, float *P1, const float *F, const float *g, GridBarrier gb, int v,
                                  cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "rof_persistent", st);
    const RofVariant &R = kRofVariants[v];
    cudaError_t e = cudaFuncSetAttribute(R.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R.smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, R.kernel, R.threads, R.smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int ntiles = ((W + kRofTX - 1) / kRofTX) * ((H + R.TY - 1) / R.TY);
    const int blocks = std::min(ntiles, sms * per_sm);
    void *args[] = {&W, &H, &niter, &tau, &sigma, &lam, &U0, &P0, &U1, &P1, (void *)&F, (void *)&g, &gb};
    lc.add(1);
    return cudaLaunchCooperativeKernel(R.kernel, dim3(blocks), dim3(R.threads), args, R.smem, st);
}

void launch_moving(size_t N, const float *A, const float *B, float thr, double *partial, cudaStream_t st,
                   LaunchCounter &lc) {
    k_moving<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(N, A, B, thr, partial);
    lc.add(1);
}
int moving_partials(size_t N) { return (int)((N + 255) / 256); }

void set_gaussian(const float k[11]) { cudaMemcpyToSymbol(c_gauss, k, sizeof(float) * 11); }

void launch_blur(int W, int H, const float *in, float *tmp, float *out, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "blur", st);
    const dim3 b(kBlurBX, kBlurBY);
    k_blur_rows<<<grid2(W, H, b), b, 0, st>>>(W, H, in, tmp);
    k_blur_cols<<<grid2(W, H, b), b, 0, st>>>(W, H, tmp, out);
    lc.add(2);
}

void launch_reduce_final(const ReduceLists &lists, int n, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "reduce_final", st);
    k_reduce_final<<<n, 1024, 0, st>>>(lists);
    lc.add(1);
}

void launch_reduce_final(int count, const double *partial, double *out, cudaStream_t st, LaunchCounter &lc) {
    ReduceLists l{};
    l.count[0] = count;
    l.partial[0] = partial;
    l.out[0] = out;
    launch_reduce_final(l, 1, st, lc);
}

void launch_trace_energy(const double *sums, float lambda, float alpha, float beta, bool grad, double *dst,
                         cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "trace_energy", st);
    k_trace_energy<<<1, 1, 0, st>>>(sums, lambda, alpha, beta, grad ? 1 : 0, dst);
    lc.add(1);
}

void launch_premultiply_dpart(int V, int n, const float *dpart3, int ch, float *dp, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "premultiply_dpart", st);
    k_premultiply_dpart<<<dim3((n + 255) / 256, V), 256, 0, st>>>(V, n, dpart3, ch, dp);
    lc.add(1);
}

void launch_copy_tau(int V, int n, const float *tau_in, int ch, float *tau, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "copy_tau", st);
    k_copy_tau<<<dim3((n + 255) / 256, V), 256, 0, st>>>(V, n, tau_in, ch, tau);
    lc.add(1);
}

}  // namespace lfrv

// kernels_tv.cu -- corrected IBR_color: the weighted TV_F objective solved to a certified primal-dual gap.
//
// No reference counterpart. The reference's ISTA step (sources/optimization.cu:1751-1832) normalises the data
// term's gradient by the coverage and clamps it, and reports an energy that is not its objective; in corrected mode
// the library minimises
//   E(u) = f(u) + lambda J_g(u) over [0, 1]^{3N},
//   f(u) = alpha sigma^2 / 2 sum_i sum_{m in S_i} w_im |A_i u - v_i|^2_m        (S_i: view i's splat set),
//   J_g(u) = sum_x g_x |grad u(x)|_F                                           (the TV_F of vtv_rof.cu:280-320),
// by FISTA in the diagonal metric D = max(alpha sigma^2 sum_i A_i^T w_i, 1) (a majoriser of f's Hessian: the rows
// of A_i sum to 1), each step a weighted ROF problem solved by the fast gradient projection (FGP) on its dual, and
// certifies E(u) - E* <= lambda sum_x [g_x |grad u|_F - <grad u, p>] + sum [u c - min(0, c)], c = grad f(u) -
// lambda div p. The host loop is color_solve_tv (host.cpp); the CPU restatement is oracle tv_solve.
#include "device_common.cuh"
#include "kernels.h"
#include "lfrv_internal.h"

#include <cmath>
#include <mutex>
#include <type_traits>

namespace lfrv {

constexpr float kTvDelta = 1.0f;  // floor of the metric D (pixels without data keep a proximal term)

// ------------------------------------------------------------------ per-pixel set-up
template <int KS>
__global__ void k_tv_metric(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                            const unsigned int *__restrict__ entries, const float *__restrict__ tau,
                            const float *__restrict__ wgt, float as2, float lambda, float *__restrict__ D,
                            float *__restrict__ lam) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const SplatSrc src{{wgt, wgt, wgt}, {(size_t)n, (size_t)n, (size_t)n}, nullptr};
    float acc[3], norm;
    splat_accumulate<KS, 1>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x;
    const float d = fmaxf(as2 * acc[0], kTvDelta);
    D[o] = d;
    lam[o] = lambda / d;
}

// Dual step 1 / L_x, L_x = 8 max(lam_x, lam_{x+1}, lam_{x+W}): the dual Hessian grad diag(lam) grad^T is at most
// diag(L) (each dual entry enters the divergence at two pixels, each divergence has four terms).
__global__ void k_tv_linv(int W, int H, const float *__restrict__ lam, float *__restrict__ linv) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t o = (size_t)y * W + x;
    float m = lam[o];
    if (x < W - 1) m = fmaxf(m, lam[o + 1]);
    if (y < H - 1) m = fmaxf(m, lam[o + W]);
    linv[o] = 1.0f / (8.0f * m);
}

template <int KS>
__global__ void k_tv_gradf(int W, int H, int n, int dsf, int BW, const unsigned int *__restrict__ start,
                           const unsigned int *__restrict__ entries, const float *__restrict__ tau,
                           const float *__restrict__ res, float as2, float *__restrict__ gf) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t s3 = (size_t)3 * n;
    const SplatSrc src{{res, res + n, res + 2 * (size_t)n}, {s3, s3, s3}, nullptr};
    float acc[3], norm;
    splat_accumulate<KS, 3>(x, y, W, H, n, dsf, BW, start, entries, tau, src, acc, norm);
    const size_t o = (size_t)y * W + x, N = (size_t)W * H;
#pragma unroll
    for (int c = 0; c < 3; ++c) gf[c * N + o] = as2 * acc[c];
}

// A plane of the dual in FP64: it is stored as an unevaluated sum of two floats, the six high planes, then the six low
// ones (12 N floats). The low planes cost nothing where the arithmetic is FP32, and no load or store of the inner
// iterations converts (a conversion holds this GPU's narrow FP64 pipe for 16 cycles a warp: with FP64 storage the
// conversions were a third of the FP32 iterations' time).
struct TvDualPlane {
    const float *hi, *lo;
    __device__ __forceinline__ TvDualPlane(const float *P, int plane, size_t N) : hi(P + plane * N), lo(P + (6 + plane) * N) {}
    __device__ __forceinline__ double operator[](size_t o) const { return (double)hi[o] + (double)lo[o]; }
};

// div of a dual field at (x, y): the negative adjoint of the forward gradient with zero at the last column / row.
__device__ __forceinline__ double tv_div(const TvDualPlane &px, const TvDualPlane &py, int W, int H, int x, int y,
                                         size_t o) {
    double d = 0;
    if (x < W - 1) d += px[o];
    if (x > 0) d -= px[o - 1];
    if (y < H - 1) d += py[o];
    if (y > 0) d -= py[o - W];
    return d;
}

// ------------------------------------------------------------------ certificate
// One-dimensional blocks of kGapBX * kGapBY threads (block_sum indexes warps by threadIdx.x), each covering a
// kGapBX x kGapBY patch of pixels.
constexpr int kGapBX = 32, kGapBY = 8;
__global__ void __launch_bounds__(kGapBX * kGapBY) k_tv_gap(int W, int H, const float *__restrict__ u,
                                                            const float *__restrict__ gf, const float *__restrict__ P,
                                                            const float *__restrict__ g, float lambda,
                                                            double *__restrict__ partial) {
    __shared__ double red[kGapBX * kGapBY / 32];
    const int x = blockIdx.x * kGapBX + (int)(threadIdx.x % kGapBX);
    const int y = blockIdx.y * kGapBY + (int)(threadIdx.x / kGapBX);
    const size_t N = (size_t)W * H;
    double tv = 0.0, inner = 0.0, box = 0.0;
    if (x < W && y < H) {
        const size_t o = (size_t)y * W + x;
        double n2 = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float *uc = u + c * N;
            const double gxv = x < W - 1 ? (double)uc[o + 1] - (double)uc[o] : 0.0;
            const double gyv = y < H - 1 ? (double)uc[o + W] - (double)uc[o] : 0.0;
            n2 += gxv * gxv + gyv * gyv;
            const TvDualPlane px(P, c, N), py(P, 3 + c, N);
            inner += gxv * px[o] + gyv * py[o];
            const double cc = (double)gf[c * N + o] - (double)lambda * tv_div(px, py, W, H, x, y, o);
            box += (double)uc[o] * cc - fmin(0.0, cc);
        }
        tv = (double)g[o] * sqrt(n2);
    }
    const int b = blockIdx.y * gridDim.x + blockIdx.x, nb = gridDim.x * gridDim.y;
    const double s0 = block_sum<kGapBX * kGapBY>(tv, red);
    if (threadIdx.x == 0) partial[b] = s0;
    const double s1 = block_sum<kGapBX * kGapBY>(inner, red);
    if (threadIdx.x == 0) partial[nb + b] = s1;
    const double s2 = block_sum<kGapBX * kGapBY>(box, red);
    if (threadIdx.x == 0) partial[2 * nb + b] = s2;
}

__global__ void k_tv_fstep(size_t N, const float *__restrict__ u, const float *__restrict__ up,
                           const float *__restrict__ gf, const float *__restrict__ gfp, const float *__restrict__ D,
                           float theta_arg, const TvLoopState *__restrict__ loop, float *__restrict__ F) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * N) return;
    const float theta = loop ? loop->theta : theta_arg;
    const float y = u[i] + theta * (u[i] - up[i]);
    const float gy = (1.0f + theta) * gf[i] - theta * gfp[i];
    F[i] = y - gy / D[i % N];
}

__global__ void k_tv_clamp(size_t n, const float *__restrict__ in, float *__restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = fminf(1.0f, fmaxf(0.0f, in[i]));
}

// ------------------------------------------------------------------ FGP on the weighted ROF dual
// One cooperative launch runs every inner iteration. Temporally blocked: a block takes a tile and a halo of K
// pixels and runs K iterations on that region before it writes the tile back and the grid synchronises (each
// iteration's dependence reaches one pixel in each direction, diagonals included, so the tile stays exact; the
// updated part of the region shrinks by a pixel per iteration to what the tile still depends on). Per iteration:
//   u = clamp(F + lam div q, 0, 1);  p' = proj_{|.|_F <= g}(q + grad u / L);  q = p' + beta_j (p' - p);  p = p'
// with beta_j = (s_j - 1) / s_{j+1}, s_0 = 1, s_{j+1} = (1 + sqrt(1 + 4 s_j^2)) / 2 (Beck and Teboulle's FGP).
// A thread owns V vertically adjacent pixels throughout: their q, p, u, F, lam, 1/L and g stay in registers, the
// neighbours above and below come from registers except at the ends, and shared memory carries u, the x components of q
// and the y components of each thread's last pixel. As in the persistent ROF no pixel has a branch for the image: a dual
// whose difference does not exist starts at 0 and has step 0, a block with one tile reads back only the halo, and threads
// the tile no longer depends on skip the iteration.
// The dual p and the momentum point q are stored as pairs of floats (TvDualPlane); u, F, lam, 1/L and g are FP32. TD is
// the dual's arithmetic type. In FP32 the dual's rounding (a few ulp of |p| <= g) leaves lambda div p, and with it the
// certificate's box term, a noise floor near 4e-4 relative at 256^2; with the double-float type below (about 44
// bits) the certificate reaches 1e-4, as with FP64 (the oracle's FP32 mirror shows the floor, its FP64 dual does
// not). FP64 arithmetic is slow on this GPU's narrow FP64 pipe and double-float costs several FP32 operations per
// operation, so the host runs TD = float while the gap is far above its floor and TD = dfloat to finish.
// 256^2, 200 iterations: FP32 640 -> 228 us, double-float 1890 -> 754, against FP64 storage and momentum weights
// converted by every thread in every iteration.
// Double-float arithmetic (an unevaluated sum hi + lo of two floats, about 44 significant bits): the dual's
// arithmetic where FP32 would leave its noise floor, on the FP32 pipes. Sums use the error-free two-sum (Knuth)
// and products the FMA-based two-product (Dekker's splitting replaced by fmaf), each renormalised with the
// fast two-sum; the add is the accurate form (both parts' errors carried), since p' - p cancels.
struct dfloat {
    float hi, lo;
    __device__ __forceinline__ dfloat() : hi(0.f), lo(0.f) {}
    __device__ __forceinline__ dfloat(int v) : hi((float)v), lo(0.f) {}
    __device__ __forceinline__ dfloat(float v) : hi(v), lo(0.f) {}
    __device__ __forceinline__ dfloat(float h, float l) : hi(h), lo(l) {}
    __device__ __forceinline__ explicit operator float() const { return hi + lo; }
};
__device__ __forceinline__ dfloat df_fast_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return dfloat(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ dfloat df_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return dfloat(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb)));
}
__device__ __forceinline__ dfloat operator+(dfloat a, dfloat b) {
    dfloat s = df_two_sum(a.hi, b.hi);
    const dfloat t = df_two_sum(a.lo, b.lo);
    s.lo = __fadd_rn(s.lo, t.hi);
    s = df_fast_two_sum(s.hi, s.lo);
    s.lo = __fadd_rn(s.lo, t.lo);
    return df_fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ dfloat operator-(dfloat a) { return dfloat(-a.hi, -a.lo); }
__device__ __forceinline__ dfloat operator-(dfloat a, dfloat b) { return a + (-b); }
__device__ __forceinline__ dfloat operator*(dfloat a, dfloat b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return df_fast_two_sum(p, e);
}
__device__ __forceinline__ dfloat &operator+=(dfloat &a, dfloat b) { return a = a + b; }
__device__ __forceinline__ dfloat &operator-=(dfloat &a, dfloat b) { return a = a - b; }
__device__ __forceinline__ bool operator>(dfloat a, dfloat b) { return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo); }
// a + b for a float b (no cancellation concerns: one two-sum, the low part added, renormalised)
__device__ __forceinline__ dfloat df_add_f(dfloat a, float b) {
    const dfloat s = df_two_sum(a.hi, b);
    return df_fast_two_sum(s.hi, __fadd_rn(s.lo, a.lo));
}
// a + b where the sum cannot cancel (both of one sign, or b much smaller): the low parts are added in float
__device__ __forceinline__ dfloat df_add_sloppy(dfloat a, dfloat b) {
    const dfloat s = df_two_sum(a.hi, b.hi);
    return df_fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
// a0 - a1 + a2 - a3 rounded to float: the high parts' sums are exact (two-sum), their errors and the low parts
// are added in float, so the result carries an error of about one float ulp of itself (not of the terms)
__device__ __forceinline__ float df_div4(dfloat a0, dfloat a1, dfloat a2, dfloat a3) {
    const dfloat h1 = df_two_sum(a0.hi, -a1.hi), h2 = df_two_sum(a2.hi, -a3.hi), h = df_two_sum(h1.hi, h2.hi);
    const float lo = __fadd_rn(__fsub_rn(a0.lo, a1.lo), __fsub_rn(a2.lo, a3.lo));
    return __fadd_rn(h.hi, __fadd_rn(__fadd_rn(__fadd_rn(h1.lo, h2.lo), h.lo), lo));
}

constexpr int kFgpTX = 32;
template <int K, int TY, int V>
__host__ __device__ constexpr int fgp_threads() {
    return ((kFgpTX + 2 * K) * ((TY + 2 * K) / V) + 31) / 32 * 32;
}
// a plane of the region with one row more and a cell on either side; of the segments' last pixels
template <int K, int TY, int V>
__host__ __device__ constexpr int fgp_plane() {
    return (kFgpTX + 2 * K) * (TY + 2 * K + 1) + 2;
}
template <int K, int TY, int V>
__host__ __device__ constexpr int fgp_plane_y() {
    return (kFgpTX + 2 * K) * ((TY + 2 * K) / V + 1);
}
template <typename TD, int K, int TY, int V>
constexpr size_t fgp_smem() {
    return sizeof(TD) * 3 * (size_t)(fgp_plane<K, TY, V>() + fgp_plane_y<K, TY, V>()) +
           sizeof(float) * 3 * (size_t)fgp_plane<K, TY, V>();
}

// The momentum weights beta_j of the first kFgpBetaTable iterations (high and low float of the FP64 value).
constexpr int kFgpBetaTable = 256;
static_assert(kTvInnerIterations <= kFgpBetaTable, "a launch stays within the table");
__constant__ float2 c_fgp_beta[kFgpBetaTable];

void set_fgp_beta() {
    float2 t[kFgpBetaTable];
    double s = 1.0;
    for (int j = 0; j < kFgpBetaTable; ++j) {
        const double s1 = 0.5 * (1.0 + std::sqrt(1.0 + 4.0 * s * s)), b = (s - 1.0) / s1;
        t[j].x = (float)b;
        t[j].y = (float)(b - (double)t[j].x);
        s = s1;
    }
    cudaMemcpyToSymbol(c_fgp_beta, t, sizeof(t));
}

__device__ __forceinline__ void fgp_load(const float *P, size_t i, size_t lo, float &v) { v = __ldcg(P + i); }
__device__ __forceinline__ void fgp_load(const float *P, size_t i, size_t lo, dfloat &v) {
    v = dfloat(__ldcg(P + i), __ldcg(P + i + lo));
}
__device__ __forceinline__ void fgp_store(float *P, size_t i, size_t lo, float v) { P[i] = v; }
__device__ __forceinline__ void fgp_store(float *P, size_t i, size_t lo, dfloat v) {
    P[i] = v.hi;
    P[i + lo] = v.lo;
}
__device__ __forceinline__ void fgp_beta(int j, float &b) { b = c_fgp_beta[j].x; }
__device__ __forceinline__ void fgp_beta(int j, dfloat &b) { b = dfloat(c_fgp_beta[j].x, c_fgp_beta[j].y); }

template <typename TD, int K, int TY, int V>
__global__ void __launch_bounds__((fgp_threads<K, TY, V>())) k_tv_fgp(int W, int H, int niter,
                                                                      const float *__restrict__ F,
                                                                      const float *__restrict__ lam,
                                                                      const float *__restrict__ linv,
                                                                      const float *__restrict__ g, float *P0, float *P1,
                                                                      float *Q0, float *Q1, float *__restrict__ U,
                                                                      GridBarrier gb) {
    constexpr bool DF = std::is_same<TD, dfloat>::value;
    constexpr int RX = kFgpTX + 2 * K, RY = TY + 2 * K;
    static_assert(RY % V == 0, "whole segments");
    constexpr int PL = fgp_plane<K, TY, V>(), PY = fgp_plane_y<K, TY, V>();
    extern __shared__ __align__(16) unsigned char fgp_sm[];
    TD *sQ = reinterpret_cast<TD *>(fgp_sm);
    float *sF = reinterpret_cast<float *>(sQ + 3 * (PL + PY));
    const int seg = threadIdx.x / RX, lx = threadIdx.x - seg * RX, ly0 = seg * V;
    const bool mine = seg < RY / V;
    TD *sQx = sQ + 1 + ly0 * RX + lx;                   // this thread's first pixel, plane 0
    TD *sQy = sQ + 3 * PL + (seg + 1) * RX + lx;        // its last pixel; - RX: the segment above
    float *sU = sF + 1 + ly0 * RX + lx;
    const int tiles_x = (W + kFgpTX - 1) / kFgpTX, ntiles = tiles_x * ((H + TY - 1) / TY);
    const bool resident = ntiles <= (int)gridDim.x;  // one tile per block
    const size_t N = (size_t)W * H, lo = 6 * N;
    // distance of the segment's column and of its nearest row from the tile
    const int dx = max(max(K - lx, lx - (K + kFgpTX - 1)), 0);
    const int dist = max(dx, max(max(K - (ly0 + V - 1), ly0 - (K + TY - 1)), 0));
    const bool tile_x = mine && lx >= K && lx < K + kFgpTX;
    // shared memory that no thread writes (pads) is read too: finite from here on
    for (int i = threadIdx.x; i < 3 * (PL + PY); i += blockDim.x) sQ[i] = TD(0);
    for (int i = threadIdx.x; i < 3 * PL; i += blockDim.x) sF[i] = 0.f;
    __syncthreads();
    unsigned int gen = 0;
    int step = 0;
    TD q[V][6], p[V][6];
    float f[V][3], u[V][3], lm[V], lx_inv[V], ly_inv[V], gg[V];
    for (int done = 0; done < niter; done += K, ++step) {
        const int iters = min(K, niter - done);
        const float *Pi = (step & 1) ? P1 : P0;
        float *Po = (step & 1) ? P0 : P1;
        const float *Qi = step == 0 ? P0 : ((step & 1) ? Q1 : Q0);  // q starts at p
        float *Qo = (step & 1) ? Q0 : Q1;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int gx = (t % tiles_x) * kFgpTX - K + lx, gy0 = (t / tiles_x) * TY - K + ly0;
            const bool inx = mine && gx >= 0 && gx < W;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int gy = gy0 + k;
                const bool in = inx && gy >= 0 && gy < H;
                const bool own = tile_x && ly0 + k >= K && ly0 + k < K + TY;
                const size_t o = in ? (size_t)gy * W + gx : 0;
                if (step == 0 || !resident) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) f[k][c] = in ? __ldg(F + c * N + o) : 0.f;
                    lm[k] = in ? __ldg(lam + o) : 0.f;
                    const float li = in ? __ldg(linv + o) : 0.f;
                    lx_inv[k] = gx < W - 1 ? li : 0.f;
                    ly_inv[k] = gy < H - 1 ? li : 0.f;
                    gg[k] = in ? __ldg(g + o) : 0.f;
                }
                if (step == 0 || !resident || !own) {
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        q[k][c] = p[k][c] = TD(0);
                        if (in) {
                            fgp_load(Qi, c * N + o, lo, q[k][c]);
                            fgp_load(Pi, c * N + o, lo, p[k][c]);
                        }
                    }
                }
                if (mine) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sQx[c * PL + k * RX] = q[k][c];
                }
            }
            if (mine) {
#pragma unroll
                for (int c = 0; c < 3; ++c) sQy[c * PY] = q[V - 1][3 + c];
            }
            __syncthreads();
            for (int it = 0; it < iters; ++it) {
                TD beta;
                fgp_beta(done + it, beta);
                // u(q) where the tile still depends on it (values next to the region's edge are stale and stay
                // outside the tile)
                if (mine && dist <= iters - it) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        TD above = sQy[c * PY - RX];
#pragma unroll
                        for (int k = 0; k < V; ++k) {
                            const TD left = sQx[c * PL + k * RX - 1];
                            float dv;
                            if constexpr (DF) dv = df_div4(q[k][c], left, q[k][3 + c], above);
                            else dv = __fsub_rn(__fadd_rn(__fsub_rn(q[k][c], left), q[k][3 + c]), above);
                            above = q[k][3 + c];
                            u[k][c] = fminf(1.0f, fmaxf(0.0f, __fmaf_rn(lm[k], dv, f[k][c])));
                            sU[c * PL + k * RX] = u[k][c];
                        }
                    }
                }
                __syncthreads();
                // p' = proj(q + grad u / L), q = p' + beta (p' - p) (own pixel)
                if (mine && dist <= iters - it - 1) {
#pragma unroll
                    for (int k = 0; k < V; ++k) {
                        TD v[6];
                        TD n2 = TD(0);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float ur = sU[c * PL + k * RX + 1];
                            const float ud = k + 1 < V ? u[k + 1 < V ? k + 1 : k][c] : sU[c * PL + V * RX];
                            const float gxv = ur - u[k][c], gyv = ud - u[k][c];
                            if constexpr (DF) {
                                v[c] = df_add_f(q[k][c], gxv * lx_inv[k]);
                                v[3 + c] = df_add_f(q[k][3 + c], gyv * ly_inv[k]);
                                n2 = df_add_sloppy(df_add_sloppy(n2, v[c] * v[c]), v[3 + c] * v[3 + c]);
                            } else {
                                // (the fusions written out: the stop test's step count hangs on these roundings)
                                v[c] = __fmaf_rn(gxv, lx_inv[k], q[k][c]);
                                v[3 + c] = __fmaf_rn(gyv, ly_inv[k], q[k][3 + c]);
                                n2 = __fadd_rn(n2, __fmaf_rn(v[c], v[c], __fmul_rn(v[3 + c], v[3 + c])));
                            }
                        }
                        // projection onto |p| <= g without a square root or division: r = 1 / sqrt(n2) from the FP32
                        // estimate, in double-float with a Newton step in FP32 and one in TD (relative error ~1e-14),
                        // applied only where the ball constraint is active
                        const TD gv = TD(gg[k]);
                        if (n2 > gv * gv) {
                            TD sc;
                            if constexpr (DF) {
                                const float n = (float)n2, e = rsqrtf(n), r0 = fmaf(e * 0.5f, fmaf(-n * e, e, 1.f), e);
                                // r0 + r0 (1 - n2 r0^2) / 2: the residual is small, so FP32 carries it
                                const dfloat h = n2 * (dfloat(r0) * dfloat(r0));
                                const float d = __fsub_rn(__fsub_rn(1.f, h.hi), h.lo);
                                sc = gv * df_fast_two_sum(r0, __fmul_rn(0.5f * r0, d));
                            } else {
                                sc = gv * rsqrtf(n2);
                            }
#pragma unroll
                            for (int c = 0; c < 6; ++c) v[c] = v[c] * sc;
                        }
#pragma unroll
                        for (int c = 0; c < 6; ++c) {
                            const TD pn = v[c];
                            if constexpr (DF) q[k][c] = df_add_sloppy(pn, beta * (pn - p[k][c]));
                            else q[k][c] = __fmaf_rn(beta, __fsub_rn(pn, p[k][c]), pn);
                            p[k][c] = pn;
                        }
#pragma unroll
                        for (int c = 0; c < 3; ++c) sQx[c * PL + k * RX] = q[k][c];
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) sQy[c * PY] = q[V - 1][3 + c];
                }
                __syncthreads();
            }
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const int gy = gy0 + k;
                if (!(tile_x && inx && ly0 + k >= K && ly0 + k < K + TY && gy < H)) continue;
                const size_t o = (size_t)gy * W + gx;
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    fgp_store(Po, c * N + o, lo, p[k][c]);
                    fgp_store(Qo, c * N + o, lo, q[k][c]);
                }
            }
        }
        if (!grid_sync(gb, gen)) return;
    }
    // the final dual sits in P0 after an even number of super-steps, else in P1; u = clamp(F + lam div p). In FP32 its
    // low planes are 0, which the solve left in P0 alone
    const int steps = (niter + K - 1) / K;
    const float *Pf = (steps & 1) ? P1 : P0;
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t o = first; o < N; o += stride) {
        const int x = (int)(o % W), y = (int)(o / W);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float *px = Pf + c * N, *py = Pf + (3 + c) * N;
            double d = 0.0;
            auto add = [&](const float *v, double sign) {
                d += sign * (double)__ldcg(v);
                if constexpr (DF) d += sign * (double)__ldcg(v + lo);
            };
            if (x < W - 1) add(px + o, 1.0);
            if (x > 0) add(px + o - 1, -1.0);
            if (y < H - 1) add(py + o, 1.0);
            if (y > 0) add(py + o - W, -1.0);
            U[c * N + o] = fminf(1.0f, fmaxf(0.0f, F[c * N + o] + lam[o] * (float)d));
        }
    }
    // the caller keeps its dual in P0
    if (steps & 1)
        for (size_t i = first; i < (DF ? 2 : 1) * lo; i += stride) P0[i] = __ldcg(P1 + i);
    if (!DF)
        for (size_t i = first; i < lo; i += stride) P0[lo + i] = 0.f;
}

// ------------------------------------------------------------------ launchers
static inline dim3 tv_grid(int W, int H, dim3 b) { return dim3((W + b.x - 1) / b.x, (H + b.y - 1) / b.y); }

void launch_tv_metric(const Geometry &G, const Buckets &B, const float *tau, const float *wgt, float as2, float lambda,
                      float *D, float *lam, float *linv, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "tv_metric", st);
    const dim3 b(32, 8), g = tv_grid(G.W, G.H, b);
    LFRV_KS_DISPATCH(G.dsf + 1, k_tv_metric, g, b, st, G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, wgt,
                     as2, lambda, D, lam);
    k_tv_linv<<<g, b, 0, st>>>(G.W, G.H, lam, linv);
    lc.add(2);
}

void launch_tv_gradf(const Geometry &G, const Buckets &B, const float *tau, const float *res, float as2, float *gf,
                     cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "tv_gradf", st);
    const dim3 b(32, 8), g = tv_grid(G.W, G.H, b);
    LFRV_KS_DISPATCH(G.dsf + 1, k_tv_gradf, g, b, st, G.W, G.H, G.n, G.dsf, B.BW, B.start, B.entries, tau, res, as2,
                     gf);
    lc.add(1);
}

int tv_gap_partials(int W, int H) { return ((W + kGapBX - 1) / kGapBX) * ((H + kGapBY - 1) / kGapBY); }

void launch_tv_gap(int W, int H, const float *u, const float *gf, const float *P, const float *g, float lambda,
                   double *partial, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "tv_gap", st);
    const dim3 gr = tv_grid(W, H, dim3(kGapBX, kGapBY));
    k_tv_gap<<<gr, kGapBX * kGapBY, 0, st>>>(W, H, u, gf, P, g, lambda, partial);
    lc.add(1);
}

void launch_tv_fstep(int W, int H, const float *u, const float *up, const float *gf, const float *gfp, const float *D,
                     float theta, float *F, cudaStream_t st, LaunchCounter &lc, const TvLoopState *loop) {
    ProfScope _ps(lc, "tv_fstep", st);
    const size_t N = (size_t)W * H;
    k_tv_fstep<<<(unsigned)((3 * N + 255) / 256), 256, 0, st>>>(N, u, up, gf, gfp, D, theta, loop, F);
    lc.add(1);
}

// The stop test and momentum update of the corrected IBR_color solve on the device (TvSolve::decide and the scalar
// part of TvSolve::step, the same double arithmetic), for a solve whose loop runs as a conditional graph: one
// thread reads the certificate sums, records the energy, decides, and sets the loop's and the arithmetic's
// conditions.
__global__ void k_tv_decide(const double *__restrict__ sums, double dt_alpha, double lambda, double tol, int niter,
                            double extended_below, TvLoopState *loop, double *trace, int trace_cap,
                            cudaGraphConditionalHandle h_loop, cudaGraphConditionalHandle h_extended) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double f = 0.5 * dt_alpha * sums[1];
    const double E = f + lambda * sums[4];
    const double gap_abs = lambda * (sums[4] - sums[5]) + sums[6];
    const double gap = E > 0 ? gap_abs / E : 1e300;
    if (trace && loop->trace_pos < trace_cap) trace[loop->trace_pos++] = E;
    bool done = loop->k >= niter || (tol > 0 && gap <= tol);
    if (!isfinite(E) || !isfinite(gap)) {
        loop->err = 1;
        done = true;
    }
    loop->E = E;
    loop->gap = gap;
    if (!done) {
        if (E > loop->E_prev) loop->t = 1.0;  // function-value restart of the momentum
        loop->E_prev = E;
        const double t = loop->t, t1 = 0.5 * (1.0 + sqrt(1.0 + 4.0 * t * t));
        loop->theta = (float)((t - 1.0) / t1);
        loop->t = t1;
        loop->extended = loop->extended || gap < extended_below;
        loop->k += 1;
    }
    loop->done = done ? 1 : 0;
    cudaGraphSetConditional(h_loop, done ? 0u : 1u);
    cudaGraphSetConditional(h_extended, loop->extended ? 1u : 0u);
}

void launch_tv_decide(const double *sums, double dt_alpha, double lambda, double tol, int niter, TvLoopState *loop,
                      double *trace, int trace_cap, cudaGraphConditionalHandle h_loop,
                      cudaGraphConditionalHandle h_extended, cudaStream_t st, LaunchCounter &lc) {
    k_tv_decide<<<1, 32, 0, st>>>(sums, dt_alpha, lambda, tol, niter, kTvExtendedBelow, loop, trace, trace_cap, h_loop,
                                  h_extended);
    lc.add(1);
}

void launch_tv_clamp(size_t n, const float *in, float *out, cudaStream_t st, LaunchCounter &lc) {
    ProfScope _ps(lc, "tv_clamp", st);
    k_tv_clamp<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, in, out);
    lc.add(1);
}

// Instantiations the FGP autotuner chooses from, per arithmetic: iterations per super-step K, tile rows TY, pixels per
// thread V. All give the same iterates.
struct FgpVariant {
    int TY, threads;
    const void *kernel;
    size_t smem;
};
#define LFRV_FGP(TD, K, TY, V) \
    {TY, fgp_threads<K, TY, V>(), (const void *)k_tv_fgp<TD, K, TY, V>, fgp_smem<TD, K, TY, V>()}
static const FgpVariant kFgpFloat[] = {LFRV_FGP(float, 4, 16, 2), LFRV_FGP(float, 6, 16, 2), LFRV_FGP(float, 8, 16, 2),
                                       LFRV_FGP(float, 8, 8, 2), LFRV_FGP(float, 6, 32, 4)};
static const FgpVariant kFgpDfloat[] = {LFRV_FGP(dfloat, 2, 16, 1), LFRV_FGP(dfloat, 2, 16, 2),
                                        LFRV_FGP(dfloat, 4, 16, 2), LFRV_FGP(dfloat, 4, 8, 1),
                                        LFRV_FGP(dfloat, 6, 16, 2)};
#undef LFRV_FGP
int tv_fgp_variant_count(bool extended) {
    return (int)(extended ? sizeof(kFgpDfloat) / sizeof(FgpVariant) : sizeof(kFgpFloat) / sizeof(FgpVariant));
}
int tv_fgp_default_variant(bool extended) { return 2; }

cudaError_t launch_tv_fgp(int W, int H, int niter, const float *F, const float *lam, const float *linv, const float *g,
                          float *P0, float *P1, float *Q0, float *Q1, float *U, GridBarrier gb, cudaStream_t st,
                          LaunchCounter &lc, bool extended, int variant) {
    if (niter > kFgpBetaTable) return cudaErrorInvalidValue;
    ProfScope _ps(lc, extended ? "tv_fgp_df" : "tv_fgp", st);
    if (variant < 0 || variant >= tv_fgp_variant_count(extended)) variant = tv_fgp_default_variant(extended);
    const FgpVariant &R = extended ? kFgpDfloat[variant] : kFgpFloat[variant];
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    static std::mutex mu;
    static bool attr_set[64] = {};
    if (dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            for (const FgpVariant &v : kFgpFloat)
                cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem);
            for (const FgpVariant &v : kFgpDfloat)
                cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem);
            attr_set[dev] = true;
        }
    }
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, R.kernel, R.threads, R.smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int ntiles = ((W + kFgpTX - 1) / kFgpTX) * ((H + R.TY - 1) / R.TY);
    const int resident = sms * per_sm;
    // as few blocks as keep the per-block tile count at its minimum (no block waits for a straggler's extra tile)
    const int per_block = (ntiles + resident - 1) / resident;
    const int blocks = std::max(1, (ntiles + per_block - 1) / per_block);
    void *args[] = {&W, &H, &niter, (void *)&F, (void *)&lam, (void *)&linv, (void *)&g, &P0, &P1, &Q0, &Q1, &U, &gb};
    lc.add(1);
    return cudaLaunchCooperativeKernel(R.kernel, dim3(blocks), dim3(R.threads), args, R.smem, st);
}

}  // namespace lfrv

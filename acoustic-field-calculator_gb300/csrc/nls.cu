// Nonlinear least-squares phase retrieval on the device: gradient descent, Gauss-Newton and
// Levenberg-Marquardt (acoustic-field-optimizer/src/multiple_foci/nls/{gradient_descent,
// gauss_newton,lm}.rs, with the shared helpers of nls/macros.rs:16-58).
//
// The reference builds B = [G | -diag(amps)] (m x N, N = n + m), the dense N x N matrix
// BhB = B^H B, and per iteration JtJ = Re(BhB o T T^H), Jtf = column sums of Im(BhB o T T^H)
// (T = exp(-i x)), F(x) = Re(t^H BhB t) (t = exp(i x)), solving N x N systems by QR (LM) or
// an SVD pseudo-inverse (Gauss-Newton).  B has only m rows, so every one of those is low rank
// and is evaluated here from B itself (the identities are exact, not approximations):
//     r = B t,  Jtf_b = Im(t_b conj((B^H r)_b)),  F = |r|^2,
//     JtJ = U^T U with U = [Re C; Im C], C = B diag(t)   (2m x N),
//     (JtJ + mu I)^-1 g = (g - U^T (mu I + U U^T)^-1 U g) / mu          (Woodbury, LM),
//     pinv(JtJ) g = U^T sum_{lambda_k > eps} w_k w_k^T U g / lambda_k^2  (U U^T = W Lambda W^T, GN),
//     U U^T from K = B B^H (fixed) and L = sum_b B_ib B_jb t_b^2.
// The device does the O(N m) and O(N m^2) work in f32 (four launches over the whole GPU per
// Gauss-Newton or LM step; gradient descent's whole loop runs in one launch); the 2m x 2m solves
// and the control flow of the reference's loops run on the host in double.
//
// A step is bound by the latency of that loop, not by its work (996 sources x 16 foci: 0.3 us of
// flops).  Its launches are programmatic dependents of each other, its results are stored straight
// into pinned memory, and it evaluates everything the next step may need at the trial point, so
// that a step takes one wait of the host: an accepted trial becomes the current point by name,
// a rejected one leaves the current point's results as they are.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "afc_internal.h"
#include "afc_solvers.h"
#include "propagate.cuh"

namespace afc {
namespace {

constexpr int kNlsThreads = 1024;

// Parameters of nls/{gradient_descent,gauss_newton,lm}.rs.
constexpr float kGdEps = 1e-6f;       // gradient_descent.rs:17
constexpr int kGdIterations = 10000;  // gradient_descent.rs:18
constexpr double kNlsEps1 = 1e-8;     // gauss_newton.rs:17, lm.rs:17
constexpr double kNlsEps2 = 1e-8;     // gauss_newton.rs:18, lm.rs:18
constexpr double kLmTau = 1e-3;       // lm.rs:19
constexpr int kNlsIterations = 200;   // gauss_newton.rs:19, lm.rs:20
constexpr double kPinvEps = 1e-3;     // gauss_newton.rs:64 (pseudo_inverse(1e-3))

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ float2 warp_sum2(float2 v) {
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide sum / max (kNlsThreads threads); `red` holds 32 floats.
__device__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    v = lane < (kNlsThreads >> 5) ? red[lane] : 0.f;
    return warp_sum(v);
}

__device__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    v = lane < (kNlsThreads >> 5) ? red[lane] : -__int_as_float(0x7f800000);
    return warp_max(v);
}

// t_b = exp(i x_b) for the N parameters.
__device__ void phasors(const float* x, int64_t N, float2* t) {
    for (int64_t b = threadIdx.x; b < N; b += blockDim.x) {
        float s, c;
        sincosf(x[b], &s, &c);
        t[b] = make_float2(c, s);
    }
}

// r = B t: warp per row i (G row i, then -amps_i t_{n+i}).
__device__ void b_times(const float2* g, const float* amps, int64_t n, int64_t m, const float2* t,
                        float2* r) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int64_t i = wid; i < m; i += nw) {
        float2 acc = make_float2(0.f, 0.f);
        for (int64_t a = lane; a < n; a += 32) {
            const float2 v = cmul(g[i * n + a], t[a]);
            acc.x += v.x;
            acc.y += v.y;
        }
        acc = warp_sum2(acc);
        if (lane == 0) {
            const float2 p = t[n + i];
            r[i] = make_float2(acc.x - amps[i] * p.x, acc.y - amps[i] * p.y);
        }
    }
}

// Jtf_b = Im(t_b conj((B^H r)_b)); returns the thread's largest Jtf.
__device__ float gradient(const float2* g, const float* amps, int64_t n, int64_t m,
                          const float2* t, const float2* r, float* jtf) {
    float mx = -__int_as_float(0x7f800000);
    for (int64_t b = threadIdx.x; b < n + m; b += blockDim.x) {
        float2 w;
        if (b < n) {
            w = make_float2(0.f, 0.f);
            for (int64_t i = 0; i < m; ++i) {
                const float2 a = g[i * n + b], q = r[i];
                // conj(a) q
                w.x += a.x * q.x + a.y * q.y;
                w.y += a.x * q.y - a.y * q.x;
            }
        } else {
            const int64_t i = b - n;
            w = make_float2(-amps[i] * r[i].x, -amps[i] * r[i].y);
        }
        const float2 tb = t[b];
        const float v = tb.y * w.x - tb.x * w.y;
        jtf[b] = v;
        mx = fmaxf(mx, v);
    }
    return mx;
}

// Gradient descent (gradient_descent.rs:31-59) in one block: x <- x - 0.1 Jtf until
// max(Jtf) <= 1e-6 or 10000 steps.  t (N), r (m), jtf (N) are workspace; *iters receives the
// number of steps taken.
__global__ void __launch_bounds__(kNlsThreads)
    nls_gd_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n,
                  int64_t m, float* x, float2* t, float2* r, float* jtf, int max_iter, float eps,
                  int* iters) {
    __shared__ float red[32];
    const int64_t N = n + m;
    int it = 0;
    for (; it < max_iter; ++it) {
        phasors(x, N, t);
        __syncthreads();
        b_times(g, amps, n, m, t, r);
        __syncthreads();
        const float mx = block_max(gradient(g, amps, n, m, t, r, jtf), red);
        if (mx <= eps) break;  // uniform: every thread holds the block maximum
        for (int64_t b = threadIdx.x; b < N; b += blockDim.x)
            x[b] = __fsub_rn(x[b], __fmul_rn(0.1f, jtf[b]));
        __syncthreads();
    }
    if (threadIdx.x == 0) *iters = it;
}

// ---- one Gauss-Newton / LM step (nls_point -> nls_rows -> nls_gradient -> nls_finish): a new
// point x and everything the next step needs at it: t, r, Jtf and, for the host, F = |r|^2,
// max(Jtf), |x|^2, U Jtf (2m: Re rows then Im rows) and L_ij = sum_b B_ib B_jb t_b^2.  Each sum has
// one fixed order (a warp's 32 lanes strided over the columns and a butterfly, or 1,024 threads
// strided and block_sum): the iterations magnify rounding into different local optima, so a split
// of the work must not change the order of a sum.

// A lane's next kAhead elements b, b + 32, ... of a row of n, all on their way before the first is
// used: left to the compiler, the loops below keep a few registers of loads in flight and wait for L2
// at every turn (996 sources x 16 foci: nls_rows 10.3 us, with this and blocks of two warps 4.0).  Gradient
// descent's block of 1,024 threads lacks the registers: its loops stay plain.
constexpr int kAhead = 8;

template <class V>
__device__ __forceinline__ void load_ahead(const V* row, int64_t b, int64_t n, V* to) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
        if (b + 32 * u < n) to[u] = row[b + 32 * u];
}

// Row i of r = B t, by a warp.
__device__ __forceinline__ void row_times(const float2* __restrict__ g, const float* __restrict__ amps,
                                          int64_t n, const float2* t, float2* r, int64_t i) {
    const int lane = threadIdx.x & 31;
    float2 acc = make_float2(0.f, 0.f);
    for (int64_t a = lane; a < n; a += 32 * kAhead) {
        float2 gi[kAhead], ta[kAhead];
        load_ahead(g + i * n, a, n, gi);
        load_ahead(t, a, n, ta);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (a + 32 * u >= n) break;
            const float2 v = cmul(gi[u], ta[u]);
            acc.x += v.x;
            acc.y += v.y;
        }
    }
    acc = warp_sum2(acc);
    if (lane == 0) {
        const float2 p = t[n + i];
        r[i] = make_float2(acc.x - amps[i] * p.x, acc.y - amps[i] * p.y);
    }
}

// Jtf_b = Im(t_b conj((B^H r)_b)).
__device__ __forceinline__ float gradient_at(const float2* g, const float* amps, int64_t n, int64_t m,
                                             const float2* t, const float2* r, int64_t b) {
    float2 w;
    if (b < n) {
        w = make_float2(0.f, 0.f);
        for (int64_t i0 = 0; i0 < m; i0 += kAhead) {
            float2 ga[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (i0 + u < m) ga[u] = g[(i0 + u) * n + b];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (i0 + u >= m) break;
                const float2 a = ga[u], q = r[i0 + u];
                // conj(a) q
                w.x += a.x * q.x + a.y * q.y;
                w.y += a.x * q.y - a.y * q.x;
            }
        }
    } else {
        const int64_t i = b - n;
        w = make_float2(-amps[i] * r[i].x, -amps[i] * r[i].y);
    }
    const float2 tb = t[b];
    return tb.y * w.x - tb.x * w.y;
}

// Solution of the host's 2m x 2m system, by value in the launch.
struct NlsY {
    float v[2 * kNlsMaxFoci];
};

// x_new = x + h with h = (coef_g Jtf - U^T y) * scale (LM: coef_g = 1, scale = -1/mu, i.e.
// h = -(Jtf - U^T y)/mu; GN: coef_g = 0, scale = -1), and t_new.  `first`: x_new = 0 instead.
__global__ void __launch_bounds__(128)
    nls_point_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n,
                     int64_t m, const float2* __restrict__ t, const float* __restrict__ jtf,
                     const __grid_constant__ NlsY y, float coef_g, float scale, int first,
                     const float* __restrict__ x, float* h, float* x_new, float2* t_new) {
    const int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    dev::pdl_wait();
    dev::pdl_release();
    if (b >= n + m) return;
    float xb = 0.f;
    if (!first) {
        float u = 0.f;  // (U^T y)_b = sum_i Re(C_ib) y_i + Im(C_ib) y_{m+i}
        const float2 tb = t[b];
        if (b < n) {
#pragma unroll 8
            for (int64_t i = 0; i < m; ++i) {
                const float2 c = cmul(g[i * n + b], tb);
                u += c.x * y.v[i] + c.y * y.v[m + i];
            }
        } else {
            const int64_t i = b - n;
            u = -amps[i] * (tb.x * y.v[i] + tb.y * y.v[m + i]);
        }
        const float hb = (coef_g * jtf[b] - u) * scale;
        h[b] = hb;
        xb = x[b] + hb;
    }
    x_new[b] = xb;
    float s, c;
    sincosf(xb, &s, &c);
    t_new[b] = make_float2(c, s);
}

// r = B t (task i < m: row i) and L (task m + p: entry p = i m + j); a warp a task.
constexpr int kRowsThreads = 64;

__global__ void __launch_bounds__(kRowsThreads)
    nls_rows_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n,
                    int64_t m, const float2* __restrict__ t, float2* r, float2* l) {
    dev::pdl_wait();
    dev::pdl_release();
    const int lane = threadIdx.x & 31;
    const int64_t task = static_cast<int64_t>(blockIdx.x) * (kRowsThreads / 32) + (threadIdx.x >> 5);
    if (task < m) {
        row_times(g, amps, n, t, r, task);
        return;
    }
    const int64_t p = task - m;
    if (p >= m * m) return;
    // L_ij = sum_{b<n} G_ib G_jb t_b^2 + delta_ij amps_i^2 t_{n+i}^2
    const int64_t i = p / m, j = p % m;
    float2 acc = make_float2(0.f, 0.f);
    for (int64_t b = lane; b < n; b += 32 * kAhead) {
        float2 gi[kAhead], gj[kAhead], tb[kAhead];
        load_ahead(g + i * n, b, n, gi);
        load_ahead(g + j * n, b, n, gj);
        load_ahead(t, b, n, tb);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (b + 32 * u >= n) break;
            const float2 t2 = make_float2(tb[u].x * tb[u].x - tb[u].y * tb[u].y, 2.f * tb[u].x * tb[u].y);
            const float2 v = cmul(cmul(gi[u], gj[u]), t2);
            acc.x += v.x;
            acc.y += v.y;
        }
    }
    acc = warp_sum2(acc);
    if (lane == 0) {
        if (i == j) {
            const float2 tp = t[n + i];
            const float a2 = amps[i] * amps[i];
            acc.x += a2 * (tp.x * tp.x - tp.y * tp.y);
            acc.y += a2 * (2.f * tp.x * tp.y);
        }
        l[p] = acc;
    }
}

// Jtf_b = Im(t_b conj((B^H r)_b)), a thread a column.
__global__ void __launch_bounds__(128)
    nls_gradient_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n,
                        int64_t m, const float2* __restrict__ t, const float2* __restrict__ r,
                        float* __restrict__ jtf) {
    dev::pdl_wait();
    dev::pdl_release();
    const int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (b < n + m) jtf[b] = gradient_at(g, amps, n, m, t, r, b);
}

// The scalars sc[0..4], one block each: F = |r|^2, max(Jtf), |x|^2, |h|^2, h.(mu h - Jtf at the point
// the step left); U Jtf: (Re C_i., Im C_i.) . Jtf, C_ib = B_ib t_b, 32 rows a block, a warp a row; and L
// to the host (stored there by nls_rows, its launch would end with a flush that the next one waits for).
constexpr int kScalars = 5;

__global__ void __launch_bounds__(kNlsThreads)
    nls_finish_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n,
                      int64_t m, const float* __restrict__ x, const float2* __restrict__ t,
                      const float2* __restrict__ r, const float* __restrict__ jtf,
                      const float* __restrict__ h, const float* __restrict__ jtf_old,
                      const float2* __restrict__ l, float mu, int first, float* __restrict__ sc,
                      float* __restrict__ ug, float2* __restrict__ l_out) {
    __shared__ float red[32];
    dev::pdl_wait();
    dev::pdl_release();
    const int64_t N = n + m;
    const int64_t l_block = static_cast<int64_t>(blockIdx.x) - kScalars - (m + 31) / 32;
    if (l_block >= 0) {
        const int64_t p = l_block * kNlsThreads + threadIdx.x;
        if (p < m * m) l_out[p] = l[p];
        return;
    }
    if (blockIdx.x >= kScalars) {
        const int lane = threadIdx.x & 31;
        const int64_t i = static_cast<int64_t>(blockIdx.x - kScalars) * 32 + (threadIdx.x >> 5);
        if (i >= m) return;
        float2 acc = make_float2(0.f, 0.f);
        for (int64_t b = lane; b < n; b += 32 * kAhead) {
            float2 gi[kAhead], tb[kAhead];
            float jb[kAhead];
            load_ahead(g + i * n, b, n, gi);
            load_ahead(t, b, n, tb);
            load_ahead(jtf, b, n, jb);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (b + 32 * u >= n) break;
                const float2 c = cmul(gi[u], tb[u]);
                acc.x += c.x * jb[u];
                acc.y += c.y * jb[u];
            }
        }
        acc = warp_sum2(acc);
        if (lane == 0) {
            const float2 p = t[n + i];
            const float gj = jtf[n + i];
            ug[i] = acc.x - amps[i] * p.x * gj;
            ug[m + i] = acc.y - amps[i] * p.y * gj;
        }
        return;
    }
    float v = 0.f;
    switch (blockIdx.x) {
        case 0:
            for (int64_t i = threadIdx.x; i < m; i += blockDim.x) v += r[i].x * r[i].x + r[i].y * r[i].y;
            break;
        case 1:
            v = -__int_as_float(0x7f800000);
            for (int64_t b = threadIdx.x; b < N; b += blockDim.x) v = fmaxf(v, jtf[b]);
            break;
        case 2:
            for (int64_t b = threadIdx.x; b < N; b += blockDim.x) v += x[b] * x[b];
            break;
        case 3:
            for (int64_t b = threadIdx.x; !first && b < N; b += blockDim.x) {
                const float hb = h[b];
                v += hb * hb;
            }
            break;
        default:
            for (int64_t b = threadIdx.x; !first && b < N; b += blockDim.x) {
                const float hb = h[b];
                v += hb * (mu * hb - jtf_old[b]);
            }
    }
    v = blockIdx.x == 1 ? block_max(v, red) : block_sum(v, red);
    if (threadIdx.x == 0) sc[blockIdx.x] = v;
}

// K = B B^H = G G^H + diag(amps^2) in double, entry (i, j) summed over the columns in order with
// every operation rounded, block (i, j) for j <= i and its conjugate.  The FP64 pipe takes a warp's
// instruction in some 60 cycles, so a block's threads convert and multiply for all columns of a chunk
// and two of them only add: 996 sources x 16 foci 430 -> 47 us against a thread an entry.  The products of
// two floats are exact, so a product summed with another by an FMA is the rounded sum of both.
// And the largest diagonal entry of JtJ, sum_i |B_ib|^2, in `a_max` (zero on entry; non-negative
// doubles order as their bits), in the blocks from row m on: a thread a column up to kKColumnBlocks
// blocks, then several columns a thread (a block each would pass the grid's 65,535 rows for one focus and
// 8.4 million sources).
constexpr int kKThreads = 128;
constexpr int kKChunk = 1024;
constexpr int64_t kKColumnBlocks = 4096;

__global__ void __launch_bounds__(kKThreads)
    nls_k_kernel(const float2* __restrict__ g, const float* __restrict__ amps, int64_t n, int m,
                 double2* __restrict__ k, unsigned long long* __restrict__ a_max) {
    __shared__ double2 s_p[kKChunk];
    const int i = blockIdx.y, j = blockIdx.x;
    if (i < m && j <= i) {
        const float2 *gi = g + i * n, *gj = g + j * n;
        double acc = 0;
        for (int64_t b0 = 0; b0 < n; b0 += kKChunk) {
            const int cnt = static_cast<int>(n - b0 < kKChunk ? n - b0 : kKChunk);
            for (int b = threadIdx.x; b < cnt; b += kKThreads) {
                const float2 u = gi[b0 + b], v = gj[b0 + b];
                const double ar = u.x, ai = u.y, br = v.x, bi = v.y;
                s_p[b] = make_double2(__fma_rn(ar, br, __dmul_rn(ai, bi)),  // a conj(b)
                                      __fma_rn(ai, br, -__dmul_rn(ar, bi)));
            }
            __syncthreads();
            if (threadIdx.x < 2) {
                const double* p = reinterpret_cast<const double*>(s_p) + threadIdx.x;
#pragma unroll 16
                for (int b = 0; b < cnt; ++b) acc = __dadd_rn(acc, p[2 * b]);
            }
            __syncthreads();
        }
        if (threadIdx.x < 2) {
            if (i == j && threadIdx.x == 0) acc = __dadd_rn(acc, __dmul_rn(amps[i], amps[i]));
            double* e = reinterpret_cast<double*>(k);
            e[2 * (i * m + j) + threadIdx.x] = acc;
            if (i != j) e[2 * (j * m + i) + threadIdx.x] = threadIdx.x ? -acc : acc;
        }
        return;
    }
    if (i < m) return;
    const int64_t stride = static_cast<int64_t>(gridDim.y - m) * gridDim.x * kKThreads;
    double top = 0;
    for (int64_t b = (static_cast<int64_t>(i - m) * gridDim.x + j) * kKThreads + threadIdx.x; b < n + m;
         b += stride) {
        double s2 = 0;
        if (b < n) {
            for (int q = 0; q < m; ++q) {
                const float2 u = g[q * n + b];
                const double ar = u.x, ai = u.y;
                s2 = __dadd_rn(s2, __fma_rn(ar, ar, __dmul_rn(ai, ai)));
            }
        } else {
            s2 = __dmul_rn(amps[b - n], amps[b - n]);
        }
        if (s2 > top) top = s2;
    }
    if (top > 0) atomicMax(a_max, static_cast<unsigned long long>(__double_as_longlong(top)));
}

// ------------------------------------------------------------------ host: small dense algebra

// Solve the SPD system a y = b (k x k, row-major, overwritten) by Cholesky; false if not SPD.  Column
// by column, each column's products taken off the rest of the lower triangle as soon as it is
// known: an entry loses them in the same order as in its own dot product, but its neighbours'
// chains run side by side.
bool cholesky_solve(std::vector<double>& a, std::vector<double>& b, int k) {
    std::vector<double> col(static_cast<size_t>(k));
    for (int p = 0; p < k; ++p) {
        double d = a[p * k + p];
        if (!(d > 0.0)) return false;
        d = std::sqrt(d);
        a[p * k + p] = d;
        for (int i = p + 1; i < k; ++i) col[i] = a[i * k + p] = a[i * k + p] / d;
        for (int i = p + 1; i < k; ++i) {
            double* row = &a[static_cast<size_t>(i) * k];
            const double l = col[i];
            for (int j = p + 1; j <= i; ++j) row[j] -= l * col[j];
        }
    }
    for (int i = 0; i < k; ++i) {  // L z = b
        double s = b[i];
        for (int p = 0; p < i; ++p) s -= a[i * k + p] * b[p];
        b[i] = s / a[i * k + i];
    }
    for (int i = k - 1; i >= 0; --i) {  // L^T y = z
        double s = b[i];
        for (int p = i + 1; p < k; ++p) s -= a[p * k + i] * b[p];
        b[i] = s / a[i * k + i];
    }
    return true;
}

// Cyclic Jacobi eigendecomposition of the symmetric k x k matrix a (row-major, destroyed):
// eigenvalues in lam, eigenvectors in the columns of v.
void jacobi_eigen(std::vector<double>& a, int k, std::vector<double>& lam, std::vector<double>& v) {
    v.assign(static_cast<size_t>(k) * k, 0.0);
    for (int i = 0; i < k; ++i) v[i * k + i] = 1.0;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j < k; ++j) {
                tot += a[i * k + j] * a[i * k + j];
                if (i != j) off += a[i * k + j] * a[i * k + j];
            }
        if (off <= 1e-30 * tot || off == 0.0) break;
        for (int p = 0; p < k; ++p)
            for (int q = p + 1; q < k; ++q) {
                const double apq = a[p * k + q];
                if (apq == 0.0) continue;
                const double theta = (a[q * k + q] - a[p * k + p]) / (2.0 * apq);
                const double tt = (theta >= 0 ? 1.0 : -1.0) /
                                  (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                const double c = 1.0 / std::sqrt(tt * tt + 1.0), s = tt * c;
                for (int r = 0; r < k; ++r) {  // columns p, q
                    const double arp = a[r * k + p], arq = a[r * k + q];
                    a[r * k + p] = c * arp - s * arq;
                    a[r * k + q] = s * arp + c * arq;
                }
                for (int r = 0; r < k; ++r) {  // rows p, q
                    const double apr = a[p * k + r], aqr = a[q * k + r];
                    a[p * k + r] = c * apr - s * aqr;
                    a[q * k + r] = s * apr + c * aqr;
                }
                for (int r = 0; r < k; ++r) {
                    const double vrp = v[r * k + p], vrq = v[r * k + q];
                    v[r * k + p] = c * vrp - s * vrq;
                    v[r * k + q] = s * vrp + c * vrq;
                }
            }
    }
    lam.resize(k);
    for (int i = 0; i < k; ++i) lam[i] = a[i * k + i];
}

// Host-level state: one stream and blocks shared by all systems.  Blocks of up to kKeepBytes stay for
// the next call (allocating and freeing them cost about as much as a call's launches) and are given back
// with the last system (release_nls_blocks); larger ones at the end of the call that needed them.
constexpr size_t kKeepBytes = 64u << 20;

struct NlsCtx {
    std::mutex mu;
    cudaStream_t stream = nullptr;
    int device = -1;
    char* d = nullptr;  // device block
    size_t d_cap = 0;
    char* h = nullptr;  // pinned block, and its address for kernels
    char* h_dev = nullptr;
    size_t h_cap = 0;
};
NlsCtx g_nls;

// under the lock, the stream idle
void give_back(NlsCtx& c) {
    if (c.d) cudaFree(c.d);
    if (c.h) cudaFreeHost(c.h);
    c.d = c.h = c.h_dev = nullptr;
    c.d_cap = c.h_cap = 0;
}

cudaError_t grow(NlsCtx& c, size_t d_bytes, size_t h_bytes) {
    cudaError_t e = cudaSuccess;
    if (d_bytes > c.d_cap) {
        if (c.d) cudaFree(c.d);
        c.d = nullptr;
        c.d_cap = 0;
        if ((e = cudaMalloc(&c.d, d_bytes)) != cudaSuccess) return e;
        c.d_cap = d_bytes;
    }
    if (h_bytes > c.h_cap) {
        if (c.h) cudaFreeHost(c.h);
        c.h = c.h_dev = nullptr;
        c.h_cap = 0;
        void* dev = nullptr;
        if ((e = cudaHostAlloc(&c.h, h_bytes, cudaHostAllocMapped)) != cudaSuccess) return e;
        c.h_cap = h_bytes;
        if ((e = cudaHostGetDevicePointer(&dev, c.h, 0)) != cudaSuccess) return e;
        c.h_dev = static_cast<char*>(dev);
    }
    return e;
}

}  // namespace

void release_nls_blocks() {
    std::lock_guard<std::mutex> lock(g_nls.mu);
    if (!g_nls.d && !g_nls.h) return;
    DeviceGuard dg;
    RelaxedCapture relaxed;
    if (dg.set(g_nls.device) == cudaSuccess) {
        cudaStreamSynchronize(g_nls.stream);
        give_back(g_nls);
    }
    (void)cudaGetLastError();  // a failure here must not surface as the next launch's
}

int solve_nls(int kind, int st, float* src, const float* k, const float* atten, int64_t n,
              const float* foci, const float* amps, int64_t m, std::string* err,
              const AfcNlsStep* first_step) {
    if (m > kNlsMaxFoci) {
        *err = "too many foci for the NLS solvers (" + std::to_string(m) + " > " +
               std::to_string(kNlsMaxFoci) + ")";
        return -1;
    }
    if (n == 0) return 0;
    const int stride = source_stride(st);
    const int iphase = st == SRC_T4010A1 ? 7 : 4;
    std::lock_guard<std::mutex> lock(g_nls.mu);
    cudaError_t e;
    auto fail = [&](const char* what) {
        *err = std::string(what) + ": " + cudaGetErrorString(e);
        return -1;
    };
    if (!g_nls.stream) {
        int count = 0;
        e = cudaGetDeviceCount(&count);
        if (e != cudaSuccess || count == 0) {
            *err = "no CUDA device available; this library has no CPU path";
            return -1;
        }
        if ((e = cudaGetDevice(&g_nls.device)) != cudaSuccess) return fail("cudaGetDevice");
        if ((e = cudaStreamCreateWithFlags(&g_nls.stream, cudaStreamNonBlocking)) != cudaSuccess) {
            g_nls.stream = nullptr;
            return fail("cudaStreamCreate");
        }
    }
    DeviceGuard dg;  // the solver's device while it runs; the caller's again on return
    if ((e = dg.set(g_nls.device)) != cudaSuccess) return fail("cudaSetDevice");
    cudaStream_t s = g_nls.stream;
    const int64_t N = n + m;
    const int mm = static_cast<int>(m), k2 = 2 * mm;

    // device block: inputs (raw | k | atten | foci | amps) | G | packed | h | r | L and, for each of two
    // points, x | t | Jtf; pinned block: inputs | x | K | a_max and, for each point, scalars | U Jtf | L
    auto a256 = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += a256(bytes ? bytes : 1);
        return o;
    };
    const size_t raw_f = static_cast<size_t>(n) * stride, in_f = raw_f + 2 * n + 4 * m;
    const size_t o_in = take(4 * in_f), o_g = take(8 * m * n), o_pk = take(48 * n), o_h = take(4 * N),
                 o_r = take(8 * m), o_l = take(8 * m * m), o_it = take(4),
                 o_amax = take(8);
    size_t o_x[2], o_t[2], o_j[2];
    for (int q = 0; q < 2; ++q) {
        o_x[q] = take(4 * N);
        o_t[q] = take(8 * N);
        o_j[q] = take(4 * N);
    }
    const size_t d_bytes = off;
    off = 0;
    const size_t p_in = take(4 * in_f), p_x = take(4 * N), p_k = take(16 * m * m), p_amax = take(8);
    size_t p_sc[2], p_ug[2], p_l[2];
    for (int q = 0; q < 2; ++q) {
        p_sc[q] = take(32);
        p_ug[q] = take(8 * m);
        p_l[q] = take(8 * m * m);
    }
    struct Trim {  // gives large blocks back when the call ends
        ~Trim() {
            if (g_nls.d_cap > kKeepBytes || g_nls.h_cap > kKeepBytes) {
                cudaStreamSynchronize(g_nls.stream);
                give_back(g_nls);
            }
        }
    } trim;
    if ((e = grow(g_nls, d_bytes, off)) != cudaSuccess) return fail("allocation");
    char *d = g_nls.d, *h = g_nls.h, *hd = g_nls.h_dev;
    auto F = [&](size_t o) { return reinterpret_cast<float*>(d + o); };
    auto F2 = [&](size_t o) { return reinterpret_cast<float2*>(d + o); };
    float* in = reinterpret_cast<float*>(h + p_in);
    memcpy(in, src, 4 * raw_f);
    // phases are zeroed first (nls/*.rs: set_phase(0.)); G is built from the zero-phase sources
    for (int64_t j = 0; j < n; ++j) in[j * stride + iphase] = 0.f;
    memcpy(in + raw_f, k, 4 * n);
    memcpy(in + raw_f + n, atten, 4 * n);
    if (m) {
        memcpy(in + raw_f + 2 * n, foci, 12 * m);
        memcpy(in + raw_f + 2 * n + 3 * m, amps, 4 * m);
    }
    const float* d_in = F(o_in);
    const float* d_amps = d_in + raw_f + 2 * n + 3 * m;
    if ((e = cudaMemcpyAsync(d + o_in, in, 4 * in_f, cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return fail("upload");
    if ((e = launch_build_g(st, d_in, d_in + raw_f, d_in + raw_f + n, n, d_in + raw_f + 2 * n, m, F2(o_g),
                            d + o_pk, s)) != cudaSuccess)
        return fail("G");
    int cur = 0;  // the current point; 1 - cur is the trial point

    if (kind == NLS_GRADIENT_DESCENT) {
        if ((e = cudaMemsetAsync(d + o_x[0], 0, 4 * N, s)) != cudaSuccess) return fail("upload");
        nls_gd_kernel<<<1, kNlsThreads, 0, s>>>(F2(o_g), d_amps, n, m, F(o_x[0]), F2(o_t[0]), F2(o_r),
                                               F(o_j[0]), kGdIterations, kGdEps,
                                               reinterpret_cast<int*>(d + o_it));
        count_launch();
        if ((e = cudaGetLastError()) != cudaSuccess) return fail("gradient descent");
    } else {
        if ((e = cudaMemsetAsync(d + o_amax, 0, 8, s)) != cudaSuccess) return fail("K");
        const unsigned kx = static_cast<unsigned>(std::max<int64_t>(m, 1));
        const int64_t col_blocks = std::min((N + kKThreads - 1) / kKThreads, kKColumnBlocks);
        nls_k_kernel<<<dim3(kx, static_cast<unsigned>(m + (col_blocks + kx - 1) / kx)), kKThreads, 0, s>>>(
            F2(o_g), d_amps, n, mm, reinterpret_cast<double2*>(hd + p_k),
            reinterpret_cast<unsigned long long*>(d + o_amax));
        count_launch();
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = cudaMemcpyAsync(h + p_amax, d + o_amax, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            return fail("K");

        // a step from point `cur` to the trial point (first: the trial point is 0) and everything at
        // the trial point; waits for it
        NlsY y{};
        auto step_launch = [&](bool first, float coef_g, float scale, float mu) -> bool {
            const int q = 1 - cur;
            const dim3 cols(static_cast<unsigned>((N + 127) / 128)), block(128);
            const unsigned tasks = static_cast<unsigned>((m + m * m + kRowsThreads / 32 - 1) / (kRowsThreads / 32));
            const dim3 finish(static_cast<unsigned>(kScalars + (m + 31) / 32 + (m * m + kNlsThreads - 1) / kNlsThreads));
            const float2* g = F2(o_g);
            if ((e = launch_after(nls_point_kernel, cols, block, 0, s, true, g, d_amps, n, m,
                                  static_cast<const float2*>(F2(o_t[cur])),
                                  static_cast<const float*>(F(o_j[cur])), y, coef_g, scale, first ? 1 : 0,
                                  static_cast<const float*>(F(o_x[cur])), F(o_h), F(o_x[q]),
                                  F2(o_t[q]))) != cudaSuccess ||
                (tasks && (e = launch_after(nls_rows_kernel, dim3(tasks), dim3(kRowsThreads), 0, s, true, g,
                                            d_amps, n, m, static_cast<const float2*>(F2(o_t[q])), F2(o_r),
                                            F2(o_l))) != cudaSuccess) ||
                (e = launch_after(nls_gradient_kernel, cols, block, 0, s, true, g, d_amps, n, m,
                                  static_cast<const float2*>(F2(o_t[q])),
                                  static_cast<const float2*>(F2(o_r)), F(o_j[q]))) != cudaSuccess ||
                (e = launch_after(nls_finish_kernel, finish, dim3(kNlsThreads), 0, s, true, g, d_amps, n, m, static_cast<const float*>(F(o_x[q])),
                                  static_cast<const float2*>(F2(o_t[q])),
                                  static_cast<const float2*>(F2(o_r)),
                                  static_cast<const float*>(F(o_j[q])), static_cast<const float*>(F(o_h)),
                                  static_cast<const float*>(F(o_j[cur])),
                                  static_cast<const float2*>(F2(o_l)), mu, first ? 1 : 0,
                                  reinterpret_cast<float*>(hd + p_sc[q]),
                                  reinterpret_cast<float*>(hd + p_ug[q]),
                                  reinterpret_cast<float2*>(hd + p_l[q]))) != cudaSuccess)
                return false;
            count_launch(tasks ? 4 : 3);
            return (e = cudaStreamSynchronize(s)) == cudaSuccess;
        };
        auto scalars = [&](int q) { return reinterpret_cast<const float*>(h + p_sc[q]); };
        const double* kk = reinterpret_cast<const double*>(h + p_k);  // K, re and im interleaved
        std::vector<double> mat(static_cast<size_t>(k2 * k2));
        // one step from the current point: M = U U^T from K and L (2m x 2m), y on the host, then the
        // device; false with *bad set when the small system cannot be solved
        auto step = [&](double mu, bool lm, bool* bad) -> bool {
            const float* lh = reinterpret_cast<const float*>(h + p_l[cur]);
            const float* ug = reinterpret_cast<const float*>(h + p_ug[cur]);
            for (int i = 0; i < mm; ++i)
                for (int j = 0; j < mm; ++j) {
                    const double lr = lh[2 * (i * mm + j)], li = lh[2 * (i * mm + j) + 1];
                    const double kr = kk[2 * (i * mm + j)], ki = kk[2 * (i * mm + j) + 1];
                    mat[i * k2 + j] = 0.5 * (kr + lr);
                    mat[i * k2 + mm + j] = 0.5 * (li - ki);
                    mat[(mm + i) * k2 + j] = 0.5 * (li + ki);
                    mat[(mm + i) * k2 + mm + j] = 0.5 * (kr - lr);
                }
            std::vector<double> rhs(ug, ug + k2);
            if (lm) {
                for (int i = 0; i < k2; ++i) mat[i * k2 + i] += mu;
                if (!cholesky_solve(mat, rhs, k2)) {
                    *bad = true;
                    return true;
                }
                for (int i = 0; i < k2; ++i) y.v[i] = static_cast<float>(rhs[i]);
            } else {
                std::vector<double> lam, v;
                jacobi_eigen(mat, k2, lam, v);
                std::vector<double> yy(static_cast<size_t>(k2), 0.0);
                for (int q = 0; q < k2; ++q) {
                    if (!(lam[q] > kPinvEps)) continue;
                    double proj = 0;
                    for (int i = 0; i < k2; ++i) proj += v[i * k2 + q] * rhs[i];
                    for (int i = 0; i < k2; ++i) yy[i] += v[i * k2 + q] * proj / (lam[q] * lam[q]);
                }
                for (int i = 0; i < k2; ++i) y.v[i] = static_cast<float>(yy[i]);
            }
            return step_launch(false, lm ? 1.f : 0.f, lm ? static_cast<float>(-1.0 / mu) : -1.f,
                               static_cast<float>(mu));
        };

        const bool lm = kind == NLS_LM;
        if (!step_launch(true, 0.f, 0.f, 0.f)) return fail("NLS evaluation");
        cur = 1 - cur;
        // diag(JtJ)_b = sum_i |B_ib|^2 (independent of x), for LM's initial mu
        double a_max;
        memcpy(&a_max, h + p_amax, 8);
        double fx = scalars(cur)[0];
        bool found = scalars(cur)[1] <= kNlsEps1;
        double mu = kLmTau * a_max, nu = 2.0;
        if (first_step) {
            const AfcNlsStep& o = *first_step;
            bool bad = false;
            if (!step(mu, lm, &bad)) return fail("NLS step");
            if (bad) {
                *err = "NLS: the first step's small system cannot be solved";
                return -1;
            }
            const int q = 1 - cur;
            auto get = [&](void* to, const void* from, size_t bytes) {
                return (e = cudaMemcpyAsync(to, from, bytes, cudaMemcpyDefault, s)) == cudaSuccess;
            };
            if (!get(o.g, d + o_g, 8 * m * n) || !get(o.k, h + p_k, 16 * m * m) ||
                !get(o.x, d + o_x[q], 4 * N) || !get(o.h, d + o_h, 4 * N) ||
                !get(o.jtf0, d + o_j[cur], 4 * N) || !get(o.jtf, d + o_j[q], 4 * N) ||
                !get(o.scalars, h + p_sc[q], 4 * kScalars) || !get(o.u_jtf, h + p_ug[q], 8 * m) ||
                !get(o.l, h + p_l[q], 8 * m * m) || (e = cudaStreamSynchronize(s)) != cudaSuccess)
                return fail("NLS step download");
            *o.a_max = a_max;
            return 0;
        }
        for (int it = 0; it < kNlsIterations && !found; ++it) {
            bool bad = false;
            const float xx = scalars(cur)[2];  // |x|^2 at the current x
            if (!step(mu, lm, &bad)) return fail("NLS step");
            if (bad) break;
            const float* sc = scalars(1 - cur);
            const float hh = sc[3], hd2 = sc[4];
            if (std::sqrt(static_cast<double>(hh)) <=
                kNlsEps2 * (std::sqrt(static_cast<double>(xx)) + kNlsEps2))
                break;  // the step found nothing further
            if (!lm) {  // Gauss-Newton: accept x + h (gauss_newton.rs:72-79)
                cur = 1 - cur;
                found = sc[1] <= kNlsEps1;
                continue;
            }
            // LM (lm.rs:75-96): gain ratio from F at x_new
            const double fx_new = sc[0];
            const double l0 = 0.5 * hd2;
            const double rho = (fx - fx_new) / l0;
            fx = fx_new;
            if (rho > 0.0) {
                cur = 1 - cur;
                found = sc[1] <= kNlsEps1;
                const double c = 2.0 * rho - 1.0;
                mu *= std::max(1.0 / 3.0, 1.0 - c * c * c);
                nu = 2.0;
            } else {
                // x, A and g stay (F takes F(x_new), as in the reference)
                mu *= nu;
                nu *= 2.0;
            }
        }
    }
    const float* x = reinterpret_cast<const float*>(h + p_x);
    if ((e = cudaMemcpyAsync(h + p_x, d + o_x[cur], 4 * N, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return fail("NLS result");
    for (int64_t j = 0; j < n; ++j) src[j * stride + iphase] = x[j];
    return 0;
}

}  // namespace afc

// Transfer matrix and multi-focus solvers on sm_103a.
//
//   build_g        G[i, j] = propagate(source j, focus i) with the sources' current amplitude
//                  and phase 0 (acoustic-field-optimizer/src/multiple_foci/macros.rs:32-53,
//                  called after the phases are zeroed, gs_pat.rs:38-45).  Row-major m x n.
//   GS-PAT         gs_pat.rs:47-80: den_j = sum_i |G_ij| (nalgebra row_sum = column sums),
//                  B = [conj(G_ij) / den_j^2]^T, R = G B (m x m), gamma = R p0, 100 times
//                  {p = gamma / |gamma| * p0; gamma = R p}, p = gamma / |gamma|^2 * p0^2,
//                  q = B p; amp_j = |q_j|, phase_j = arg q_j.  B is never materialised:
//                  R_ik = sum_j G_ij conj(G_kj) / den_j^2 and q_j = sum_i conj(G_ij) p_i / den_j^2.
//   GS             gs.rs:42-77: q = q0; 100 times {gamma = G q; p = gamma/|gamma| p0;
//                  xi = G^H p; q = xi/|xi| q0}.
//   Naive          naive.rs:37-49: q = G^H p0.
//
// Sizes are small (m <= 64 foci, n ~ 1e3 sources in the serving mix), so GS-PAT is bound by the
// latency of its chain of launches and of its 100 dependent products, not by bytes or flops.  Its
// four launches: G with its column sums (packing included), R in 4 x 4 tiles, the iterations with
// R in registers (one block up to 64 foci, a cluster of 8 above, so that a dependent step costs a
// barrier and not a launch), the back-propagation.  Every sum is added in one fixed order (stated
// at each kernel): GS-PAT amplifies rounding when the foci make R ill-conditioned, so a split of
// the work must not change the order of a sum.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "afc_internal.h"
#include "afc_solvers.h"
#include "field_body.cuh"
#include "gspat_share.h"
#include "propagate.cuh"

namespace afc {

namespace {

__constant__ float4 c_dir_table_s[dev::kDirTableSize] = AFC_DIR_TABLE_INIT;

constexpr int kIterThreads = 1024;
constexpr float kPiF = 3.14159265358979323846f;  // f32 PI of the reference (core/mod.rs)

size_t align256(size_t b) { return (b + 255) & ~static_cast<size_t>(255); }

struct SolverWs {
    PackedSource* packed;
    float2* g;
    float* inv_den2;
    float2* r;
    float2* p;
    float2* q;
};

SolverWs carve(void* ws, int64_t n, int64_t m) {
    char* b = static_cast<char*>(ws);
    SolverWs w;
    w.packed = reinterpret_cast<PackedSource*>(b);
    b += align256(sizeof(PackedSource) * n);
    w.g = reinterpret_cast<float2*>(b);
    b += align256(sizeof(float2) * n * m);
    w.inv_den2 = reinterpret_cast<float*>(b);
    b += align256(sizeof(float) * n);
    w.r = reinterpret_cast<float2*>(b);
    b += align256(sizeof(float2) * m * m);
    w.p = reinterpret_cast<float2*>(b);
    b += align256(sizeof(float2) * m);
    w.q = reinterpret_cast<float2*>(b);
    return w;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// conj(a) * b
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.x, b.y, -a.y * b.x));
}

__device__ __forceinline__ float2 warp_sum(float2 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

template <int ST>
__global__ void build_g_kernel(const PackedSource* __restrict__ src, int64_t n,
                               const float* __restrict__ foci, int64_t m, float2* __restrict__ g) {
    __shared__ float4 s_dir[dev::kDirTableSize];
    if (threadIdx.x < dev::kDirTableSize) s_dir[threadIdx.x] = c_dir_table_s[threadIdx.x];
    dev::pdl_wait();  // the packed sources
    dev::pdl_release();
    __syncthreads();
    const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t i = blockIdx.y;
    if (j >= n) return;
    const PackedSource s = src[j];
    float w, red;
    // the phases are zeroed before G is built (gs_pat.rs:39-41): phase' is pi for A < 0
    dev::pair_terms<ST>(s.a, s.b, s.c.x, s.c.z < 0.f ? 3.14159265358979323846f : 0.0f, s_dir,
                        foci[3 * i], foci[3 * i + 1], foci[3 * i + 2], w, red);
    g[i * n + j] = make_float2(w * dev::mufu_cos(red), w * dev::mufu_sin(red));
}

// The kernels over the columns of G (sources) below take 32 sources by 8 groups of foci a block: the
// groups evaluate their foci's terms side by side into shared memory, kColChunk foci at a time,
// and one warp then adds them per source in focus order.  As one thread per source the terms'
// latencies (hypotf, the loads) lay end to end: 64 us of column sums and 29 us of back-propagation
// at 996 sources x 128 foci; see the launch code for the whole chain's times.
constexpr int kColThreads = 256;
constexpr int kColSources = 32;
constexpr int kColGroups = kColThreads / kColSources;
constexpr int kColChunk = 64;

// G from the ABI records (packed as pack_source packs them, phases zeroed) and inv_den2[j] =
// 1 / (sum_i |G_ij|)^2, the sum in focus order.
template <int ST>
__global__ void __launch_bounds__(kColThreads)
    gspat_g_kernel(const float* __restrict__ raw, const float* __restrict__ k,
                   const float* __restrict__ atten, int64_t n, const float* __restrict__ foci,
                   int64_t m, float2* __restrict__ g, float* __restrict__ inv_den2) {
    __shared__ float4 s_dir[dev::kDirTableSize];
    __shared__ float s_abs[kColChunk][kColSources];
    dev::pdl_release();
    if (threadIdx.x < dev::kDirTableSize) s_dir[threadIdx.x] = c_dir_table_s[threadIdx.x];
    const int lane = threadIdx.x % kColSources, group = threadIdx.x / kColSources;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * kColSources + lane;
    const bool live = j < n;
    PackedSource s{};
    if (live) s = fb::pack_source(ST, raw, k, atten, j);
    // the phases are zeroed before G is built (gs_pat.rs:39-41): phase' is pi for A < 0
    const float phase = s.c.z < 0.f ? 3.14159265358979323846f : 0.0f;
    __syncthreads();
    float sum = 0.f;
    for (int64_t i0 = 0; i0 < m; i0 += kColChunk) {
        const int cnt = static_cast<int>(m - i0 < kColChunk ? m - i0 : kColChunk);
        if (live) {
            for (int i = group; i < cnt; i += kColGroups) {
                const float* f = foci + 3 * (i0 + i);
                float w, red;
                dev::pair_terms<ST>(s.a, s.b, s.c.x, phase, s_dir, f[0], f[1], f[2], w, red);
                const float2 v = make_float2(w * dev::mufu_cos(red), w * dev::mufu_sin(red));
                g[(i0 + i) * n + j] = v;
                s_abs[i][lane] = hypotf(v.x, v.y);
            }
        }
        __syncthreads();
        if (group == 0 && live) {
#pragma unroll 8
            for (int i = 0; i < cnt; ++i) sum += s_abs[i][lane];
        }
        __syncthreads();
    }
    if (group == 0 && live) inv_den2[j] = 1.0f / (sum * sum);
}

// R[i, k] = sum_j G_ij conj(G_kj) inv_den2_j, one block per 4 x 4 entries, so that a row of G is
// read m / 4 times instead of m (996 sources x 128 foci: 24.7 us as one block per entry).  Thread t
// sums j = t, t + 128, ... in order; a butterfly over 16, 8, 4, 2, 1 lanes adds a warp's partial
// sums, (p0 + p2) + (p1 + p3) the four warps'.  The butterfly halves the entries it carries at
// every level (lane l ends with entry l of the 32 floats), which leaves each entry's tree as it is.
constexpr int kRThreads = 128;
constexpr int kRTile = 4;

__global__ void __launch_bounds__(kRThreads)
    gspat_r_kernel(const float2* __restrict__ g, const float* __restrict__ inv_den2, int64_t n,
                   int64_t m, float2* __restrict__ r) {
    __shared__ float part[kRThreads / 32][32];
    dev::pdl_wait();
    dev::pdl_release();
    const int64_t i0 = static_cast<int64_t>(blockIdx.y) * kRTile;
    const int64_t k0 = static_cast<int64_t>(blockIdx.x) * kRTile;
    const float2 *gi[kRTile], *gk[kRTile];
#pragma unroll
    for (int a = 0; a < kRTile; ++a) {
        gi[a] = g + (i0 + a < m ? i0 + a : m - 1) * n;  // past the edge: computed, never stored
        gk[a] = g + (k0 + a < m ? k0 + a : m - 1) * n;
    }
    float v[2 * kRTile * kRTile];
#pragma unroll
    for (int q = 0; q < 2 * kRTile * kRTile; ++q) v[q] = 0.f;
    for (int64_t j = threadIdx.x; j < n; j += kRThreads) {
        const float s = inv_den2[j];
        float2 vi[kRTile], vk[kRTile];
#pragma unroll
        for (int a = 0; a < kRTile; ++a) {
            vi[a] = gi[a][j];
            vk[a] = gk[a][j];
        }
#pragma unroll
        for (int a = 0; a < kRTile; ++a) {
#pragma unroll
            for (int b = 0; b < kRTile; ++b) {
                const float2 t = cmulc(vk[b], vi[a]);  // G_ij conj(G_kj)
                float* acc = v + 2 * (a * kRTile + b);
                acc[0] = fmaf(t.x, s, acc[0]);
                acc[1] = fmaf(t.y, s, acc[1]);
            }
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;  // keeps the upper half of the entries still carried
#pragma unroll
        for (int q = 0; q < o; ++q) {
            const float mine = up ? v[q + o] : v[q], other = up ? v[q] : v[q + o];
            v[q] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
    }
    part[wid][lane] = v[0];
    __syncthreads();
    if (wid == 0) {
        const float sum = (part[0][lane] + part[2][lane]) + (part[1][lane] + part[3][lane]);
        const int64_t i = i0 + (lane >> 3), c = k0 + ((lane >> 1) & 3);
        if (i < m && c < m) reinterpret_cast<float*>(r)[2 * (i * m + c) + (lane & 1)] = sum;
    }
}

// The GS-PAT iteration (gs_pat.rs:54-71) for up to kGspatSmallFoci foci: one block, kSmallLanes
// threads a row, R in registers.  A row's sum is that of 16 lanes, lane l over columns l, l + 16, ...
// in order, added by a butterfly over 8, 4, 2, 1; thread `sub` carries lanes sub, sub + 4, sub + 8 and
// sub + 12, adds the first two levels by itself and the others by shuffles.  p is double-buffered in
// shared memory (zeros past m), so one barrier separates an iteration's reads of p from the next
// one's writes; up to 8 foci are one warp.  Bound by the chain load, products, two shuffles,
// hypotf, division, store, barrier: 0.2 us an iteration at 8 foci, 0.35 at 64.  With 16 threads a
// row and R in shared memory (four shuffles and twice the shared loads) 8 foci took 38 us and 64 foci
// 92; with two threads a row in packed operations 64 foci took 5 us more.
constexpr int64_t kGspatSmallFoci = 64;
constexpr int kSmallLanes = 4;

__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 shfl_xor2(float2 v, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

template <int NC, bool ONE_WARP>
__global__ void __launch_bounds__(kGspatSmallFoci * kSmallLanes, 1)
    gspat_iterate_small_kernel(const float2* __restrict__ r, const float* __restrict__ amps, int m,
                               int repeat, float2* __restrict__ p_out) {
    __shared__ float2 s_p[2][16 * NC];
    dev::pdl_wait();
    dev::pdl_release();
    const int row = threadIdx.x / kSmallLanes, sub = threadIdx.x % kSmallLanes;
    const bool live = row < m;
    float2 rr[4][NC];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int t = 0; t < NC; ++t) {
            const int c = sub + 4 * u + 16 * t;
            rr[u][t] = live && c < m ? r[row * m + c] : make_float2(0.f, 0.f);
        }
    }
    // threads without a row divide 1 by 1: a zero would take the division's slow path and hold up
    // the warp (7 foci took 13 us more than 8)
    const float amp = live ? amps[row] : 1.f;
    for (int i = threadIdx.x; i < 16 * NC; i += blockDim.x) {
        s_p[0][i] = make_float2(i < m ? amps[i] : 0.f, 0.f);
        s_p[1][i] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    int cur = 0;
    for (int it = 0;; ++it) {
        float2 acc[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            acc[u] = make_float2(0.f, 0.f);
#pragma unroll
            for (int t = 0; t < NC; ++t)
                acc[u] = add(acc[u], cmul(rr[u][t], s_p[cur][sub + 4 * u + 16 * t]));
        }
        float2 gv = add(add(acc[0], acc[2]), add(acc[1], acc[3]));
        gv = add(gv, shfl_xor2(gv, 2));
        gv = add(gv, shfl_xor2(gv, 1));
        if (!live) gv.x = 1.f;
        const float a = hypotf(gv.x, gv.y);
        if (it == repeat) {
            if (live && sub == 0) {
                const float s = amp * amp / (a * a);
                p_out[row] = make_float2(gv.x * s, gv.y * s);
            }
            break;
        }
        cur ^= 1;
        const float s = amp / a;
        if (live && sub == 0) s_p[cur][row] = make_float2(gv.x * s, gv.y * s);
        if constexpr (ONE_WARP) __syncwarp();
        else __syncthreads();
    }
}

// mbarrier and cluster primitives of the iteration below.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Expect `bytes` more of remote stores on the barrier's current phase, and arrive once.
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait for the phase of the given parity; false once limit_ns of the global timer has passed or,
// should the timer stand still, after 2^26 polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try(bar, parity)) return true;
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t i = 0; i < (1u << 26); ++i) {
        if (mbar_try(bar, parity)) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > limit_ns) return false;
    }
    return false;
}
// Let `ns` of the global timer pass (or 2^16 polls).
__device__ __forceinline__ void let_pass(uint64_t ns) {
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t i = 0; i < (1u << 16); ++i) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > ns) return;
    }
}
// Store a, b at a 16-byte aligned shared::cluster address; the 16 bytes complete on the mbarrier
// `bar` beside it.
__device__ __forceinline__ void store_remote(uint32_t addr, float2 a, float2 b, uint32_t bar) {
    asm volatile(
        "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
        "r"(__float_as_uint(a.x)), "r"(__float_as_uint(a.y)), "r"(__float_as_uint(b.x)),
        "r"(__float_as_uint(b.y)), "r"(bar)
        : "memory");
}

// The same iteration above kGspatSmallFoci foci: a cluster of kIterCluster blocks, each with a
// contiguous share of the rows, kWideLanes threads a row.  A row's sum is that of 32 lanes, lane l
// over columns l, l + 32, ... in order, added by a butterfly over 16, 8, 4, 2, 1; thread `sub` carries
// lanes sub, sub + 8, sub + 16 and sub + 24 and adds the first two levels by itself.  NC > 0: up to
// 32 NC foci with R in registers (4 NC entries a thread); NC == 0: any number, R read from L2.
//
// Every block holds the whole of p twice.  A row's thread u stores the row's new entry into block
// u's other copy (st.async), whose mbarrier completes once all m entries have arrived: no block
// waits for more than the entries it reads, and no cluster barrier stands in the loop.  Two copies
// suffice: a block that has all entries of step k + 1 knows that every block has finished reading
// step k's, since it sent its entries after that.  The waits are bounded: a warp whose wait runs out
// leaves NaN in its rows of p_out, sets *wait.status, meets all blocks at the last cluster barrier and
// then lets the stores still on their way into its block land (a block whose waits all ended has
// received everything that was sent to it).
//
// One block can do no better than its flops: 0.4 us an iteration at 128 foci, and took 1.03 with R
// in registers, 2.9 with R in L2.  With a cluster barrier a step instead of the mbarriers the
// iteration took 1.1 us.
constexpr int kWideLanes = 8;
static_assert(kWideLanes == kIterCluster, "a row's thread u writes block u's copy of p");
static_assert(kGspatSmallFoci >= 2 * kIterCluster, "every block of the cluster has rows");

// The bounded waits: their limit (a working step takes under a microsecond), where a wait that ran
// out is reported, and, for the test of that, whether block 0 withholds its entries.
struct IterWait {
    unsigned* status;
    uint64_t limit_ns;
    int withhold;
};
constexpr uint64_t kIterWaitNs = 1000000000;    // a second
constexpr uint64_t kIterWaitTestNs = 10000000;  // where no wait can end
constexpr uint64_t kDrainNs = 20000;            // a store into another block takes about one microsecond

template <int NC>
__global__ void __launch_bounds__(NC > 0 ? 32 * NC : 1024)
    gspat_iterate_cluster_kernel(const float2* __restrict__ r, const float* __restrict__ amps,
                                 int64_t m, int repeat, float2* __restrict__ p_out, IterWait wait) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char gspat_dyn_smem[];
    __shared__ __align__(8) uint64_t s_bar[2];  // one per copy of p
    const int cols = static_cast<int>((m + 31) / 32 * 32);
    float2* s_p = reinterpret_cast<float2*>(gspat_dyn_smem);  // [2][cols], zeros past m
    const uint32_t bytes = static_cast<uint32_t>((m + 1) / 2 * sizeof(float4));  // rows go in pairs
    cg::cluster_group cluster = cg::this_cluster();
    dev::pdl_wait();
    dev::pdl_release();
    const int64_t rank = cluster.block_rank(), lo = iter_first(m, rank);
    const int64_t hi = iter_first(m, rank + 1) < m ? iter_first(m, rank + 1) : m;
    const int sub = threadIdx.x % kWideLanes;
    const int64_t first = lo + threadIdx.x / kWideLanes, step = blockDim.x / kWideLanes;
    constexpr int kRegs = NC > 0 ? NC : 1;
    float2 rr[4][kRegs];
    if constexpr (NC > 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int t = 0; t < NC; ++t) {
                const int64_t c = sub + 8 * u + 32 * t;
                rr[u][t] = first < hi && c < m ? r[first * m + c] : make_float2(0.f, 0.f);
            }
        }
    }
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
        s_p[i] = make_float2(i < m ? amps[i] : 0.f, 0.f);
        s_p[cols + i] = make_float2(0.f, 0.f);
    }
    const uint32_t bar0 = smem_addr(&s_bar[0]), p0 = smem_addr(s_p);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect(bar0, bytes);
        mbar_expect(bar0 + 8, bytes);
    }
    cluster.sync();  // every block's copies and barriers are set up before any remote store
    // block `sub`'s copies of p and their barriers
    const uint32_t peer_p = cluster_addr(p0, sub), peer_bar = cluster_addr(bar0, sub);
    bool ok = true;
    // a warp without a row takes no part: nothing would keep it within a phase of the others (every
    // other warp's entries are part of every phase).  Every block's first warp has rows (iter_first).
    const bool takes_part = lo + (threadIdx.x & ~31u) / kWideLanes < hi;
    for (int it = 0; takes_part; ++it) {
        const int cur = it & 1;
        if (it > 0) {
            // step `it` reads copy `cur` for the ((it - 1) / 2)-th time after its first filling
            ok = __all_sync(0xffffffffu, mbar_wait(bar0 + 8 * cur, ((it - 1) >> 1) & 1, wait.limit_ns));
            if (!ok) break;
            if (threadIdx.x == 0) mbar_expect(bar0 + 8 * cur, bytes);  // for step it + 2
        }
        const float2* p = s_p + cur * cols;
        const uint32_t next_p = peer_p + static_cast<uint32_t>((cur ^ 1) * cols * sizeof(float2));
        const uint32_t next_bar = peer_bar + 8 * (cur ^ 1);
        // NC > 0: one row a thread; NC == 0: whole warps of rows until the share's end
        for (int64_t row = first; NC > 0 ? row == first : row - threadIdx.x / kWideLanes < hi;
             row += step) {
            const bool live = row < hi;
            float2 acc[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                acc[u] = make_float2(0.f, 0.f);
                if constexpr (NC > 0) {
#pragma unroll
                    for (int t = 0; t < NC; ++t)
                        if (32 * t < cols) acc[u] = add(acc[u], cmul(rr[u][t], p[sub + 8 * u + 32 * t]));
                } else {
                    const float2* rrow = r + (live ? row : 0) * m;
                    for (int64_t c = sub + 8 * u; c < m; c += 32) acc[u] = add(acc[u], cmul(rrow[c], p[c]));
                }
            }
            float2 gv = add(add(acc[0], acc[2]), add(acc[1], acc[3]));
            gv = add(gv, shfl_xor2(gv, 4));
            gv = add(gv, shfl_xor2(gv, 2));
            gv = add(gv, shfl_xor2(gv, 1));
            if (!live) gv = make_float2(1.f, 0.f);
            const float amp = live ? amps[row] : 1.f, a = hypotf(gv.x, gv.y);
            if (it == repeat) {
                const float s = amp * amp / (a * a);
                if (live && sub == 0) p_out[row] = make_float2(gv.x * s, gv.y * s);
            } else {
                // an even row's threads store it and the odd row after it (zero past m)
                const float s = live ? amp / a : 0.f;
                const float2 own = make_float2(gv.x * s, gv.y * s), odd = shfl_xor2(own, kWideLanes);
                if (live && !(threadIdx.x & kWideLanes) && !(wait.withhold && rank == 0))
                    store_remote(next_p + static_cast<uint32_t>(row * sizeof(float2)), own, odd, next_bar);
            }
        }
        if (it == repeat) break;
    }
    if (!ok) {
        const float nan = __int_as_float(0x7fffffff);
        for (int64_t row = first; row < hi; row += step) p_out[row] = make_float2(nan, nan);
        *wait.status = 1;
        __threadfence_system();
    }
    cluster.sync();  // no block leaves while another may still store into it
    if (!ok) let_pass(kDrainNs);
}

// q_j = scale_j * sum_i conj(G_ij) p_i, the sum in focus order; writes (|q_j|, arg q_j).  scale =
// inv_den2 or 1.  G and scale were complete before the launch ahead released this one (that
// launch waits for the launches that write them before it releases), so a first chunk of G is
// loaded before the wait for p.
__global__ void __launch_bounds__(kColThreads)
    backpropagate_kernel(const float2* __restrict__ g, const float* __restrict__ scale,
                         const float2* __restrict__ p, int64_t n, int64_t m,
                         float* __restrict__ out) {
    __shared__ float2 s_t[kColChunk][kColSources];
    constexpr int kPer = kColChunk / kColGroups;
    const int lane = threadIdx.x % kColSources, group = threadIdx.x / kColSources;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * kColSources + lane;
    const bool live = j < n;
    float2 v[kPer];
    auto load = [&](int64_t i0) {
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            const int64_t i = i0 + group + t * kColGroups;
            v[t] = live && i < m ? g[i * n + j] : make_float2(0.f, 0.f);
        }
    };
    load(0);
    const float s = live && scale ? scale[j] : 1.0f;
    dev::pdl_wait();
    dev::pdl_release();
    float2 acc = make_float2(0.f, 0.f);
    for (int64_t i0 = 0; i0 < m; i0 += kColChunk) {
        if (i0 > 0) load(i0);
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            const int64_t i = i0 + group + t * kColGroups;
            if (i < m) s_t[group + t * kColGroups][lane] = cmulc(v[t], p[i]);
        }
        __syncthreads();
        if (group == 0) {
            const int cnt = static_cast<int>(m - i0 < kColChunk ? m - i0 : kColChunk);
#pragma unroll 8
            for (int i = 0; i < cnt; ++i) acc = add(acc, s_t[i][lane]);
        }
        __syncthreads();
    }
    if (group != 0 || !live) return;
    acc.x *= s;
    acc.y *= s;
    reinterpret_cast<float2*>(out)[j] = make_float2(hypotf(acc.x, acc.y), atan2f(acc.y, acc.x));
}

// Gerchberg-Saxton (gs.rs:42-77) in one block; q0 are the sources' amplitudes.
__global__ void __launch_bounds__(kIterThreads)
    gs_iterate_kernel(const float2* __restrict__ g, const PackedSource* __restrict__ src,
                      const float* __restrict__ amps, int64_t n, int64_t m, int repeat, float2* q,
                      float2* p, float* __restrict__ out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int64_t j = threadIdx.x; j < n; j += blockDim.x) q[j] = make_float2(src[j].c.z, 0.f);
    __syncthreads();
    for (int it = 0; it < repeat; ++it) {
        // gamma = G q, p = gamma / |gamma| * p0
        for (int64_t row = wid; row < m; row += nw) {
            float2 acc = make_float2(0.f, 0.f);
            for (int64_t j = lane; j < n; j += 32) {
                const float2 t = cmul(g[row * n + j], q[j]);
                acc.x += t.x;
                acc.y += t.y;
            }
            acc = warp_sum(acc);
            if (lane == 0) {
                const float s = amps[row] / hypotf(acc.x, acc.y);
                p[row] = make_float2(acc.x * s, acc.y * s);
            }
        }
        __syncthreads();
        // xi = G^H p, q = xi / |xi| * q0
        for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
            float2 acc = make_float2(0.f, 0.f);
            for (int64_t i = 0; i < m; ++i) {
                const float2 t = cmulc(g[i * n + j], p[i]);
                acc.x += t.x;
                acc.y += t.y;
            }
            const float s = src[j].c.z / hypotf(acc.x, acc.y);
            q[j] = make_float2(acc.x * s, acc.y * s);
        }
        __syncthreads();
    }
    for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
        const float2 v = q[j];
        out[2 * j] = hypotf(v.x, v.y);
        out[2 * j + 1] = atan2f(v.y, v.x);
    }
}

// Greedy (greedy.rs:39-83) in one block.  Source i (in order) tries every candidate phasor
// c_k: thread k sums |amp_j - |G_ji c_k + cache_j|| over the foci j in order (f32, no
// contraction, as the reference); the first minimum wins; cache_j += G_ji c_best.
__global__ void __launch_bounds__(kIterThreads)
    greedy_kernel(const float2* __restrict__ g, const PackedSource* __restrict__ src, int64_t n,
                  int64_t m, const float* __restrict__ amps, const float2* __restrict__ cand,
                  const float* __restrict__ cand_arg, int div, float2* cache,
                  float* __restrict__ out) {
    __shared__ float s_v[kGreedyMaxDiv];
    __shared__ int s_best;
    for (int64_t j = threadIdx.x; j < m; j += blockDim.x) cache[j] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int64_t i = 0; i < n; ++i) {
        if (threadIdx.x < div) {
            const float2 c = cand[threadIdx.x];
            float v = 0.f;
            for (int64_t j = 0; j < m; ++j) {
                const float2 a = g[j * n + i];
                const float2 t = make_float2(__fsub_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y)),
                                             __fadd_rn(__fmul_rn(a.x, c.y), __fmul_rn(a.y, c.x)));
                const float2 q = cache[j];
                const float re = __fadd_rn(t.x, q.x), im = __fadd_rn(t.y, q.y);
                v = __fadd_rn(v, fabsf(__fsub_rn(amps[j], hypotf(re, im))));
            }
            s_v[threadIdx.x] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int best = 0;
            float min_v = __int_as_float(0x7f800000);  // +inf
            for (int k = 0; k < div; ++k) {
                if (s_v[k] < min_v) {
                    min_v = s_v[k];
                    best = k;
                }
            }
            s_best = best;
            out[2 * i] = src[i].c.z;
            out[2 * i + 1] = cand_arg[best];
        }
        __syncthreads();
        const float2 c = cand[s_best];
        for (int64_t j = threadIdx.x; j < m; j += blockDim.x) {
            const float2 a = g[j * n + i];
            const float2 t = make_float2(__fsub_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y)),
                                         __fadd_rn(__fmul_rn(a.x, c.y), __fmul_rn(a.y, c.x)));
            cache[j] = make_float2(__fadd_rn(cache[j].x, t.x), __fadd_rn(cache[j].y, t.y));
        }
        __syncthreads();
    }
}

__global__ void real_to_complex_kernel(const float* __restrict__ v, int64_t m,
                                       float2* __restrict__ out) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < m) out[i] = make_float2(v[i], 0.f);
}

__global__ void fill_amp_phase_kernel(float* out, int64_t n, float amp, float phase) {
    const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n) return;
    out[2 * j] = amp;
    out[2 * j + 1] = phase;
}

unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

size_t solver_workspace_bytes(int64_t n, int64_t m) {
    return align256(sizeof(PackedSource) * n) + align256(sizeof(float2) * n * m) +
           align256(sizeof(float) * n) + align256(sizeof(float2) * m * m) +
           align256(sizeof(float2) * m) + align256(sizeof(float2) * n);
}

cudaError_t launch_build_g(int st, const float* d_raw, const float* d_k, const float* d_atten,
                           int64_t n, const float* d_foci, int64_t m, float2* d_g,
                           void* ws_packed, cudaStream_t s) {
    if (n <= 0 || m <= 0) return cudaSuccess;
    if (m > 65535) return cudaErrorInvalidValue;
    PackedSource* packed = static_cast<PackedSource*>(ws_packed);
    cudaError_t e = launch_pack_sources(st, d_raw, d_k, d_atten, n, packed, s);
    if (e != cudaSuccess) return e;
    const dim3 grid(blocks_for(n, 128), static_cast<unsigned>(m));
    const bool pdl = !stream_capturing(s);
    e = st == SRC_T4010A1
            ? launch_after(build_g_kernel<SRC_T4010A1>, grid, dim3(128), 0, s, pdl, packed, n,
                           d_foci, m, d_g)
            : launch_after(build_g_kernel<SRC_SPHERE>, grid, dim3(128), 0, s, pdl, packed, n,
                           d_foci, m, d_g);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_greedy(int st, const float* d_raw, const float* d_k, const float* d_atten,
                          int64_t n, const float* d_foci, const float* d_amps, int64_t m,
                          const float2* d_cand, const float* d_cand_arg, int div, float* d_out,
                          void* ws, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (m > kSolverMaxFoci || div < 1 || div > kGreedyMaxDiv) return cudaErrorInvalidValue;
    SolverWs w = carve(ws, n, m);
    cudaError_t e = launch_build_g(st, d_raw, d_k, d_atten, n, d_foci, m, w.g, w.packed, s);
    if (e != cudaSuccess) return e;
    if (m == 0) {
        // no foci: launch_build_g did nothing; the packed sources still carry the amplitudes
        if ((e = launch_pack_sources(st, d_raw, d_k, d_atten, n, w.packed, s)) != cudaSuccess)
            return e;
    }
    greedy_kernel<<<1, kIterThreads, 0, s>>>(w.g, w.packed, n, m, d_amps, d_cand, d_cand_arg, div,
                                             w.p, d_out);
    count_launch();
    return cudaGetLastError();
}

namespace {

// The iteration kernel of a GS-PAT solve of m foci on s.
cudaError_t launch_iterate(const float2* r, const float* amps, int64_t m, int repeat, float2* p,
                           cudaStream_t s, bool pdl, unsigned* status, bool wait_test) {
    if (m <= kGspatSmallFoci) {
        const int mi = static_cast<int>(m);
        const dim3 one(1), threads(static_cast<unsigned>((m * kSmallLanes + 31) / 32 * 32));
        if (m <= 8) return launch_after(gspat_iterate_small_kernel<1, true>, one, threads, 0, s, pdl, r, amps, mi, repeat, p);
        if (m <= 16) return launch_after(gspat_iterate_small_kernel<1, false>, one, threads, 0, s, pdl, r, amps, mi, repeat, p);
        if (m <= 32) return launch_after(gspat_iterate_small_kernel<2, false>, one, threads, 0, s, pdl, r, amps, mi, repeat, p);
        if (m <= 48) return launch_after(gspat_iterate_small_kernel<3, false>, one, threads, 0, s, pdl, r, amps, mi, repeat, p);
        return launch_after(gspat_iterate_small_kernel<4, false>, one, threads, 0, s, pdl, r, amps, mi, repeat, p);
    }
    const int64_t share = iter_share(m);
    unsigned threads = static_cast<unsigned>((share * kWideLanes + 31) / 32 * 32);
    if (m > 384) threads = 1024;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kIterCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kIterCluster);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 2 * sizeof(float2) * static_cast<size_t>((m + 31) / 32 * 32);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    const IterWait wait{status, wait_test ? kIterWaitTestNs : kIterWaitNs, wait_test ? 1 : 0};
    if (m <= 128) return cudaLaunchKernelEx(&cfg, gspat_iterate_cluster_kernel<4>, r, amps, m, repeat, p, wait);
    if (m <= 256) return cudaLaunchKernelEx(&cfg, gspat_iterate_cluster_kernel<8>, r, amps, m, repeat, p, wait);
    if (m <= 384) return cudaLaunchKernelEx(&cfg, gspat_iterate_cluster_kernel<12>, r, amps, m, repeat, p, wait);
    const cudaError_t e = fb::allow_dynamic_smem<gspat_iterate_cluster_kernel<0>>(
        static_cast<int>(2 * sizeof(float2) * kSolverMaxFoci));
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, gspat_iterate_cluster_kernel<0>, r, amps, m, repeat, p, wait);
}

}  // namespace

cudaError_t launch_solver(int kind, int st, const float* d_raw, const float* d_k,
                          const float* d_atten, int64_t n, const float* d_foci,
                          const float* d_amps, int64_t m, int repeat, float* d_out, void* ws,
                          cudaStream_t s, unsigned* status, bool wait_test) {
    if (n <= 0) return cudaSuccess;
    if (m > kSolverMaxFoci || repeat < 0 || (kind == SOLVER_GSPAT && !status)) return cudaErrorInvalidValue;
    SolverWs w = carve(ws, n, m);
    if (m == 0) {
        // An empty focus list leaves q = 0 (GS-PAT, naive) or q = NaN (GS, normalising zero).
        const float v = kind == SOLVER_GS ? __builtin_nanf("") : 0.f;
        fill_amp_phase_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d_out, n, v, v);
        count_launch();
        return cudaGetLastError();
    }
    const dim3 col_grid(blocks_for(n, kColSources)), col_block(kColThreads);
    cudaError_t e = cudaSuccess;
    if (kind == SOLVER_GSPAT) {
        // each launch a programmatic dependent of the one before (the kernels wait first)
        const bool pdl = !stream_capturing(s);
        if (st == SRC_T4010A1)
            gspat_g_kernel<SRC_T4010A1><<<col_grid, col_block, 0, s>>>(d_raw, d_k, d_atten, n, d_foci,
                                                                       m, w.g, w.inv_den2);
        else
            gspat_g_kernel<SRC_SPHERE><<<col_grid, col_block, 0, s>>>(d_raw, d_k, d_atten, n, d_foci, m,
                                                                      w.g, w.inv_den2);
        const unsigned tiles = blocks_for(m, kRTile);
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = launch_after(gspat_r_kernel, dim3(tiles, tiles), dim3(kRThreads), 0, s, pdl,
                              static_cast<const float2*>(w.g), static_cast<const float*>(w.inv_den2),
                              n, m, w.r)) != cudaSuccess ||
            (e = launch_iterate(w.r, d_amps, m, repeat, w.p, s, pdl, status, wait_test)) != cudaSuccess ||
            (e = launch_after(backpropagate_kernel, col_grid, col_block, 0, s, pdl,
                              static_cast<const float2*>(w.g), static_cast<const float*>(w.inv_den2),
                              static_cast<const float2*>(w.p), n, m, d_out)) != cudaSuccess)
            return e;
        count_launch(4);
        return cudaGetLastError();
    }
    if ((e = launch_build_g(st, d_raw, d_k, d_atten, n, d_foci, m, w.g, w.packed, s)) != cudaSuccess)
        return e;
    if (kind == SOLVER_NAIVE) {
        real_to_complex_kernel<<<blocks_for(m, 256), 256, 0, s>>>(d_amps, m, w.p);
        backpropagate_kernel<<<col_grid, col_block, 0, s>>>(w.g, nullptr, w.p, n, m, d_out);
        count_launch(2);
    } else if (kind == SOLVER_GS) {
        gs_iterate_kernel<<<1, kIterThreads, 0, s>>>(w.g, w.packed, d_amps, n, m, repeat, w.q, w.p,
                                                     d_out);
        count_launch();
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

namespace {

// Host-level solver state: one stream and grow-only buffers shared by all systems.
struct SolverCtx {
    std::mutex mu;
    int device = -1;
    cudaStream_t stream = nullptr;
    void* d_in = nullptr;
    size_t d_in_cap = 0;
    void* d_ws = nullptr;
    size_t d_ws_cap = 0;
    float* h_io = nullptr;
    float* h_io_dev = nullptr;  // h_io's address for kernels; NULL where the device has none
    size_t h_io_cap = 0;
};

SolverCtx g_solver;

cudaError_t grow_dev(void** p, size_t* cap, size_t bytes) {
    if (bytes <= *cap) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) *cap = bytes;
    return e;
}

}  // namespace

int solve_multi_focus(int kind, int st, float* src, const float* k, const float* atten,
                      int64_t n, const float* foci, const float* amps, int64_t m,
                      std::string* err, int phase_div, bool wait_test) {
    if (m > kSolverMaxFoci) {
        *err = "too many foci (" + std::to_string(m) + " > " + std::to_string(kSolverMaxFoci) + ")";
        return -1;
    }
    const bool greedy = kind == SOLVER_GREEDY;
    if (greedy && (phase_div < 1 || phase_div > kGreedyMaxDiv)) {
        *err = "phase_div must be 1.." + std::to_string(kGreedyMaxDiv);
        return -1;
    }
    if (n == 0) return 0;
    std::lock_guard<std::mutex> lock(g_solver.mu);
    SolverCtx& c = g_solver;
    cudaError_t e;
    auto fail = [&](const char* what) {
        *err = std::string(what) + ": " + cudaGetErrorString(e);
        return -1;
    };
    if (!c.stream) {
        int count = 0;
        e = cudaGetDeviceCount(&count);
        if (e != cudaSuccess || count == 0) {
            *err = "no CUDA device available; this library has no CPU path";
            return -1;
        }
        if ((e = cudaGetDevice(&c.device)) != cudaSuccess) return fail("cudaGetDevice");
        if ((e = cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking)) != cudaSuccess) {
            c.stream = nullptr;
            return fail("cudaStreamCreate");
        }
    }
    DeviceGuard dg;  // the solver's device while it runs; the caller's again on return
    if ((e = dg.set(c.device)) != cudaSuccess) return fail("cudaSetDevice");
    const int stride = source_stride(st);
    // input block: raw | k | atten | foci | amps [| candidate phasors | their arguments, from a
    // 16-byte boundary] ; output: 2n floats
    const size_t base_floats = static_cast<size_t>(n) * (stride + 2) + 4 * static_cast<size_t>(m);
    const size_t cand_off = (base_floats + 3) & ~static_cast<size_t>(3);
    const size_t in_floats = greedy ? cand_off + 3 * static_cast<size_t>(phase_div) : base_floats;
    // a word for GS-PAT's status follows the inputs, and in the pinned block the outputs too
    const size_t o_status = in_floats > static_cast<size_t>(2 * n) ? in_floats : 2 * n;
    const size_t io_floats = o_status + 1;
    if (io_floats * sizeof(float) > c.h_io_cap) {
        if (c.h_io) cudaFreeHost(c.h_io);
        c.h_io = c.h_io_dev = nullptr;
        c.h_io_cap = 0;
        if ((e = cudaHostAlloc(&c.h_io, io_floats * sizeof(float), cudaHostAllocDefault)) !=
            cudaSuccess)
            return fail("cudaHostAlloc");
        c.h_io_cap = io_floats * sizeof(float);
        void* dev = nullptr;
        if (cudaHostGetDevicePointer(&dev, c.h_io, 0) == cudaSuccess) c.h_io_dev = static_cast<float*>(dev);
        else (void)cudaGetLastError();
    }
    float* h = c.h_io;
    memcpy(h, src, sizeof(float) * n * stride);
    memcpy(h + n * stride, k, sizeof(float) * n);
    memcpy(h + n * (stride + 1), atten, sizeof(float) * n);
    memcpy(h + n * (stride + 2), foci, sizeof(float) * 3 * m);
    memcpy(h + n * (stride + 2) + 3 * m, amps, sizeof(float) * m);
    if (greedy) {
        // greedy.rs:21-27: exp(i 2 pi k / phase_div) in f32 (num-complex exp = from_polar(e^0, a))
        // and, for set_phase, their arguments (greedy.rs:79)
        float* hc = h + cand_off;
        for (int q = 0; q < phase_div; ++q) {
            const float a = 2.0f * kPiF * static_cast<float>(q) / static_cast<float>(phase_div);
            hc[2 * q] = 1.0f * cosf(a);
            hc[2 * q + 1] = 1.0f * sinf(a);
            hc[2 * phase_div + q] = atan2f(hc[2 * q + 1], hc[2 * q]);
        }
    }
    auto* h_status = reinterpret_cast<volatile unsigned*>(h + o_status);
    *h_status = 0;
    if (!c.h_io_dev) h[in_floats] = 0.f;  // the device's own word, sent with the inputs
    const size_t in_copy = (in_floats + (c.h_io_dev ? 0 : 1)) * sizeof(float);
    const size_t in_bytes = align256(in_copy) + align256(2 * n * sizeof(float));
    if ((e = grow_dev(&c.d_in, &c.d_in_cap, in_bytes)) != cudaSuccess) return fail("cudaMalloc");
    if ((e = grow_dev(&c.d_ws, &c.d_ws_cap, solver_workspace_bytes(n, m))) != cudaSuccess)
        return fail("cudaMalloc");
    float* d = static_cast<float*>(c.d_in);
    // the solvers write each source's result once, at their end: straight into the pinned block
    // (whose inputs the copy below has taken by then), so that no copy follows the last launch
    float* d_out = c.h_io_dev ? c.h_io_dev
                              : reinterpret_cast<float*>(static_cast<char*>(c.d_in) + align256(in_copy));
    auto* d_status = reinterpret_cast<unsigned*>(c.h_io_dev ? c.h_io_dev + o_status : d + in_floats);
    if ((e = cudaMemcpyAsync(d, h, in_copy, cudaMemcpyHostToDevice, c.stream)) != cudaSuccess)
        return fail("cudaMemcpyAsync");
    if (greedy)
        e = launch_greedy(st, d, d + n * stride, d + n * (stride + 1), n, d + n * (stride + 2),
                          d + n * (stride + 2) + 3 * m, m,
                          reinterpret_cast<const float2*>(d + cand_off),
                          d + cand_off + 2 * phase_div, phase_div, d_out, c.d_ws, c.stream);
    else
        e = launch_solver(kind, st, d, d + n * stride, d + n * (stride + 1), n,
                          d + n * (stride + 2), d + n * (stride + 2) + 3 * m, m, kSolverRepeat,
                          d_out, c.d_ws, c.stream, d_status, wait_test);
    if (e != cudaSuccess) return fail("solver launch");
    if (!c.h_io_dev &&
        ((e = cudaMemcpyAsync(h, d_out, 2 * n * sizeof(float), cudaMemcpyDeviceToHost, c.stream)) !=
             cudaSuccess ||
         (e = cudaMemcpyAsync(h + o_status, d_status, sizeof(unsigned), cudaMemcpyDeviceToHost,
                              c.stream)) != cudaSuccess))
        return fail("cudaMemcpyAsync");
    if ((e = cudaStreamSynchronize(c.stream)) != cudaSuccess) return fail("solver");
    if (*h_status != 0) {  // the drive stays as it was
        *err = kGspatWaitError;
        return -1;
    }
    const int iamp = st == SRC_T4010A1 ? 6 : 3;
    const int iphase = st == SRC_T4010A1 ? 7 : 4;
    for (int64_t j = 0; j < n; ++j) {
        src[j * stride + iamp] = h[2 * j];
        src[j * stride + iphase] = h[2 * j + 1];
    }
    return 0;
}

}  // namespace afc

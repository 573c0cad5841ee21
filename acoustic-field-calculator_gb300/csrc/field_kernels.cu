// Direct source->point summation on sm_103a.
//
// For every observation point x the kernels form
//     p(x) = sum_j A_j D(theta_j) exp(-alpha_j r_j) / r_j * exp(i (phi_j + k_j r_j))
// in FP32, sources in index order, which is the per-pair math of
// acoustic-field-calculator/src/system/uniform_medium.rs:111-120 summed as in :122-128, then
// apply the field transform of field_buffer/{pressure,power,complex_pressure}_field.rs:35-37.
//
// Layout and schedule (the per-block body is in field_body.cuh)
//   * Sources are packed once per call (PackedSource, 48 B) and staged tile by tile into
//     shared memory with every per-source scalar stored twice ((v, v) pairs), so that one
//     LDS.128 yields two packed f32x2 broadcast operands.  All threads of a block read the
//     same source at the same time: shared-memory broadcasts.
//   * Each thread owns 2*PAIRS observation points spaced kThreads apart and processes them two
//     at a time with the sm_100 packed FP32 instructions (FFMA2 / FMUL2 / FADD2), which halves
//     the FP32 instructions issued; MUFU operations stay per point.  The PAIRS pairs of one
//     source are independent, so their instructions interleave; when any of a thread's
//     points has its theta next to a directivity bin edge (a single predicate), those points
//     are corrected after the source, off the interleaved path.
//   * On grids with more than one point along the second axis a thread's points are
//     consecutive along that axis (field_rows_kernel), so the offsets along the other two axes
//     are computed once per source and thread.  A warp's points are a small box there, and where
//     a source sees it inside one directivity bin the warp takes D from a polynomial of its own
//     (field_rows.cuh).  Otherwise both bodies take it from a cos(theta)-indexed table (no acos,
//     no MUFU square root; propagate.cuh): the rows body from the plain table, whose entries
//     neighbouring grid points share, the general body from a lane-replicated copy in dynamic
//     shared memory that scattered points read without bank conflicts.
//   * When every source of a tile points the same way as source 0 (a planar array), cos(theta)
//     comes from n.x - n.s with n.x precomputed per point and n.s per source: two FP32
//     operations per pair instead of four.  Each block decides this per tile.
//   * Each of the 2*PAIRS stores (4 B or 8 B a point) is one contiguous warp store in the general body;
//     in the rows bodies a warp's box makes it several pieces of 32 to 128 bytes (8 points along the first
//     axis by 4 planes of a volume).
//   * Grid points are generated from the grid description, never read from memory.
//   * Launches whose tiles would leave the last wave short either split each point tile's
//     sources over the blocks of a thread-block cluster (field_split_kernel,
//     field_rows_split_kernel): rank r sums its share of the sources, and rank 0 adds the
//     others' partial sums, read from their shared memory, in rank order -- deterministic, no
//     workspace; or, with scratch for partial sums, run the chunked launch (field_chunk_kernel,
//     field_rows_chunk_kernel): persistent blocks over contiguous ranges of the (tile, source)
//     pairs, whose partial sums a second launch adds in source order (field_chunk_combine_kernel;
//     for few points field_chunk_combine_wide_kernel).  A cost model
//     (launch_model.h) picks among the single pass, the split and the chunked launch.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "afc_internal.h"
#include "field_body.cuh"
#include "field_rows.cuh"
#include "launch_model.h"
#include "propagate.cuh"

namespace afc {

namespace {

using namespace fb;

__constant__ float4 c_dir_table[kDirTableSize] = AFC_DIR_TABLE_INIT;

// The general body's lane-replicated directivity table lives in dynamic shared memory
// (kGTableBytes for T4010A1 sources, none for sphere sources).
__device__ __forceinline__ GTable& dynamic_gtab() {
    extern __shared__ __align__(16) unsigned char afc_dyn_smem[];
    return *reinterpret_cast<GTable*>(afc_dyn_smem);
}

// The rows kernels' shared memory (kRowsSmemBytes).
__device__ __forceinline__ RowsSmem& dynamic_rows() {
    extern __shared__ __align__(16) unsigned char afc_dyn_smem[];
    return *reinterpret_cast<RowsSmem*>(afc_dyn_smem);
}

// The field kernels run as programmatic dependents of the launch before them on the stream (the
// source packing, normally): they fill their tables first and call pdl_wait before they read a
// source.

template <int ST, int SUM, bool GRID, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_direct_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g,
                        const float* __restrict__ pts, int64_t m, int field,
                        void* __restrict__ out) {
    __shared__ SmemTile sm;
    GTable& gt = dynamic_gtab();
    load_theta_table(sm, c_dir_table);
    if constexpr (ST == SRC_T4010A1) load_gtab(gt);
    pdl_wait();
    const int64_t first = static_cast<int64_t>(blockIdx.x) * (kThreads * 2 * PAIRS);
    block_points<ST, SUM, PAIRS>(sm, gt, src, n, GRID, g, pts, m, first, field, out);
}

// The partial sums of a cluster's blocks, combined into rank 0's: every rank writes its sums
// into its own staging arrays (free once its last tile is done), rank 0 adds ranks 1 .. S-1's
// (read from their shared memory through the cluster) in rank order.  Both cluster barriers
// are reached by every thread of every block; the second keeps the other ranks' shared memory
// alive until rank 0 has read it.
template <int SUM, int PAIRS>
__device__ __forceinline__ void cluster_combine(float4* staging, float2 (&RE)[PAIRS],
                                                float2 (&IM)[PAIRS], float2 (&CRE)[PAIRS],
                                                float2 (&CIM)[PAIRS]) {
    namespace cg = cooperative_groups;
    constexpr int kPPT = 2 * PAIRS;
    // partial sums (and compensations) of every thread, in the staging arrays once free
    static_assert(sizeof(float2) * (SUM == SUM_COMPENSATED ? 2 : 1) * kPPT * kThreads <=
                      4 * sizeof(float4) * kTile,
                  "partial sums must fit in the first four staging arrays");
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned S = cluster.num_blocks();
    const unsigned rank = cluster.block_rank();
    __syncthreads();  // the staging arrays are free
    float2* part = reinterpret_cast<float2*>(staging);
#pragma unroll
    for (int k = 0; k < kPPT; ++k) {
        part[k * kThreads + threadIdx.x] =
            make_float2(lane_of(RE[k >> 1], k & 1), lane_of(IM[k >> 1], k & 1));
        if constexpr (SUM == SUM_COMPENSATED)
            part[(kPPT + k) * kThreads + threadIdx.x] =
                make_float2(lane_of(CRE[k >> 1], k & 1), lane_of(CIM[k >> 1], k & 1));
    }
    cluster.sync();
    if (rank == 0) {
        for (unsigned q = 1; q < S; ++q) {
            const float2* rp = cluster.map_shared_rank(part, q);
#pragma unroll
            for (int k = 0; k < kPPT; ++k) {
                const float2 v = rp[k * kThreads + threadIdx.x];
                if constexpr (SUM == SUM_PLAIN) {
                    lane_of(RE[k >> 1], k & 1) += v.x;
                    lane_of(IM[k >> 1], k & 1) += v.y;
                } else {
                    const float2 c = rp[(kPPT + k) * kThreads + threadIdx.x];
                    neumaier_add(lane_of(RE[k >> 1], k & 1), lane_of(CRE[k >> 1], k & 1), v.x);
                    neumaier_add(lane_of(RE[k >> 1], k & 1), lane_of(CRE[k >> 1], k & 1), c.x);
                    neumaier_add(lane_of(IM[k >> 1], k & 1), lane_of(CIM[k >> 1], k & 1), v.y);
                    neumaier_add(lane_of(IM[k >> 1], k & 1), lane_of(CIM[k >> 1], k & 1), c.y);
                }
            }
        }
    }
    cluster.sync();
}

// Source range [r c, (r + 1) c) of rank r of S, c = ceil(n / S).
__device__ __forceinline__ void rank_sources(int64_t n, int64_t& s_lo, int64_t& s_hi) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int64_t S = cluster.num_blocks(), rank = cluster.block_rank();
    const int64_t chunk = (n + S - 1) / S;
    s_lo = rank * chunk < n ? rank * chunk : n;
    s_hi = s_lo + chunk < n ? s_lo + chunk : n;
}

// Small launches: a cluster of S blocks per point tile, block rank r summing its share of the
// sources (rank_sources); rank 0 combines the partial sums (cluster_combine) and stores.
template <int ST, int SUM, bool GRID, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_split_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g,
                       const float* __restrict__ pts, int64_t m, int field,
                       void* __restrict__ out) {
    namespace cg = cooperative_groups;
    __shared__ SmemTile sm;
    constexpr int kPPT = 2 * PAIRS;
    GTable& gt = dynamic_gtab();
    load_theta_table(sm, c_dir_table);
    if constexpr (ST == SRC_T4010A1) load_gtab(gt);
    pdl_wait();
    const unsigned S = cg::this_cluster().num_blocks();
    const int64_t first = static_cast<int64_t>(blockIdx.x / S) * (kThreads * kPPT);
    int64_t s_lo, s_hi;
    rank_sources(n, s_lo, s_hi);
    float2 RE[PAIRS], IM[PAIRS], CRE[PAIRS], CIM[PAIRS];
    block_accumulate<ST, SUM, PAIRS>(sm, gt, src, n, s_lo, s_hi, GRID, g, pts, m, first, RE, IM,
                                     CRE, CIM);
    cluster_combine<SUM, PAIRS>(sm.v0, RE, IM, CRE, CIM);
    if (cg::this_cluster().block_rank() == 0)
        block_store<SUM, PAIRS>(RE, IM, CRE, CIM, src, n, GRID, g, pts, first, m, field,
                                out);
}

// Work split of a chunked launch: `items` = tiles x chunks items in tile-major order (item
// t * chunks + c: point tile t against source chunk c); block b of G takes the contiguous items
// [start(b), start(b + 1)), `base` = items / G each and one more for the first `rem` blocks.
struct ChunkSplit {
    int64_t tiles, chunks, chunk;  // chunk: sources per chunk (the last one shorter)
    int64_t base, rem;
    // block that takes item i
    __device__ __forceinline__ int64_t block_of(int64_t i) const {
        const int64_t big = rem * (base + 1);
        return i < big ? i / (base + 1) : rem + (i - big) / base;
    }
    __device__ __forceinline__ int64_t start(int64_t b) const {
        return b * base + (b < rem ? b : rem);
    }
};

// The point tile of point q: blocks of tile_points consecutive points (flat numbering), or the
// rows tiling's tiles (tile_points == 0; warp tiles of 1 << shift[k] indices along axis k, eight
// to a tile, numbered as RowsCell numbers them).
struct TileMap {
    int64_t tile_points;
    int shift[3];
    int64_t tiles0, tiles1, c0, c1;
    __device__ __forceinline__ int64_t tile_of(int64_t q) const {
        if (tile_points > 0) return q / tile_points;
        int64_t i0, i1, i2, rest;
        div_rem(q, c0, rest, i0);
        div_rem(rest, c1, i2, i1);
        return ((i0 >> shift[0]) + tiles0 * ((i1 >> shift[1]) + tiles1 * (i2 >> shift[2]))) /
               (kThreads / 32);
    }
};

// Persistent chunked launch of the general body for launches whose point tiles alone would
// leave the last wave short.  A block's items of one tile are consecutive chunks, i.e. one
// source range: a segment, summed by one block_accumulate pass.  A tile's segments are
// numbered in chunk order (segment k of tile t begins where the k-th block after the tile's
// first item's block begins), and segment k writes its sums at the tile's points to
// partial[k * m + point]; field_chunk_combine_kernel adds them in that order.  The blocks'
// loads differ by one chunk at most.  Each block fills its directivity tables once.
template <int ST, bool GRID, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_chunk_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g,
                       const float* __restrict__ pts, int64_t m, ChunkSplit cs,
                       float2* __restrict__ partial) {
    constexpr int kPPT = 2 * PAIRS;
    __shared__ SmemTile sm;
    GTable& gt = dynamic_gtab();
    load_theta_table(sm, c_dir_table);
    if constexpr (ST == SRC_T4010A1) load_gtab(gt);
    pdl_wait();
    pdl_release();  // the combine launch may be scheduled now; it waits for this grid's end
    const int64_t end = cs.start(blockIdx.x + 1);
    for (int64_t it = cs.start(blockIdx.x); it < end;) {
        const int64_t tile = it / cs.chunks;
        const int64_t tile_end = (tile + 1) * cs.chunks;
        const int64_t seg_end = end < tile_end ? end : tile_end;
        const int64_t c0 = it - tile * cs.chunks, c1 = seg_end - tile * cs.chunks;
        const int64_t lo = c0 * cs.chunk < n ? c0 * cs.chunk : n;
        const int64_t hi = c1 * cs.chunk < n ? c1 * cs.chunk : n;
        const int64_t k = cs.block_of(it) - cs.block_of(tile * cs.chunks);
        const int64_t first = tile * (kThreads * kPPT);
        float2 RE[PAIRS], IM[PAIRS], CRE[PAIRS], CIM[PAIRS];
        block_accumulate<ST, SUM_PLAIN, PAIRS>(sm, gt, src, n, lo, hi, GRID, g, pts, m, first, RE,
                                               IM, CRE, CIM);
        float2* part = partial + k * m;
#pragma unroll
        for (int j = 0; j < kPPT; ++j) {
            const int64_t q = first + threadIdx.x + static_cast<int64_t>(j) * kThreads;
            if (q >= m) break;
            part[q] = make_float2(lane_of(RE[j >> 1], j & 1), lane_of(IM[j >> 1], j & 1));
        }
        it = seg_end;
    }
}

// The same over the rows tiling's tiles (rows_accumulate): a segment writes its sums at its
// tile's grid points.
template <int ST, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_rows_chunk_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g, RowsMap map,
                            int64_t m, ChunkSplit cs, float2* __restrict__ partial) {
    RowsSmem& rs = dynamic_rows();
    load_theta_table(rs.sm, c_dir_table);
    load_rows_table(rs.rt);
    pdl_wait();
    pdl_release();
    const int64_t end = cs.start(blockIdx.x + 1);
    for (int64_t it = cs.start(blockIdx.x); it < end;) {
        const int64_t tile = it / cs.chunks;
        const int64_t tile_end = (tile + 1) * cs.chunks;
        const int64_t seg_end = end < tile_end ? end : tile_end;
        const int64_t ca = it - tile * cs.chunks, cb = seg_end - tile * cs.chunks;
        const int64_t lo = ca * cs.chunk < n ? ca * cs.chunk : n;
        const int64_t hi = cb * cs.chunk < n ? cb * cs.chunk : n;
        const int64_t k = cs.block_of(it) - cs.block_of(tile * cs.chunks);
        float2 RE[PAIRS], IM[PAIRS], CRE[PAIRS], CIM[PAIRS];
        rows_accumulate<ST, SUM_PLAIN, PAIRS>(rs, src, n, lo, hi, g, map, tile, RE, IM, CRE, CIM);
        rows_store_partial<PAIRS>(g, map, tile, RE, IM, partial + k * m);
        it = seg_end;
    }
}

// A combined point's field: the field transform, and the coincident-source fix-up of the single-pass
// kernels for NaN sums.
template <bool GRID>
__device__ __forceinline__ void store_combined(const PackedSource* __restrict__ src, int64_t n,
                                               const GridDev& g, const float* __restrict__ pts,
                                               int64_t q, int field, void* __restrict__ out, float re,
                                               float im) {
    store_field(out, q, field, re, im);
    if (isnan(re) || isnan(im)) {
        float x, y, z;
        if (GRID) {
            grid_point(g, q, x, y, z);
        } else {
            x = pts[3 * q];
            y = pts[3 * q + 1];
            z = pts[3 * q + 2];
        }
        fix_coincident(src, n, x, y, z, q, field, out);
    }
}

// The fields of a chunked launch: each point's segment sums added in segment order.
template <bool GRID>
__global__ void __launch_bounds__(256)
    field_chunk_combine_kernel(const float2* __restrict__ partial, ChunkSplit cs, TileMap tm,
                               const PackedSource* __restrict__ src, int64_t n, GridDev g,
                               const float* __restrict__ pts, int64_t m, int field,
                               void* __restrict__ out) {
    // launched as a programmatic dependent of the chunk kernel: its partial sums are complete
    // and visible once this returns
    pdl_wait();
    for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < m;
         q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t t0 = tm.tile_of(q) * cs.chunks;
        const int64_t segs = cs.block_of(t0 + cs.chunks - 1) - cs.block_of(t0) + 1;
        float re = 0.f, im = 0.f;
        for (int64_t k = 0; k < segs; ++k) {
            const float2 v = partial[k * m + q];
            re = __fadd_rn(re, v.x);
            im = __fadd_rn(im, v.y);
        }
        store_combined<GRID>(src, n, g, pts, q, field, out, re, im);
    }
}

// The same for few points of many segments (few tiles; a point's segments then number up to the GPU's
// blocks): a block takes 32 points, its eight warps bring in their segments, kWideAhead loads a
// thread on the way at once, and one warp adds them, in the same order.  Bound by those loads'
// latency: a thread a point waits for them a few at a time (2,089 points x 153 segments 12.4 us, so
// 5.7).  From kWideSegments on, about ten tiles: the call takes 21.9 us against 38 at 1,000 points x
// 2,490 sources, 60.0 against 62.1 at 16,000, 73.0 both at 20,000 (31 segments), and 112.9 against
// 111.2 at 33,553 (19).
constexpr int kWideAhead = 16;
constexpr int kWideSegments = 32;

template <bool GRID>
__global__ void __launch_bounds__(256)
    field_chunk_combine_wide_kernel(const float2* __restrict__ partial, ChunkSplit cs, TileMap tm,
                                    const PackedSource* __restrict__ src, int64_t n, GridDev g,
                                    const float* __restrict__ pts, int64_t m, int field,
                                    void* __restrict__ out) {
    constexpr int kRound = 8 * kWideAhead;
    __shared__ float2 s_v[kRound][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    int segs = 0;
    if (q < m) {
        const int64_t t0 = tm.tile_of(q) * cs.chunks;
        segs = static_cast<int>(cs.block_of(t0 + cs.chunks - 1) - cs.block_of(t0)) + 1;
    }
    const int most = __reduce_max_sync(0xffffffffu, segs);  // of the block: its warps hold the same points
    pdl_wait();
    float re = 0.f, im = 0.f;
    for (int k0 = 0; k0 < most; k0 += kRound) {
        float2 v[kWideAhead];
#pragma unroll
        for (int u = 0; u < kWideAhead; ++u) {
            const int k = k0 + warp + 8 * u;
            if (k < segs) v[u] = partial[k * m + q];
        }
#pragma unroll
        for (int u = 0; u < kWideAhead; ++u) {
            const int k = k0 + warp + 8 * u;
            if (k < segs) s_v[k - k0][lane] = v[u];
        }
        __syncthreads();
        if (warp == 0) {
            const int end = min(segs - k0, kRound);
#pragma unroll 8
            for (int k = 0; k < end; ++k) {
                const float2 w = s_v[k][lane];
                re = __fadd_rn(re, w.x);
                im = __fadd_rn(im, w.y);
            }
        }
        __syncthreads();
    }
    if (warp == 0 && q < m) store_combined<GRID>(src, n, g, pts, q, field, out, re, im);
}

// Mid-size grids: the rows tiling with every tile's sources split over a cluster of S blocks,
// S chosen so that the launch fills whole waves (split_width); rank 0 combines and stores.
template <int ST, int SUM, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_rows_split_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g, RowsMap map,
                            int field, void* __restrict__ out) {
    namespace cg = cooperative_groups;
    RowsSmem& rs = dynamic_rows();
    load_theta_table(rs.sm, c_dir_table);
    load_rows_table(rs.rt);
    pdl_wait();
    const int64_t tile = blockIdx.x / cg::this_cluster().num_blocks();
    int64_t s_lo, s_hi;
    rank_sources(n, s_lo, s_hi);
    float2 RE[PAIRS], IM[PAIRS], CRE[PAIRS], CIM[PAIRS];
    rows_accumulate<ST, SUM, PAIRS>(rs, src, n, s_lo, s_hi, g, map, tile, RE, IM, CRE, CIM);
    cluster_combine<SUM, PAIRS>(rs.sm.v[0], RE, IM, CRE, CIM);
    if (cg::this_cluster().block_rank() == 0)
        rows_store<SUM, PAIRS>(src, n, g, map, tile, RE, IM, CRE, CIM, field, out);
}

// Grids with more than one point along their second axis: one tile of the rows tiling a block
// (field_rows.cuh).
template <int ST, int SUM, int PAIRS>
__global__ void __launch_bounds__(kThreads, 2)
    field_rows_kernel(const PackedSource* __restrict__ src, int64_t n, GridDev g, RowsMap map,
                      int field, void* __restrict__ out) {
    RowsSmem& rs = dynamic_rows();
    load_theta_table(rs.sm, c_dir_table);
    load_rows_table(rs.rt);
    pdl_wait();
    block_rows<ST, SUM, PAIRS>(rs, src, n, g, map, blockIdx.x, field, out);
}

__global__ void pack_sources_kernel(int st, const float* __restrict__ raw,
                                    const float* __restrict__ k, const float* __restrict__ atten,
                                    int64_t n, PackedSource* __restrict__ out) {
    // the launch after this one (a field kernel or the G build) may start its table fills now;
    // it waits for this grid before it reads a source
    pdl_release();
    const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n) return;
    out[j] = pack_source(st, raw, k, atten, j);
}

// SM count per device (0: not queried yet); devices past the cache are queried every time.
constexpr int kSmCacheDevices = 64;
constexpr int kFallbackSms = 148;
std::atomic<int> g_num_sms[kSmCacheDevices] = {};

// Blocks of Kernel that can be resident at once: launched alone (S = 1) or in clusters of S
// blocks, where the occupancy calculator's count of co-resident clusters also sees how clusters
// pack into the GPCs (7-block clusters, for one, leave some slots of every GPC empty).  Cached
// per device and S; 2 blocks per SM if the query fails.
template <auto Kernel>
int64_t resident_blocks(int64_t S, int dyn) {
    static std::atomic<int> cache[kSmCacheDevices][model::kMaxClusterBlocks + 1];
    if (S < 1 || S > model::kMaxClusterBlocks) return 2LL * num_sms();
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = kSmCacheDevices;
    if (dev < kSmCacheDevices) {
        const int v = cache[dev][S].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    int64_t v = 0;
    if (allow_dynamic_smem<Kernel>(dyn) == cudaSuccess) {
        if (S == 1) {
            int b = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, Kernel, kThreads, dyn) ==
                cudaSuccess)
                v = static_cast<int64_t>(b) * num_sms();
        } else {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(S), 1, 1);
            cfg.blockDim = dim3(kThreads, 1, 1);
            cfg.dynamicSmemBytes = static_cast<size_t>(dyn);
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = static_cast<unsigned>(S);
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int c = 0;
            if (cudaOccupancyMaxActiveClusters(&c, Kernel, &cfg) == cudaSuccess)
                v = static_cast<int64_t>(c) * S;
        }
    }
    if (v <= 0) {
        (void)cudaGetLastError();  // a failed query must not surface as the next launch's error
        return 2LL * num_sms();
    }
    if (dev < kSmCacheDevices) cache[dev][S].store(static_cast<int>(v), std::memory_order_relaxed);
    return v;
}

// Launches a field kernel on `grid` blocks of kThreads with `dyn` bytes of dynamic shared memory
// on s: in clusters of `cluster` blocks when that is above one, and with `pdl` as a programmatic
// dependent of the launch before it (the kernel fills its tables, then waits in pdl_wait).
template <typename... KArgs, typename... Args>
cudaError_t launch_field_kernel(void (*kernel)(KArgs...), int64_t grid, int dyn, cudaStream_t s,
                                unsigned cluster, bool pdl, Args... args) {
    cudaLaunchAttribute attr[2];
    unsigned na = 0;
    if (cluster > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = cluster;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(dyn);
    cfg.stream = s;
    cfg.attrs = na ? attr : nullptr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Chunked launches (field_chunk_kernel): chunks of kChunkSources sources (one: the blocks'
// loads differ by one source iteration at most; a block's consecutive chunks of a tile are one
// pass whatever their size), partial sums of at most kChunkMaxBytes.
constexpr int64_t kChunkSources = 1;
constexpr int64_t kChunkMaxBytes = 256LL << 20;

// The work split of a chunked launch of `tiles` tiles and n sources on `blocks` blocks, and the
// partial-sum slots it needs per point (the most segments any tile has).
ChunkSplit chunk_split(int64_t tiles, int64_t n, int64_t blocks, int64_t* slots_per_point) {
    ChunkSplit cs{};
    cs.tiles = tiles;
    cs.chunks = (n + kChunkSources - 1) / kChunkSources;
    cs.chunk = kChunkSources;
    const int64_t items = tiles * cs.chunks;
    if (blocks > items) blocks = items;
    cs.base = items / blocks;
    cs.rem = items % blocks;
    // a tile's chunks - 1 item boundaries after its first item start at most
    // ceil((chunks - 1) / base) more blocks
    *slots_per_point = cs.base > 0 ? (cs.chunks - 1 + cs.base - 1) / cs.base + 1 : cs.chunks;
    return cs;
}

// Per-device pool of the chunked launches' partial sums: stream-ordered allocations that keep
// up to kChunkMaxBytes after they are freed, so that repeated calls do not return memory to the
// driver and take it again.
std::mutex g_pool_mu;
cudaMemPool_t g_pools[kSmCacheDevices] = {};

cudaError_t scratch_alloc(void** ptr, size_t bytes, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kSmCacheDevices) return cudaErrorMemoryAllocation;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        if (!g_pools[dev]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.handleTypes = cudaMemHandleTypeNone;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            if ((e = cudaMemPoolCreate(&pool, &props)) != cudaSuccess) return e;
            uint64_t keep = static_cast<uint64_t>(kChunkMaxBytes);
            if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)) !=
                cudaSuccess) {
                cudaMemPoolDestroy(pool);
                return e;
            }
            g_pools[dev] = pool;
        }
        pool = g_pools[dev];
    }
    return cudaMallocFromPoolAsync(ptr, bytes, pool, s);
}

// Dynamic shared memory of a general-body kernel for source type ST.
template <int ST>
constexpr int gtab_bytes() {
    return ST == SRC_T4010A1 ? kGTableBytes : 0;
}

// A chunked launch of the general body (field_chunk_kernel + field_chunk_combine_kernel) on
// `blocks` persistent blocks.  cudaErrorMemoryAllocation: no scratch for the partial sums
// (nothing was launched).
template <int ST, bool GRID, int PAIRS>
cudaError_t launch_chunked(const PackedSource* src, int64_t n, const PointSet& ps, int field,
                           void* out, cudaStream_t s, int64_t tiles, int64_t blocks, bool pdl,
                           const RowsTiling* rows = nullptr) {
    constexpr int kDyn = gtab_bytes<ST>();
    int64_t slots = 0;
    const ChunkSplit cs = chunk_split(tiles, n, blocks, &slots);
    const size_t bytes = sizeof(float2) * static_cast<size_t>(slots) * static_cast<size_t>(ps.m);
    if (static_cast<int64_t>(bytes) > kChunkMaxBytes) return cudaErrorMemoryAllocation;
    void* partial = nullptr;
    if (scratch_alloc(&partial, bytes, s) != cudaSuccess) {
        (void)cudaGetLastError();
        return cudaErrorMemoryAllocation;
    }
    const int64_t items = tiles * cs.chunks;
    const unsigned grid_blocks = static_cast<unsigned>(blocks < items ? blocks : items);
    TileMap tm{static_cast<int64_t>(kThreads) * 2 * PAIRS, {0, 0, 0}, 0, 0, 0, 0};
    cudaError_t e = cudaSuccess;
    if (rows) {
        constexpr int kPairBits = PAIRS == 4 ? 3 : 2;  // log2 of a thread's points
        const RowsMap& map = rows->map;
        tm = TileMap{0, {map.bits[0], map.bits[1] + kPairBits, map.bits[2]}, map.tiles0, map.tiles1,
                     static_cast<int64_t>(ps.grid.count[0]), static_cast<int64_t>(ps.grid.count[1])};
        e = allow_dynamic_smem<field_rows_chunk_kernel<ST, PAIRS>>(kRowsSmemBytes);
        if (e == cudaSuccess)
            e = launch_field_kernel(field_rows_chunk_kernel<ST, PAIRS>, grid_blocks, kRowsSmemBytes,
                                    s, 1, pdl, src, n, ps.grid, map, ps.m, cs,
                                    static_cast<float2*>(partial));
        count_launch();
        if (e == cudaSuccess) e = cudaGetLastError();
    } else if ((e = allow_dynamic_smem<field_chunk_kernel<ST, GRID, PAIRS>>(kDyn)) == cudaSuccess) {
        e = launch_field_kernel(field_chunk_kernel<ST, GRID, PAIRS>, grid_blocks, kDyn, s, 1, pdl,
                                src, n, ps.grid, ps.pts, ps.m, cs, static_cast<float2*>(partial));
        count_launch();
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        // a programmatic dependent of the chunk kernel: its launch overlaps that grid's tail
        const bool wide = slots >= kWideSegments;
        const int64_t want = wide ? (ps.m + 31) / 32 : std::min<int64_t>((ps.m + 255) / 256, 8LL * num_sms());
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(want));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, wide ? field_chunk_combine_wide_kernel<GRID> : field_chunk_combine_kernel<GRID>,
                               static_cast<const float2*>(partial), cs, tm, src, n, ps.grid,
                               ps.pts, ps.m, field, out);
        count_launch();
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    const cudaError_t ef = cudaFreeAsync(partial, s);
    return e != cudaSuccess ? e : ef;
}

// `capturing`: s is being captured into a graph, which takes neither the chunked launch nor
// programmatic dependences.
template <int ST, int SUM, int PAIRS>
cudaError_t launch_pairs(const PackedSource* src, int64_t n, const PointSet& ps, int field,
                         void* out, cudaStream_t s, bool scratch_ok, bool capturing) {
    constexpr int kDyn = gtab_bytes<ST>();
    const bool pdl = !capturing;
    const int64_t per_block = static_cast<int64_t>(kThreads) * 2 * PAIRS;
    const int64_t flat_blocks = (ps.m + per_block - 1) / per_block;
    const RowsTiling rows = ps.is_grid ? rows_tiling(ST, ps.grid, ps.m, PAIRS) : RowsTiling{};
    // the chunked launch numbers tiles x sources work items in 64 bits: only below 2^62 of them
    const bool chunk_fits = n < (1LL << 31) && flat_blocks < (1LL << 31);
    auto flat_slots = [](int64_t w) {
        return w <= 1 ? resident_blocks<field_direct_kernel<ST, SUM, false, PAIRS>>(1, kDyn)
                      : resident_blocks<field_split_kernel<ST, SUM, false, PAIRS>>(w, kDyn);
    };
    if constexpr (PAIRS == 4 && SUM == SUM_PLAIN) if (!rows.use && scratch_ok && chunk_fits && n >= 2 * kChunkSources) {
        // chunked (not while the stream is being captured: the partial sums are allocated on
        // the stream) when the model puts it below the launch that would run instead
        if (!capturing) {
            const int64_t S = model::split_width(flat_blocks, n, flat_slots);
            const int64_t blocks =
                ps.is_grid ? resident_blocks<field_chunk_kernel<ST, true, PAIRS>>(1, kDyn)
                           : resident_blocks<field_chunk_kernel<ST, false, PAIRS>>(1, kDyn);
            if (model::chunk_cost(flat_blocks, n, blocks, num_sms()) <
                model::chunk_bar(flat_blocks, n, S, flat_slots(S), num_sms(), model::kSplitMargin)) {
                const cudaError_t e =
                    ps.is_grid ? launch_chunked<ST, true, PAIRS>(src, n, ps, field, out, s, flat_blocks, blocks, pdl)
                               : launch_chunked<ST, false, PAIRS>(src, n, ps, field, out, s, flat_blocks, blocks, pdl);
                if (e != cudaErrorMemoryAllocation) return e;
            }
        }
    }
    if (!rows.use) {
        // flat numbering whose blocks would leave the last wave short (or the GPU part empty):
        // split each tile's sources over a cluster
        const int64_t S = model::split_width(flat_blocks, n, flat_slots);
        if (S >= 2 && flat_blocks * S <= 0x7fffffffLL) {
            const unsigned cl = static_cast<unsigned>(S);
            const bool overlap =
                pdl && model::split_overlaps_packing(flat_blocks * S, n, S, flat_slots(S));
            cudaError_t e;
            if (ps.is_grid) {
                e = allow_dynamic_smem<field_split_kernel<ST, SUM, true, PAIRS>>(kDyn);
                if (e == cudaSuccess)
                    e = launch_field_kernel(field_split_kernel<ST, SUM, true, PAIRS>, flat_blocks * S,
                                            kDyn, s, cl, overlap, src, n, ps.grid,
                                            static_cast<const float*>(nullptr), ps.m, field, out);
            } else {
                e = allow_dynamic_smem<field_split_kernel<ST, SUM, false, PAIRS>>(kDyn);
                if (e == cudaSuccess)
                    e = launch_field_kernel(field_split_kernel<ST, SUM, false, PAIRS>, flat_blocks * S,
                                            kDyn, s, cl, overlap, src, n, ps.grid, ps.pts, ps.m, field,
                                            out);
            }
            count_launch();
            return e != cudaSuccess ? e : cudaGetLastError();
        }
    }
    if (ps.is_grid) {
        const RowsTiling& t = rows;
        if (t.use) {
            if (t.blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
            auto rows_slots = [](int64_t w) {
                return w <= 1 ? resident_blocks<field_rows_kernel<ST, SUM, PAIRS>>(1, kRowsSmemBytes)
                              : resident_blocks<field_rows_split_kernel<ST, SUM, PAIRS>>(w, kRowsSmemBytes);
            };
            const int64_t S = model::split_width(t.blocks, n, rows_slots);
            if constexpr (PAIRS == 4 && SUM == SUM_PLAIN) if (scratch_ok && chunk_fits && n >= 2 * kChunkSources) {
                // the chunked launch over the rows tiles, on the same terms as the flat one
                if (!capturing) {
                    const int64_t blocks = resident_blocks<field_rows_chunk_kernel<ST, PAIRS>>(1, kRowsSmemBytes);
                    if (model::chunk_cost(t.blocks, n, blocks, num_sms()) <
                        model::chunk_bar(t.blocks, n, S, rows_slots(S), num_sms(), 1.0)) {
                        const cudaError_t e = launch_chunked<ST, true, PAIRS>(
                            src, n, ps, field, out, s, t.blocks, blocks, pdl, &t);
                        if (e != cudaErrorMemoryAllocation) return e;
                    }
                }
            }
            if (S >= 2 && t.blocks * S <= 0x7fffffffLL) {
                cudaError_t e = allow_dynamic_smem<field_rows_split_kernel<ST, SUM, PAIRS>>(kRowsSmemBytes);
                if (e == cudaSuccess)
                    e = launch_field_kernel(
                        field_rows_split_kernel<ST, SUM, PAIRS>, t.blocks * S, kRowsSmemBytes, s,
                        static_cast<unsigned>(S),
                        pdl && model::split_overlaps_packing(t.blocks * S, n, S, rows_slots(S)), src, n,
                        ps.grid, t.map, field, out);
                count_launch();
                return e != cudaSuccess ? e : cudaGetLastError();
            }
            cudaError_t e = allow_dynamic_smem<field_rows_kernel<ST, SUM, PAIRS>>(kRowsSmemBytes);
            if (e == cudaSuccess)
                e = launch_field_kernel(field_rows_kernel<ST, SUM, PAIRS>, t.blocks, kRowsSmemBytes, s,
                                        1, pdl, src, n, ps.grid, t.map, field, out);
            count_launch();
            return e != cudaSuccess ? e : cudaGetLastError();
        }
    }
    const int64_t blocks = flat_blocks;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    cudaError_t e;
    if (ps.is_grid) {
        if ((e = allow_dynamic_smem<field_direct_kernel<ST, SUM, true, PAIRS>>(kDyn)) != cudaSuccess)
            return e;
        e = launch_field_kernel(field_direct_kernel<ST, SUM, true, PAIRS>, blocks, kDyn, s, 1, pdl,
                                src, n, ps.grid, static_cast<const float*>(nullptr), ps.m, field, out);
    } else {
        if ((e = allow_dynamic_smem<field_direct_kernel<ST, SUM, false, PAIRS>>(kDyn)) != cudaSuccess)
            return e;
        e = launch_field_kernel(field_direct_kernel<ST, SUM, false, PAIRS>, blocks, kDyn, s, 1, pdl,
                                src, n, ps.grid, ps.pts, ps.m, field, out);
    }
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

// Points per thread, the cluster split or the chunked launch refilling the waves.  Scatter
// points and single-row grids: 4 point pairs from 32,768 points, one below (3,984 sources:
// 65,536 points ran 24 % and 262,144 points 2 % faster with 4 pairs than with one; 16,384
// points ran 40 % slower with 2 pairs than with one, its 16 tiles too few even split 8 ways).
// Where the chunked launch is open, point sets from 2,048 points against at least 1,024
// sources (and 5e6 evaluations), and any against at least 1,536, take 4 point pairs too (below), T4010A1
// grids of the rows tiling from 768 sources where the model says so (rows_four_pairs), and sphere
// sources fewer than 1,024 only from kSphereFourFrom evaluations.
// Grids with more than one point along their second axis, whose rows body shares two
// coordinates per thread: 4 point pairs from 32,768 points where the chunked launch is open
// (scratch allowed, no stream capture; 3,984 sources: 40^3 and 48^3 grids ran 12 % and 6 %
// faster, 200^2, 256^2 and 360^2 slices 19-25 %), else from 73,728 or 131,072 points and 2 from 32,768
// (40^3, 64^3 and 80^3 grids ran 4-9 % faster than with fewer pairs under the cluster split);
// slices against 768 sources or more 2 from 28,672 (160 x 200 points, 996 sources: 49.7 us against 56.4 with
// one; 256 x 100: 49.6 against 45.1; 178 x 182, 249 sources: 24.6 against 22.6).
constexpr double kSphereFourFrom = 7e7;
constexpr double kSphereFourFromUncut = 2e9;

// T4010A1 grids in the rows tiling, whose polynomials want four pairs, against 768 to 1,023 sources: whether
// the chunked launch of four pairs models below the cluster split of one pair, whose source iterations
// take kOnePairRate of the time (0.20 us against 0.56).  996 sources, split and chunked: 64 x 42 x 2
// points 24.7 us and 21.0, 49 x 32 x 9 32.9 and 30.8, 44 x 45 x 9 (one full wave of the split) 32.9 and
// 37.4, 201 x 160 53.4 and 47.7.  38 such grids of 5,376 to 32,160 points take 0.2 % longer than the better
// way on average, at most 4.6 % (51 x 56 x 9).
constexpr double kOnePairRate = 0.36;

template <int ST>
bool rows_four_pairs(int64_t n, const PointSet& ps) {
    const RowsTiling four = rows_tiling(ST, ps.grid, ps.m, 4), one = rows_tiling(ST, ps.grid, ps.m, 1);
    if (!four.use) return false;
    auto slots = [&](int64_t w) {
        if (one.use)
            return w <= 1 ? resident_blocks<field_rows_kernel<ST, SUM_PLAIN, 1>>(1, kRowsSmemBytes)
                          : resident_blocks<field_rows_split_kernel<ST, SUM_PLAIN, 1>>(w, kRowsSmemBytes);
        constexpr int kDyn = gtab_bytes<ST>();
        return w <= 1 ? resident_blocks<field_direct_kernel<ST, SUM_PLAIN, false, 1>>(1, kDyn)
                      : resident_blocks<field_split_kernel<ST, SUM_PLAIN, false, 1>>(w, kDyn);
    };
    const int64_t tiles = one.use ? one.blocks : (ps.m + 2 * kThreads - 1) / (2 * kThreads);
    const int64_t S = model::split_width(tiles, n, slots);
    const int64_t blocks = resident_blocks<field_rows_chunk_kernel<ST, 4>>(1, kRowsSmemBytes);
    return model::chunk_cost(four.blocks, n, blocks, num_sms()) <
           kOnePairRate * model::pass_cost(tiles, n, S, slots(S), num_sms());
}

template <int ST>
cudaError_t launch_st(int sum_mode, const PackedSource* src, int64_t n, const PointSet& ps,
                      int field, void* out, cudaStream_t s, bool scratch_ok) {
    const bool capturing = stream_capturing(s);
    if (sum_mode == SUM_COMPENSATED)
        return launch_pairs<ST, SUM_COMPENSATED, 2>(src, n, ps, field, out, s, false, capturing);
    const bool chunk_open = scratch_ok && !capturing;
    const bool rows_grid = ps.is_grid && ps.grid.count[1] > 1;  // the rows body can take it
    // without the chunked launch (serving, capture, no-alloc calls) the cluster split wants tiles to
    // spare: T4010A1 grids in the rows tiling take four pairs from 73,728 points (two pairs, four: 249
    // sources on 90,534 points 43.2 us and 37.1, 996 on 75,600 118.6 and 102.9, 2,490 on 90,761 275 and 249;
    // 498 on 91,709 64.3 and 71.9), other grids from 131,072
    int64_t four_from = 32768;
    if (rows_grid && !chunk_open)
        four_from = ST == SRC_T4010A1 && rows_tiling(ST, ps.grid, ps.m, 4).use ? 73728 : 131072;
    // small point sets against many sources: the split's S <= 8 ranks leave most SMs idle, the
    // chunked launch spreads the sources over all of them (3,984 sources: 2,048 to 24,576
    // scatter points ran 1.2-2.4x faster, 100^2 and 150^2 slices 1.5x and 1.2x); below about
    // 5e6 evaluations its fixed cost outweighs that (249 sources on 101^2: 21 -> 35 us), except
    // against so many sources that eight ranks sum them longer than it (100 to 2,000 points against
    // 996 sources: split 21-23 us, chunked 26-30; 2,490: 41-43 and 30-33; 3,984: 60-64 and 33-38)
    const double evals = static_cast<double>(n) * static_cast<double>(ps.m);
    if (chunk_open && n >= 1536)
        four_from = 1;
    else if (chunk_open && n >= 1024 && evals >= 5e6)
        four_from = 2048;
    else if (chunk_open && ST == SRC_T4010A1 && rows_grid && n >= 768 && evals >= 5e6 &&
             rows_four_pairs<ST>(n, ps))
        four_from = 2048;
    // Against fewer sources those of one pair are short passes too, and sphere sources, which share no
    // directivity, gain nothing by four pairs until then: the whole range is one pair's (one pair, four
    // pairs: 249 sources on 45,954 points 18.5 us and 28.8, on 94,068 27.9 and 32.9; 498 on 53,628 31.7
    // and 41.1; 996 on 33,936 37.1 and 45.6, on 69,776 65.8 and 69.9, on 84,064 86.3 and 78.3)
    // Without the chunked launch one pair's small tiles split best at nearly any size (old choice, one
    // pair: 3,984 sources on 41,360 points 182 us and 146, on 234,360 918 and 746, 996 on 240,540 241 and 202,
    // 2,490 on 783,900 1,626 and 1,535; 249 on 2,508,800 520 and 531).
    if (ST == SRC_SPHERE && (chunk_open ? n < 1024 && evals < kSphereFourFrom : evals < kSphereFourFromUncut))
        return launch_pairs<ST, SUM_PLAIN, 1>(src, n, ps, field, out, s, scratch_ok, capturing);
    const int64_t two_from =
        rows_grid ? (ps.grid.count[2] == 1 && n >= 768 ? 28672 : 32768) : INT64_MAX;
    if (ps.m >= four_from)
        return launch_pairs<ST, SUM_PLAIN, 4>(src, n, ps, field, out, s, scratch_ok, capturing);
    if (ps.m >= two_from)
        return launch_pairs<ST, SUM_PLAIN, 2>(src, n, ps, field, out, s, scratch_ok, capturing);
    return launch_pairs<ST, SUM_PLAIN, 1>(src, n, ps, field, out, s, scratch_ok, capturing);
}

}  // namespace

std::atomic<uint64_t> g_launches{0};

// Threads past the grid's edges are idle in the rows tiling; its pairs cost 25 % less than the flat
// numbering's (T4010A1: with 76 % of its threads busy 95 us against 97, with 83 % 670 against 765),
// those of sphere sources, which have no directivity to share, 6 % (83 % busy: 303 us against 277,
// 93 %: 2,148 against 2,112, 95 %: 1,891 against 1,910, 99 %: 606 against 639).
constexpr double kRowsBusy = 0.8;
constexpr double kRowsBusyTwo = 0.9;  // two pairs: 88 % busy 407 us (flat 354), 61 (56); 90 % 174 (182)
constexpr double kRowsBusySphere = 0.94;
// With one pair a thread the rows body has no polynomials and shares its per-source work between
// two points only: 249 sources on 128 x 80 points took 14.6 us in the flat numbering and 16.4 in
// the rows tiling, 996 sources 34.9 and 34.9; on 256 x 100 points 49.3 and 45.1 (996 sources).  Sphere
// sources gain nothing by it at any size (249 sources on 163 x 124 14.4 and 15.2, 498 on 396 x 161 37.0 and 38.2).
constexpr int64_t kRowsOnePairFrom = 16384;

RowsTiling rows_tiling(int st, const GridDev& g, int64_t m, int pairs) {
    RowsTiling t{};
    if (g.count[1] <= 1 || m <= 0) return t;
    if (pairs == 1 && (st == SRC_SPHERE || g.count[2] > 1 || m < kRowsOnePairFrom)) return t;
    const int pair_bits = pairs == 4 ? 3 : (pairs == 2 ? 2 : 1);  // log2 of a thread's points
    // The warp's 5 lane bits over the three axes: among all splits the fewest warp tiles, each
    // index of the warp box's extents (their sum) counted as 0.5 % of the time, since the longer a
    // warp's box, the fewer sources see it inside one directivity bin (256^3 at 0.5 mm, 4 pairs:
    // 91 % of the (warp, source) pairs at 8 x 8 x 4 points, 89 % at 16 x 8 x 2, 80 % at 32 x 8 x 1).
    double best = 0.0;
    int64_t warps = 0;
    for (int b0 = 0; b0 <= 5; ++b0) {
        for (int b1 = 0; b0 + b1 <= 5; ++b1) {
            const int b2 = 5 - b0 - b1, e1 = b1 + pair_bits;
            const int64_t tiles0 = (g.count[0] + (1LL << b0) - 1) >> b0;
            const int64_t tiles1 = (g.count[1] + (1LL << e1) - 1) >> e1;
            const int64_t w = tiles0 * tiles1 * ((g.count[2] + (1LL << b2) - 1) >> b2);
            const double score = static_cast<double>(w) *
                                 (1.0 + 0.005 * static_cast<double>((1 << b0) + (1 << e1) + (1 << b2)));
            if (best > 0.0 && score >= best) continue;
            best = score;
            t.map = RowsMap{{b0, b1, b2}, tiles0, tiles1};
            warps = w;
        }
    }
    t.blocks = (warps + kThreads / 32 - 1) / (kThreads / 32);
    const int64_t per_warp = 64LL * pairs;
    t.use = static_cast<double>((m + per_warp - 1) / per_warp) >=
            (st != SRC_T4010A1 ? kRowsBusySphere : (pairs == 2 ? kRowsBusyTwo : kRowsBusy)) *
                static_cast<double>(warps);
    return t;
}

int num_sms() {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return kFallbackSms;
    if (dev < kSmCacheDevices) {
        v = g_num_sms[dev].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
        return kFallbackSms;
    if (dev < kSmCacheDevices) g_num_sms[dev].store(v, std::memory_order_relaxed);
    return v;
}

cudaError_t launch_pack_sources(int st, const float* raw, const float* k, const float* atten,
                                int64_t n, PackedSource* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    const int64_t blocks = (n + threads - 1) / threads;
    pack_sources_kernel<<<static_cast<unsigned>(blocks), threads, 0, s>>>(st, raw, k, atten, n, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_field(int st, int field, int sum_mode, const PackedSource* src, int64_t n,
                         const PointSet& ps, void* out, cudaStream_t s, bool scratch_ok) {
    if (ps.m <= 0) return cudaSuccess;
    if (field < FIELD_PRESSURE || field > FIELD_COMPLEX) return cudaErrorInvalidValue;
    if (st == SRC_T4010A1) return launch_st<SRC_T4010A1>(sum_mode, src, n, ps, field, out, s, scratch_ok);
    if (st == SRC_SPHERE) return launch_st<SRC_SPHERE>(sum_mode, src, n, ps, field, out, s, scratch_ok);
    return cudaErrorInvalidValue;
}

}  // namespace afc

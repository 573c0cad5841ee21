// How the GS-PAT cluster iteration's rows are shared over its blocks (host and device).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define AFC_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AFC_HOST_DEVICE inline
#endif

namespace afc {

constexpr int kIterCluster = 8;  // blocks of the cluster

// The first of the m rows of block `rank` (rank == kIterCluster: m, rounded up to even).  Rows are stored in
// pairs, so pairs are shared, as evenly as they go: no block is left without rows from
// 2 * kIterCluster - 1 foci on.  A block without rows would not arm its barriers' next phases, and the
// other blocks' stores would count on the first phase for the whole iteration.
AFC_HOST_DEVICE int64_t iter_first(int64_t m, int64_t rank) {
    return (m + 1) / 2 * rank / kIterCluster * 2;
}

// Rows of the largest share.
AFC_HOST_DEVICE int64_t iter_share(int64_t m) {
    return (m + 2 * kIterCluster - 1) / (2 * kIterCluster) * 2;
}

}  // namespace afc

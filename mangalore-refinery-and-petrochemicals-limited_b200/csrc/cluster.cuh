// Thread-block clusters as one small machine: every CTA owns a contiguous range of 32-row
// slices of each orientation, and keeps a full copy of the gathered vectors in its shared
// memory.  The owner of an element stores it into every CTA's copy (distributed shared
// memory), and a cluster barrier ends each phase -- a fraction of a microsecond, where a
// kernel boundary with its first loads from L2 costs three or four.
#pragma once

#include <cooperative_groups.h>

#include <cstdint>

namespace b2p {

constexpr int kClusterCtas = 8;      // the portable cluster size
constexpr int kClusterThreads = 512;

// first slice of CTA `rank` of NC
template <int NC>
__host__ __device__ __forceinline__ int cluster_slice(int slices, int rank) {
    return (int)((long long)slices * rank / NC);
}

// End of a phase: every CTA's stores into the copies are visible to all.
template <int NC>
__device__ __forceinline__ void cluster_phase(cooperative_groups::cluster_group& cl) {
    if constexpr (NC == 1) __syncthreads();
    else cl.sync();
}

// Writes v to element i of the copy of a vector in every CTA of the cluster; `copies` holds the
// CTAs' base addresses of it.
template <typename T, int NC>
struct ClusterVec {
    T* copy[NC];
    __device__ __forceinline__ ClusterVec(cooperative_groups::cluster_group& cl, T* mine) {
#pragma unroll
        for (int r = 0; r < NC; ++r) copy[r] = NC == 1 ? mine : cl.map_shared_rank(mine, r);
    }
    __device__ __forceinline__ void store(int i, T v) const {
#pragma unroll
        for (int r = 0; r < NC; ++r) copy[r][i] = v;
    }
};

}  // namespace b2p

// Thread-block clusters as one small machine: every CTA owns 32-row slices of each orientation
// and keeps a full copy of the gathered vectors in its shared memory.  The owner of an element
// stores it into every CTA's copy (distributed shared memory).  A phase ends with a cluster
// barrier (ClusterVec, cluster_phase: about 1 us with the stores before it) or, in the loops that
// run by the thousand, when the CTA's own copy is complete (ClusterPost: half of that) -- where
// a kernel boundary with its first loads from L2 costs three or four.
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

// Phases without a barrier: every CTA has one mbarrier per exchanged vector, and an element's
// owner posts it into every CTA's copy with st.async, which counts its bytes on that CTA's
// mbarrier.  A CTA goes on when its own copy is complete.  Safe with two vectors that are
// gathered in turn: a CTA posts elements of one only after its copy of the other is complete,
// that is, after every CTA has finished its reads of the first.  No thread may fall two phases
// of a vector behind (parities repeat): the CTA meets once per turn, and every CTA must own
// elements, so that none is passed by.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void tx_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Opens the next phase of this CTA's mbarrier: it completes when `bytes` have arrived.
__device__ __forceinline__ void tx_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// How long a wait for the peers' elements may take: thousands of times what they ever need, and within
// what a caller can wait for an error.
constexpr unsigned long long kTxWaitNs = 1000000000ull;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Waits for the phase of the given parity, kTxWaitNs at most; false: it did not complete.  The limit is
// one of time, because a single try_wait may suspend the thread for as long as the hardware likes.
__device__ __forceinline__ bool tx_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_addr(bar);
    unsigned long long since = 0;
    for (int spin = 0; spin < (1 << 24); ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if (spin > 256) {
            const unsigned long long now = global_ns();
            if (since == 0) since = now;
            if (now - since > kTxWaitNs) return false;
            __nanosleep(128);
        }
    }
    return false;
}
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_int(v)), "r"(bar)
                 : "memory");
}
// The CTAs' shared memory: where an address of this CTA's lies in CTA r's.
template <int NC>
struct ClusterPeers {
    uint32_t origin, base[NC];
    __device__ __forceinline__ explicit ClusterPeers(const void* any) : origin(smem_addr(any)) {
#pragma unroll
        for (int r = 0; r < NC; ++r) base[r] = NC == 1 ? origin : peer_addr(origin, r);
    }
};
// Element i of a vector into every CTA's copy (NC = 1: this CTA's, ordered by its own barrier).
// One base address a peer serves all vectors: two a vector and peer spilled.
template <typename T, int NC>
struct ClusterPost {
    uint32_t vec, bar;  // from the peers' origin
    T* mine;
    __device__ __forceinline__ ClusterPost(const ClusterPeers<NC>& to, T* v, uint64_t* b)
        : vec(smem_addr(v) - to.origin), bar(smem_addr(b) - to.origin), mine(v) {}
    __device__ __forceinline__ void store(const ClusterPeers<NC>& to, int i, T v) const {
        if constexpr (NC == 1) {
            mine[i] = v;
        } else {
            const uint32_t at = vec + i * (uint32_t)sizeof(T);
#pragma unroll
            for (int r = 0; r < NC; ++r) st_async(to.base[r] + at, v, to.base[r] + bar);
        }
    }
};

// Launch of one block shape on clusters of `ctas` CTAs (dims must outlive the configuration).
inline cudaLaunchConfig_t cluster_config(int grid, int ctas, int threads, size_t smem, cudaStream_t s,
                                         cudaLaunchAttribute* dims) {
    cudaLaunchConfig_t lc{};
    dims->id = cudaLaunchAttributeClusterDimension;
    dims->val.clusterDim.x = ctas;
    dims->val.clusterDim.y = dims->val.clusterDim.z = 1;
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    lc.attrs = dims;
    lc.numAttrs = 1;
    return lc;
}
// Clusters of a launch that the device can hold at once.  0 where its SMs cannot be brought together for
// one (a partition of a GPU): such a device keeps the forms without clusters.
template <typename F>
int clusters_resident(F* fn, int ctas, int threads, size_t smem) {
    cudaLaunchAttribute dims;
    const cudaLaunchConfig_t lc = cluster_config(ctas, ctas, threads, smem, nullptr, &dims);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &lc) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace b2p

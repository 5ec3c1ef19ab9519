// Launches of one thread-block cluster per world, and what their kernels share.
#pragma once

#include "prims.cuh"

namespace avbdg {

constexpr int kMaxTeam = 16; // CTAs a cluster (above 8 the kernel must allow it, and the device have room)

// This CTA's place in its cluster, and the cluster's CTAs.
__device__ __forceinline__ int clusterRank() {
    int r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ int clusterSize() {
    int s;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(s));
    return s;
}

// Cluster barrier: writes before it, to global memory and to any CTA's shared memory, are visible to the
// cluster's threads after it.
__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void clusterSync(int size) {
    if (size == 1) {
        __syncthreads();
    } else {
        clusterArrive();
        clusterWait();
    }
}

// Shared-memory addresses, of this CTA or (mapped) of another of the cluster. Another CTA's memory may be
// touched once that CTA is known to run (a cluster barrier after the kernel's start) and until it may end (a
// cluster barrier before the kernel's end, or after the last access).
__device__ __forceinline__ unsigned sharedAddress(const void *p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ unsigned mapShared(unsigned a, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void storeClusterInt(unsigned a, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Cluster and (programmatic) stream attributes of a launch.
struct TeamLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2]{};
    TeamLaunch(int team, int worlds, int threads, size_t smem, cudaStream_t s) {
        cfg.gridDim = dim3(static_cast<unsigned>(team) * static_cast<unsigned>(worlds));
        cfg.blockDim = dim3(static_cast<unsigned>(threads));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(team);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = pdlEnabled() ? 1 : 0;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
    }
};

// Allows `kernel` clusters of up to kMaxTeam CTAs with `smem` dynamic shared bytes on the current device; the
// largest cluster (a power of two) the device can hold.
inline int allowTeam(const void *kernel, int threads, size_t smem) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int team = kMaxTeam; team > 1; team >>= 1) {
        TeamLaunch l(team, 1, threads, smem, nullptr);
        l.cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &l.cfg) == cudaSuccess && n > 0)
            return team;
        cudaGetLastError();
    }
    return 1;
}

// Sum of `v` over the block, to every thread. `warpSums`: a word per warp.
__device__ __forceinline__ int blockSum(int v, int *warpSums) {
    const int sum = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        warpSums[threadIdx.x >> 5] = sum;
    __syncthreads();
    int all = 0;
    for (int k = 0; k < static_cast<int>(blockDim.x >> 5); k++)
        all += warpSums[k];
    return all;
}

// Exclusive prefix of one value a thread over the block; `total` is the block's sum.
__device__ __forceinline__ int blockPrefix(int v, int *warpSums, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int upTo = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upTo, o);
        if (lane >= o)
            upTo += y;
    }
    __syncthreads();
    if (lane == 31)
        warpSums[warp] = upTo;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int k = 0; k < static_cast<int>(blockDim.x >> 5); k++) {
        before += k < warp ? warpSums[k] : 0;
        total += warpSums[k];
    }
    return before + upTo - v;
}

// This CTA's share [lo, hi) of n items dealt in order, and the sum of counts over the items before it and
// over all: a scan over the cluster without a pass between its CTAs, each of which reads every count.
struct Share {
    int lo, hi, before, total;
};
__device__ __forceinline__ Share clusterShare(const int *counts, int n, int rank, int size, int *warpSums) {
    const int per = (n + size - 1) / size;
    Share s;
    s.lo = min(n, rank * per);
    s.hi = min(n, s.lo + per);
    int before = 0, all = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int c = counts[i];
        all += c;
        before += i < s.lo ? c : 0;
    }
    s.before = blockSum(before, warpSums);
    s.total = blockSum(all, warpSums);
    return s;
}

} // namespace avbdg

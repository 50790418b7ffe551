// Thread-block clusters: the meeting point, reads of a peer's shared memory, and the launch.
#pragma once

#include "common.cuh"

namespace ri {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the two halves of a meeting point, for one that nobody has to wait at: arrive early, wait late
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the float at the same place in the shared memory of the cluster's block `rank`
__device__ __forceinline__ float peer_float(const float* own, uint32_t rank) {
    uint32_t there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
    return v;
}
// ... and a store to it
__device__ __forceinline__ void store_peer_float(const float* own, uint32_t rank, float v) {
    uint32_t there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(there), "f"(v) : "memory");
}
// four of them (16-byte aligned)
__device__ __forceinline__ float4 peer_float4(const float* own, uint32_t rank) {
    uint32_t there;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(own)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(there) : "memory");
    return v;
}
// Sets an int of the shared memory, which lies at the same place in every block, in all of the cluster's `blocks`.  Other blocks
// must have set up theirs (a meeting point before) and look at it behind the next `cluster_sync`.
__device__ __forceinline__ void set_in_all(volatile int* own, int blocks) {
    for (int p = 0; p < blocks; ++p) {
        uint32_t there;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there)
                     : "r"((uint32_t)__cvta_generic_to_shared(const_cast<int*>(own))), "r"(p));
        asm volatile("st.shared::cluster.s32 [%0], 1;" ::"r"(there) : "memory");
    }
}

// How many blocks the device holds at once in clusters of `size` (2 to 8) when a block has an SM to itself: clusters lie within groups of
// SMs, whose numbers of SMs leave some over (148 SMs: less than 138 blocks in clusters of three, 144 in clusters of four).
// Asked once per device and size, with a kernel that may have the `smem` bytes, more than half of an SM's.
inline int blocks_alone(const void* kernel, int threads, size_t smem, int size) {
    static std::atomic<int> known[64][9];
    if (size <= 1) return sm_count();
    int dev = 0, n = 0;
    if (size > 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() - 20;
    n = known[dev][size].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)size);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = (sm_count() - 20) / size;
        }
        n *= size;
        known[dev][size].store(n, std::memory_order_relaxed);
    }
    return n;
}

// A launch that may start under the kernel before it (`launch_dependent`), its blocks in clusters of `cluster` along x.
template <typename... KArgs, typename... Args>
int launch_cluster(const char* what, void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t stream,
                   Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return check_launch(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...), what);
}

}  // namespace ri

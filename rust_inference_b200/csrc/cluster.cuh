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

// PTX of kernels whose CTAs work together in a cluster: ranks, barriers and loads from one another's shared memory.  No copy is multicast.
#pragma once
#include "tc_ptx.cuh"

namespace mx {
namespace tc {

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the shared::cluster address of the location `local` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
    return v;
}

// A split product whose slices are the CTAs of one cluster: four neighbouring results of the partial ones that lie at the same place `at` of each
// CTA's shared memory, added in slice order.
constexpr int CLUSTER_MOST = 8;  // portable cluster size
__device__ __forceinline__ float4 sum_slices(uint32_t at, int slices) {
    float4 v[CLUSTER_MOST];
#pragma unroll
    for (int i = 0; i < CLUSTER_MOST; i++)
        if (i < slices) v[i] = ld_cluster_f4(map_to_cta(at, i));
    float4 sum = v[0];
#pragma unroll
    for (int i = 1; i < CLUSTER_MOST; i++)
        if (i < slices) sum = make_float4(sum.x + v[i].x, sum.y + v[i].y, sum.z + v[i].z, sum.w + v[i].w);
    return sum;
}

// A launch on the calling thread's stream, its CTAs in clusters of `cluster` (0: none).
template <class... P, class... A>
inline void launch_clusters(void (*kernel)(P...), int grid, int threads, size_t shared, int cluster, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = ctx().stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_kernel
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
// Clusters of n CTAs of `kernel` that can be resident at once; 0: cannot be asked.
int resident_clusters(const void* kernel, int threads, size_t shared, int n);
// The number of slices (CTAs of a cluster) for a product of `tiles` output tiles and `num_kb` k-blocks whose cost comes out below `below`, and the
// cost in it; 0: none does.  resident(n): the clusters of n that fit the device.
template <class Resident>
int cluster_slices(uint64_t tiles, uint64_t num_kb, int sms, double kb_cost, double fixed, double& below, Resident resident) {
    int best = 0;
    for (int n = 2; n <= CLUSTER_MOST && 2 * (uint64_t)n <= num_kb && tiles * n <= (uint64_t)sms; n++) {
        const uint64_t per = (num_kb + n - 1) / n;
        if ((num_kb + per - 1) / per != (uint64_t)n) continue;  // the last slices would be empty
        const double cost = (double)per * kb_cost + fixed;
        if (cost >= below || tiles > (uint64_t)resident(n)) continue;
        below = cost;
        best = n;
    }
    return best;
}

}  // namespace tc
}  // namespace mx

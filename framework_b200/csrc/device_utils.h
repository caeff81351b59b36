// Device helpers shared by the streaming kernels: asynchronous copies to shared memory and thread-block clusters.
#pragma once

#include <cuda_runtime.h>

namespace mni {

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid) {
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    const int bytes = valid ? 16 : 0;                       // 0: nothing is read, the slot is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}
// ... of which only the first `bytes` are read, the rest of the slot is zero-filled.
__device__ __forceinline__ void cp_async16_part(void *smem, const void *gmem, int bytes) {
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Thread-block-cluster helpers for the ring kernel's finish: the K splits of a strip form one cluster, every
// CTA leaves its block sums in its own shared memory and the sums are added straight from there.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(const void *own_smem, unsigned rank) {
    const unsigned local = static_cast<unsigned>(__cvta_generic_to_shared(own_smem));
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

constexpr int kMaxClusterRanks = 8;
// Sum over the cluster's ranks, in ascending order, of the vector at the same place of each one's shared memory.  All
// loads are issued before the first is used: one after the other they cost 0.25 us each.
__device__ __forceinline__ float4 cluster_sum_f4(const void *own_smem, int ranks) {
    float4 p[kMaxClusterRanks];
#pragma unroll
    for (int r = 0; r < kMaxClusterRanks; ++r) p[r] = ld_cluster_f4(own_smem, static_cast<unsigned>(r < ranks ? r : 0));
    float4 sum = p[0];
#pragma unroll
    for (int r = 1; r < kMaxClusterRanks; ++r)
        if (r < ranks) { sum.x += p[r].x; sum.y += p[r].y; sum.z += p[r].z; sum.w += p[r].w; }
    return sum;
}

}  // namespace mni

// Thread-block clusters whose CTAs exchange data through each other's shared
// memory: stores counted on the receiver's mbarrier, a bounded wait for them,
// and the launch.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace bem {

constexpr int MAX_CLUSTER = 16;

// 16 bytes into another CTA's shared memory, counted on a barrier there.
__device__ __forceinline__ uint32_t peer_addr(uint32_t saddr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async16(uint32_t dst, uint32_t bar, uint4 v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint4 as_uint4(double2 v) {
    return make_uint4((unsigned)__double2loint(v.x), (unsigned)__double2hiint(v.x), (unsigned)__double2loint(v.y),
                      (unsigned)__double2hiint(v.y));
}
// Bounded wait for data written by other CTAs of the cluster: false when it ran out.
__device__ __forceinline__ bool peers_arrived(uint64_t* bar, uint32_t phase) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(phase)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The largest cluster the device schedules with a kernel's shared memory.
inline int max_cluster(const void* kernel, int threads, size_t smem) {
    for (int cs = MAX_CLUSTER; cs > 1; cs /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)cs);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {(unsigned)cs, 1, 1};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int num = 0;
        if (cudaOccupancyMaxActiveClusters(&num, kernel, &cfg) == cudaSuccess && num >= 1) return cs;
        cudaGetLastError();
    }
    return 1;
}

template <class... K, class... Args>
void launch_cluster(Context& ctx, void (*kernel)(K...), int grid, int cs, int threads, size_t smem, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)cs, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    BEM_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    BEM_CHECK_LAUNCH(&ctx);
}

}  // namespace bem

// cluster_caps.cuh - how many clusters of s CTAs of a kernel are resident at once, per device.
#pragma once
#include <mutex>

#include "pdk_common.cuh"

constexpr uint32_t kPdkMaxCluster = 8;   // portable cluster size

struct PdkClusterCaps {
    std::mutex mu;
    uint32_t cap[64][kPdkMaxCluster + 1];   // 0 = not asked for yet, or not possible
};

// On the first call for a device: raises the kernel's dynamic shared memory limit there and asks the driver (clusters stay
// within a GPC, so the counts are not SMs / s).  *caps is the current device's row; 0 or a cudaError_t.
static inline int pdk_cluster_caps(PdkClusterCaps& t, const void* kern, uint32_t threads, size_t smem, const uint32_t** caps) {
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(t.mu);
    uint32_t* c = t.cap[dev];
    if (c[1] == 0u) {
        if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); e != cudaSuccess)
            return (int)e;
        for (uint32_t s = kPdkMaxCluster; s >= 1u; --s) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr = {};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = s;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.gridDim = dim3(s);
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = smem;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) c[s] = (uint32_t)n;
        }
        (void)cudaGetLastError();
        if (c[1] == 0u) c[1] = (uint32_t)pdk_sm_count();
    }
    *caps = c;
    return 0;
}

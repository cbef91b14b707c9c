// Kernels that run as one thread-block cluster (vb_ref1d.cu, vb_tube.cu): where
// the CTAs meet, and how many a cluster may have.
#pragma once
#include <cuda_runtime.h>

namespace vb {

// Every thread of the cluster; what one stored before is visible to the others
// after. The lanes of a warp come from loops of their own lengths (con2prim's
// Newton), and the .aligned forms want the warp as one.
__device__ __forceinline__ void cluster_meet() {
    __threadfence();
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr int CLUSTER_MAX = 16;  // CTAs, where the GPU grants such a cluster of `kern`; else 8 (portable)

// the larger of the two that the current device grants, remembered in widest[64] per
// device (one array per kernel; racing writers store the same value)
template <typename K> int widest_cluster(K kern, int threads, size_t smem, int* widest) {
    int dev = 0;
    cudaGetDevice(&dev);
    int& wide = widest[dev & 63];
    if (wide) return wide;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = CLUSTER_MAX;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(CLUSTER_MAX);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    int fit = 0;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) == cudaSuccess && fit > 0;
    if (!ok) cudaGetLastError();  // a refused cluster size is no error of the call
    return wide = ok ? CLUSTER_MAX : 8;
}

// one cluster of `ctas` CTAs
template <typename K, typename... A>
cudaError_t launch_cluster(K kern, int ctas, int threads, size_t smem, cudaStream_t s, const A&... a) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    return cudaLaunchKernelEx(&cfg, kern, a...);
}

}  // namespace vb

// Launcher of the cluster run kernel (resident_cluster.cuh).

#include <cuda_runtime.h>

#include <type_traits>

#include "resident_launch.h"

namespace flbp {

namespace {

template <typename T>
const void *cluster_fn(bool damp) {
    return damp ? (const void *)cluster_kernel<T, true> : (const void *)cluster_kernel<T, false>;
}

void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, unsigned size, unsigned clusters, int threads,
                    size_t smem, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(size * clusters);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

}  // namespace

template <typename T>
cudaError_t cluster_launch(bool damp, unsigned size, unsigned clusters, size_t smem, const ClusterArgs<T> &a,
                           cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(cfg, attr, size, clusters, kClusterThreads<T>, smem, st);
    ClusterArgs<T> args = a;
    void *params[] = {&args};
    return cudaLaunchKernelExC(&cfg, cluster_fn<T>(damp), params);
}

template <typename T>
int cluster_max_active(bool damp, unsigned size, size_t smem) {
    const void *fn = cluster_fn<T>(damp);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmemMax) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(cfg, attr, size, 1, kClusterThreads<T>, smem, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template cudaError_t cluster_launch<float>(bool, unsigned, unsigned, size_t, const ClusterArgs<float> &, cudaStream_t);
template cudaError_t cluster_launch<double>(bool, unsigned, unsigned, size_t, const ClusterArgs<double> &,
                                            cudaStream_t);
template int cluster_max_active<float>(bool, unsigned, size_t);
template int cluster_max_active<double>(bool, unsigned, size_t);

}  // namespace flbp

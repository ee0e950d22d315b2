// Launcher of the resident run kernel (resident.cuh).

#include <cuda_runtime.h>

#include "resident_launch.h"

namespace flbp {

template <typename T>
static const void *kernel_of(bool damp, bool cache) {
    if (damp) return cache ? (const void *)resident_kernel<T, true, true> : (const void *)resident_kernel<T, true, false>;
    return cache ? (const void *)resident_kernel<T, false, true> : (const void *)resident_kernel<T, false, false>;
}

template <typename T>
cudaError_t resident_launch(bool damp, bool cache, unsigned grid, size_t smem, const ResArgs<T> &a,
                            cudaStream_t st) {
    ResArgs<T> args = a;
    void *params[] = {&args};
    return cudaLaunchCooperativeKernel(kernel_of<T>(damp, cache), dim3(grid), dim3(kResThreads), params, smem, st);
}

template <typename T>
int resident_blocks_per_sm(bool damp, bool cache, size_t smem) {
    const void *fn = kernel_of<T>(damp, cache);
    int n = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kResThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template cudaError_t resident_launch<float>(bool, bool, unsigned, size_t, const ResArgs<float> &, cudaStream_t);
template cudaError_t resident_launch<double>(bool, bool, unsigned, size_t, const ResArgs<double> &,
                                             cudaStream_t);
template int resident_blocks_per_sm<float>(bool, bool, size_t);
template int resident_blocks_per_sm<double>(bool, bool, size_t);

}  // namespace flbp

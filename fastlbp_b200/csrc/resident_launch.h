// Host launchers of the resident run kernel (resident.cu) and of the cluster
// run kernel (resident_cluster.cu).
#pragma once

#include <cuda_runtime.h>

#include "resident.cuh"
#include "resident_cluster.cuh"

namespace flbp {

constexpr size_t kResSmemMax = 214 * 1024;  // cached constants of a block at most (static shared memory beside them)

// One cooperative launch of `grid` blocks with `smem` bytes of cached constants (cache).
template <typename T>
cudaError_t resident_launch(bool damp, bool cache, unsigned grid, size_t smem, const ResArgs<T> &a,
                            cudaStream_t st);

// Resident blocks per SM with `smem` bytes of dynamic shared memory; 0 when
// the kernel cannot run so.
template <typename T>
int resident_blocks_per_sm(bool damp, bool cache, size_t smem);

constexpr size_t kClusterSmemMax = 225 * 1024;  // dynamic shared memory of a cluster kernel's block at most

// One launch of `clusters` clusters of `size` blocks.
template <typename T>
cudaError_t cluster_launch(bool damp, unsigned size, unsigned clusters, size_t smem, const ClusterArgs<T> &a,
                           cudaStream_t st);

// Clusters of `size` blocks that run at once; 0 when the kernel cannot run so.
template <typename T>
int cluster_max_active(bool damp, unsigned size, size_t smem);

}  // namespace flbp

// Host-only helpers (no device code: this header is also compiled by the host compiler alone).
#pragma once

#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

#include "../../include/gsq.h"

namespace gsq {

// thread-local record of the last failing CUDA call (read through gsq_last_cuda_error)
int record_cuda_error(cudaError_t e);
#define GSQ_CUDA_TRY(expr)                                   \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) return gsq::record_cuda_error(_e); \
  } while (0)

// Co-resident clusters of `cs` CTAs with `smem` bytes each, kept per kernel, device and cluster size (`smem` is the device's
// most): the number plus one, 0 where it was not asked for yet. Several threads may ask at the same time: each finds the same.
struct ClusterCount {
  std::atomic<int> n[32][4];
};
inline int max_clusters(ClusterCount& o, const void* kern, int cs, int threads, size_t smem, int sm_count, int* out) {
  int dev = 0;
  GSQ_CUDA_TRY(cudaGetDevice(&dev));
  std::atomic<int>* const kept = dev < 32 ? &o.n[dev][cs == 1 ? 0 : cs == 2 ? 1 : cs == 4 ? 2 : 3] : nullptr;
  if (kept && *kept) {
    *out = *kept - 1;
    return GSQ_OK;
  }
  GSQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  GSQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 0));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sm_count / cs * cs));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cs;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cs == 1) {
    n = sm_count;
  } else if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  n = n < sm_count / cs ? n : sm_count / cs;
  if (kept) *kept = n + 1;
  *out = n;
  return GSQ_OK;
}

}  // namespace gsq

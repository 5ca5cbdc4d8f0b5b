// mmv_pair_kernel (gsq_mmv.cuh) for the pairs of types that fused layers have (mmv_pair_types). Activations: X itself, quantised while it is staged.
#include "gsq_mmv.cuh"

namespace gsq {
int mmv_launch_pair_xq81(int ta, int tb, const MmvArgs& a, const MmvArgs& b, int sm_count, int max_smem, cudaStream_t st) {
  return mmv_launch_pair_of<XL_XQ81>(ta, tb, a, b, sm_count, max_smem, st);
}
}  // namespace gsq

// mmv_pair_kernel (gsq_mmv.cuh) for the pairs of types that fused layers have: a main type and the one that a file keeps some
// shards at. Activations: X itself, quantised while it is staged.
#include "gsq_mmv.cuh"

namespace gsq {
int mmv_launch_pair_xq81(int ta, int tb, const MmvArgs& a, const MmvArgs& b, int sm_count, int max_smem, cudaStream_t st) {
  if (tb == GSQ_TYPE_Q6_K) {
    switch (ta) {
      case GSQ_TYPE_Q4_K: return mmv_launch_pair<MK_Q4K, MK_Q6K, XL_XQ81>(a, b, sm_count, max_smem, st);
      case GSQ_TYPE_IQ3_S: return mmv_launch_pair<MK_IQ3S, MK_Q6K, XL_XQ81>(a, b, sm_count, max_smem, st);
      case GSQ_TYPE_IQ4_XS: return mmv_launch_pair<MK_IQ4XS, MK_Q6K, XL_XQ81>(a, b, sm_count, max_smem, st);
      default: return MMV_DECLINED;
    }
  }
  if (ta == GSQ_TYPE_IQ3_S && tb == GSQ_TYPE_IQ4_XS) return mmv_launch_pair<MK_IQ3S, MK_IQ4XS, XL_XQ81>(a, b, sm_count, max_smem, st);
  return MMV_DECLINED;
}
}  // namespace gsq

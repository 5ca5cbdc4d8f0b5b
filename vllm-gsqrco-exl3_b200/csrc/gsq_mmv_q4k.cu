// gsq_mmv.cuh for one weight type (a translation unit each, so that they compile in parallel)
#include "gsq_mmv.cuh"

namespace gsq {
int mmv_launch_q4k(const MmvArgs& a, int x_layout, int sm_count, int max_smem, cudaStream_t st) {
  return mmv_launch_kind<MK_Q4K>(a, x_layout, sm_count, max_smem, st);
}
int mmv_errors_q4k(int* peer, int* copy) { return mmv_errors(peer, copy); }
}  // namespace gsq

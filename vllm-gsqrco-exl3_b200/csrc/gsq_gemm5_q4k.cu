// gsq_gemm5.cuh for one weight type (a translation unit each, so that they compile in parallel)
#include "gsq_gemm5.cuh"

namespace gsq {
namespace g5 {
int launch_q4k(const Args& g, int n_cta, cudaStream_t st) { return launch_kind<G5_Q4K>(g, n_cta, st); }
int error_flag_q4k(int* flag) { return error_flag(flag); }
}  // namespace g5
}  // namespace gsq

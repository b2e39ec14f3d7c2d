// Q4_K instantiations of the tensor-core matmul for matrices with rows whose blocks differ widely.
#include "qk_gemm_tc.cuh"

cudaError_t qktc::launch_wide_q4k(const TcPlan &P, const TcArgs &A, __half *x16, const QkTcCall &c, bool beside, cudaStream_t s) {
  return launch_matmul<QK_T_Q4_K | QK_TC_WIDE>(P, A, x16, c, beside, s);
}

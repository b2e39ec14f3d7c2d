// Q4_0 instantiations of the tensor-core matmul.
#include "qk_gemm_tc.cuh"

QK_TC_DEFINE(q40, QK_T_Q4_0)

// Q6_K instantiations of the tensor-core matmul.
#include "qk_gemm_tc.cuh"

QK_TC_DEFINE(q6k, QK_T_Q6_K)

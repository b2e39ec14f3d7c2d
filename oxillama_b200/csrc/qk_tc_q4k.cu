// Q4_K instantiations of the tensor-core matmul.
#include "qk_gemm_tc.cuh"

QK_TC_DEFINE(q4k, QK_T_Q4_K)

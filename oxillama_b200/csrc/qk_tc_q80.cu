// Q8_0 instantiations of the tensor-core matmul.
#include "qk_gemm_tc.cuh"

QK_TC_DEFINE(q80, QK_T_Q8_0)

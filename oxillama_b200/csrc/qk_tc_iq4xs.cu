// IQ4_XS instantiations of the tensor-core matmul.
#include "qk_gemm_tc.cuh"

QK_TC_DEFINE(iq4xs, QK_T_IQ4_XS)

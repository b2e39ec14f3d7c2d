// Mixture-of-experts decode kernels of one format (policy qkdec::DecQ80).
#include "qk_dec_fmts.cuh"
#include "qk_gemv_moe.cuh"

QK_MOE_DEC_DEFINE(q80, qkdec::DecQ80, qkdec::DecQ80)

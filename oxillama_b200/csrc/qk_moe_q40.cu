// Mixture-of-experts decode kernels of one format (policy qkdec::DecQ40).
#include "qk_dec_fmts.cuh"
#include "qk_gemv_moe.cuh"

QK_MOE_DEC_DEFINE(q40, qkdec::DecQ40, qkdec::DecQ40)

// Mixture-of-experts decode kernels of one format (policy qkdec::DecQ6K).
#include "qk_dec_fmts.cuh"
#include "qk_gemv_moe.cuh"

QK_MOE_DEC_DEFINE(q6k, qkdec::DecQ6K, qkdec::DecQ6KOne)

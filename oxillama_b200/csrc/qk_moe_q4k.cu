// Mixture-of-experts decode kernels of one format (policy qkdec::DecQ4K).
#include "qk_dec_q4k.cuh"
#include "qk_gemv_moe.cuh"

QK_MOE_DEC_DEFINE(q4k, qkdec::DecQ4K, qkdec::DecQ4KOne)

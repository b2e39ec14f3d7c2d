// Mixture-of-experts decode kernels of one format (policy qkdec::DecIQ4XS).
#include "qk_dec_fmts.cuh"
#include "qk_gemv_moe.cuh"

QK_MOE_DEC_DEFINE(iq4xs, qkdec::DecIQ4XS, qkdec::DecIQ4XS)

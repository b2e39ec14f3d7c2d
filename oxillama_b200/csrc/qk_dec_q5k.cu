// Instantiates the decode kernels of one format (policy qkdec::DecQ5K, qk_dec_kq.cuh).
#include "qk_dec_kq.cuh"

QK_DEC_DEFINE(q5k, qkdec::DecQ5K)

// Instantiates the decode kernels of one format (policy qkdec::DecQ2K, qk_dec_kq.cuh).
#include "qk_dec_kq.cuh"

QK_DEC_DEFINE(q2k, qkdec::DecQ2K)

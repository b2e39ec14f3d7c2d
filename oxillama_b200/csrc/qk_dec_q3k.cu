// Instantiates the decode kernels of one format (policy qkdec::DecQ3K, qk_dec_kq.cuh).
#include "qk_dec_kq.cuh"

QK_DEC_DEFINE(q3k, qkdec::DecQ3K)

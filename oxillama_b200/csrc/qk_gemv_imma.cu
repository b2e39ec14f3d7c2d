// Decode matvec (1..4 activation rows): the instantiations
// of the integer-MMA decode kernel (qk_gemv_skel.cuh) with the policies of qk_dec_fmts.cuh and qk_dec_kq.cuh
// live in qk_dec_<format>.cu; this is the per-type dispatch of the decode path.
#include "qk_kernels.h"

// per-format entry points (qk_dec_<format>.cu)
#define QK_DEC_DECLARE(NAME)                                                                                    \
  bool qk_dec_##NAME##_supported(const QkLayout &L, uint32_t m);                                                \
  size_t qk_dec_##NAME##_scratch(const QkLayout &L, uint32_t m);                                                \
  cudaError_t qk_dec_##NAME##_launch(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,         \
                                     uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,        \
                                     int sm_count, cudaStream_t s, const QkPeers *peers, const uint8_t *tiled2, bool host_x);
QK_DEC_DECLARE(q80)
QK_DEC_DECLARE(q40)
QK_DEC_DECLARE(iq4xs)
QK_DEC_DECLARE(q6k)
QK_DEC_DECLARE(q5k)
QK_DEC_DECLARE(q3k)
QK_DEC_DECLARE(q2k)

#define QK_BY_TYPE(L, call_q4k, call)            \
  switch ((L).type) {                            \
    case QK_T_Q4_K:                              \
      return call_q4k;                           \
    case QK_T_Q8_0:                              \
      return call(q80);                          \
    case QK_T_Q4_0:                              \
      return call(q40);                          \
    case QK_T_IQ4_XS:                            \
      return call(iq4xs);                        \
    case QK_T_Q6_K:                              \
      return call(q6k);                          \
    case QK_T_Q5_K:                              \
      return call(q5k);                          \
    case QK_T_Q3_K:                              \
      return call(q3k);                          \
    case QK_T_Q2_K:                              \
      return call(q2k);                          \
    default:                                     \
      break;                                     \
  }

bool qk_gemv_fast_supported(const QkLayout &L, uint32_t m) {
  if (m < 1 || m > QK_GEMV_MAX_M) return false;
#define CALL(F) qk_dec_##F##_supported(L, m)
  QK_BY_TYPE(L, qk_gemv_mma_supported(L, m), CALL)
#undef CALL
  return false;
}

size_t qk_gemv_fast_scratch_bytes(const QkLayout &L, uint32_t m) {
#define CALL(F) qk_dec_##F##_scratch(L, m)
  QK_BY_TYPE(L, qk_gemv_mma_scratch_bytes(L, m), CALL)
#undef CALL
  return 0;
}

cudaError_t qk_launch_gemv_fast(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,
                                uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,
                                int sm_count, cudaStream_t s, bool host_x) {
#define CALL(F) qk_dec_##F##_launch(L, tiled, x, y, m, ldy, status, scratch, sm_count, s, nullptr, nullptr, host_x)
  QK_BY_TYPE(L, qk_launch_gemv_mma(L, tiled, x, y, m, ldy, status, scratch, sm_count, s, nullptr, nullptr, host_x), CALL)
#undef CALL
  return cudaErrorNotSupported;
}

// ---- the same kernels with the output fan-out of a row-sharded layer built in
bool qk_gemv_peer_supported(const QkLayout &L, uint32_t m) {
  return L.type != QK_T_Q5_K && L.type != QK_T_Q3_K && L.type != QK_T_Q2_K && qk_gemv_fast_supported(L, m);
}

size_t qk_gemv_peer_scratch_bytes(const QkLayout &L, uint32_t m) { return qk_gemv_fast_scratch_bytes(L, m); }

cudaError_t qk_launch_gemv_peer(const QkLayout &L, const uint8_t *tiled, const float *x, uint32_t m,
                                uint64_t ldy, unsigned *status, unsigned char *scratch, int sm_count,
                                cudaStream_t s, const QkPeers *peers) {
#define CALL(F) qk_dec_##F##_launch(L, tiled, x, nullptr, m, ldy, status, scratch, sm_count, s, peers, nullptr, false)
  QK_BY_TYPE(L, qk_launch_gemv_mma(L, tiled, x, nullptr, m, ldy, status, scratch, sm_count, s, peers), CALL)
#undef CALL
  return cudaErrorNotSupported;
}

// ---- gate and up projection of a feed-forward block in one launch:
// h[i][j] = silu(gate_j . x_i) * (up_j . x_i)
bool qk_gemv_dual_supported(const QkLayout &L, uint32_t m) { return L.type != QK_T_Q6_K && qk_gemv_fast_supported(L, m); }

cudaError_t qk_launch_gemv_dual(const QkLayout &L, const uint8_t *gate_tiled, const uint8_t *up_tiled, const float *x,
                                float *h, uint32_t m, uint64_t ldh, unsigned *status, unsigned char *scratch,
                                int sm_count, cudaStream_t s) {
#define CALL(F) qk_dec_##F##_launch(L, gate_tiled, x, h, m, ldh, status, scratch, sm_count, s, nullptr, up_tiled, false)
  QK_BY_TYPE(L, qk_launch_gemv_mma(L, gate_tiled, x, h, m, ldh, status, scratch, sm_count, s, nullptr, up_tiled), CALL)
#undef CALL
  return cudaErrorNotSupported;
}

// ---- mixture-of-experts projections of a handful of tokens (qk_gemv_moe.cuh)
#define QK_MOE_DEC_DECLARE(NAME)                                                                                         \
  uint32_t qk_moe_dec_##NAME##_rows(const QkLayout &L);                                                                  \
  size_t qk_moe_dec_##NAME##_image(const QkLayout &L);                                                                   \
  cudaError_t qk_moe_dec_##NAME##_split(const QkLayout &L, const float *x, uint32_t rows, unsigned char *img, \
                                        const qkmoe::PlanArgs *plan, cudaStream_t s); \
  cudaError_t qk_moe_dec_##NAME##_launch(const QkLayout &L, const uint8_t *const *w, const uint8_t *const *w2, uint32_t n, \
                                         uint32_t rows_per_job, const QkMoeJobs *jobs, const unsigned char *img,         \
                                         uint32_t div, float *y, uint64_t ldy, unsigned *status, int sm_count, cudaStream_t s);
QK_MOE_DEC_DECLARE(q4k)
QK_MOE_DEC_DECLARE(q80)
QK_MOE_DEC_DECLARE(q40)
QK_MOE_DEC_DECLARE(iq4xs)
QK_MOE_DEC_DECLARE(q6k)
#define QK_MOE_BY_TYPE(L, SUFFIX, ARGS)              \
  switch ((L).type) {                                \
    case QK_T_Q4_K:                                  \
      return qk_moe_dec_q4k_##SUFFIX ARGS;           \
    case QK_T_Q8_0:                                  \
      return qk_moe_dec_q80_##SUFFIX ARGS;           \
    case QK_T_Q4_0:                                  \
      return qk_moe_dec_q40_##SUFFIX ARGS;           \
    case QK_T_IQ4_XS:                                \
      return qk_moe_dec_iq4xs_##SUFFIX ARGS;         \
    case QK_T_Q6_K:                                  \
      return qk_moe_dec_q6k_##SUFFIX ARGS;           \
    default:                                         \
      break;                                         \
  }

uint32_t qk_moe_dec_rows(const QkLayout &L) {
  QK_MOE_BY_TYPE(L, rows, (L))
  return 0;
}

size_t qk_moe_dec_image_bytes(const QkLayout &L) {
  QK_MOE_BY_TYPE(L, image, (L))
  return 0;
}

cudaError_t qk_launch_moe_dec_split(const QkLayout &L, const float *x, uint32_t rows, unsigned char *img,
                                    const qkmoe::PlanArgs *plan, cudaStream_t s) {
  QK_MOE_BY_TYPE(L, split, (L, x, rows, img, plan, s))
  return cudaErrorNotSupported;
}

cudaError_t qk_launch_moe_dec(const QkLayout &L, const uint8_t *const *w, const uint8_t *const *w2, uint32_t n,
                              uint32_t rows_per_job, const QkMoeJobs *jobs, const unsigned char *img, uint32_t div, float *y,
                              uint64_t ldy, unsigned *status, int sm_count, cudaStream_t s) {
  QK_MOE_BY_TYPE(L, launch, (L, w, w2, n, rows_per_job, jobs, img, div, y, ldy, status, sm_count, s))
  return cudaErrorNotSupported;
}

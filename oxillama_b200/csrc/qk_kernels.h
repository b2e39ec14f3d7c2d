// Internal launch interface between the C-ABI layer and the kernel translation units.
#pragma once
#include <cstdlib>

#include "qk_layout.cuh"

// Developer knobs (environment variables that change ring depths, warp counts and the like)
// exist only in builds made with -DQK_DEV_KNOBS; the default build never reads the
// environment, so nothing outside the caller's arguments changes what a call computes.
static inline const char *qk_knob(const char *name) {
#ifdef QK_DEV_KNOBS
  return getenv(name);
#else
  (void)name;
  return nullptr;
#endif
}

// A flag per CUDA device: function attributes (e.g. the dynamic shared-memory limit) and
// occupancy figures belong to a device, and one process may drive several.
struct QkPerDevice {
  bool done[64] = {};
  // true the first time it is asked on the current device
  bool first() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return true;
    if (done[d]) return false;
    done[d] = true;
    return true;
  }
  void reset() {  // the first-time work failed: try again on the next call
    int d = 0;
    if (cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < 64) done[d] = false;
  }
};

// Device status word bits (read back by qk_check_device_status).
#define QK_DEV_TIMEOUT 1u
#define QK_DEV_BOUNDS 2u

// raw_dev: GGUF-layout bytes of rows [0, L.rows) of the shard; tiled_dev: L.total_bytes, zeroed.
cudaError_t qk_launch_repack(const QkLayout &L, const uint8_t *raw_dev, uint8_t *tiled_dev,
                             cudaStream_t s);
cudaError_t qk_launch_dequant(const QkLayout &L, const uint8_t *tiled, float *out, cudaStream_t s);
// Generic any-shape path: f32 dequant in registers, f32 FMA, one warp per weight row.
cudaError_t qk_launch_gemm_simple(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,
                                  uint32_t m, uint64_t ldy, cudaStream_t s);
cudaError_t qk_launch_fused_simple(const QkLayout &L, const uint8_t *tiled, const uint8_t *acts,
                                   float *out, cudaStream_t s);
cudaError_t qk_launch_quantize_q8_0(const float *x, uint64_t n, uint8_t *out, cudaStream_t s);

// Output fan-out of a row-sharded matvec.  Every rank of the node owns a buffer of 8-byte
// slots, one per output element of the gathered [m x world * rows] result: the f32 value in
// the low half, the call's tag (its ordinal on that buffer, from 1) in the high half.  The
// kernel that computes a result stores the pair, as one 64-bit word, into the slot of every
// rank (plain peer stores over NVLink; entry `rank` is the local buffer).  A naturally
// aligned 64-bit store is single-copy atomic, so a reader that sees the tag it expects has
// the value that belongs to it: no fence, flag or counter stands between the data and its
// consumer, and nothing waits for a peer's acknowledgement.  n == 0: ordinary local output.
#define QK_MAX_PEERS 8
struct QkPeers {
  unsigned long long *slots[QK_MAX_PEERS];  // each rank's slot array, already offset to this rank's columns
  unsigned *counter;                        // local: CTAs of this launch counted in (returns to 0)
  unsigned *epoch;                          // local: calls issued so far on this buffer (the latest tag)
  uint32_t n, rank;
  // optional: the activations are the gathered output of an earlier sharded call and are
  // read straight from its slots, each read waiting (bounded) for the tag *wait_epoch
  const unsigned long long *wait_slots;     // slot of x[0][0]; row stride = wait_ld slots
  const unsigned *wait_epoch;
  uint64_t wait_ld;
  // optional: while its first weight tiles are on their way the kernel also unpacks the
  // latest call of another gather object (unpack_n slots, each waited for with a bound, tag
  // *unpack_epoch) into that object's plain buffer: the gather's completion costs no kernel
  // of its own and no gap between two matvecs
  const unsigned long long *unpack_slots;
  const unsigned *unpack_epoch;
  float *unpack_out;
  uint64_t unpack_n;
};

// Bandwidth-bound decode path (m <= QK_GEMV_MAX_M): bulk-copied tiles, integer dot.
#define QK_GEMV_MAX_M 4
// Up to this many activations (rows x padded columns) every CTA of the decode kernel splits them itself;
// above, a kernel of its own does it once into scratch -- if the call has any (scratch == null: in the CTAs).
#define QK_SPLIT_IN_CTA 8192u
bool qk_gemv_fast_supported(const QkLayout &L, uint32_t m);
// Q4_K decode path on the integer tensor-core MMA (m16n8k32 u8 x s8).  `scratch`
// is device memory of at least qk_gemv_mma_scratch_bytes(L, m) bytes, 16-byte
// aligned, that the call may overwrite (the split activations live there
// between its two kernels).
bool qk_gemv_mma_supported(const QkLayout &L, uint32_t m);
size_t qk_gemv_mma_scratch_bytes(const QkLayout &L, uint32_t m);
cudaError_t qk_launch_gemv_mma(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,
                               uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,
                               int sm_count, cudaStream_t s, const QkPeers *peers = nullptr,
                               const uint8_t *tiled2 = nullptr, bool host_x = false);
cudaError_t qk_launch_gemv_mma_split(const QkLayout &L, const uint8_t *tiled, const float *x,
                                     float *y, uint32_t m, uint64_t ldy, unsigned *status,
                                     unsigned char *scratch, int sm_count, cudaStream_t s);
// Decode kernels that can store their results into every rank's tagged slots themselves
// (and read gathered activations out of slots): `peers` as described at QkPeers.
bool qk_gemv_peer_supported(const QkLayout &L, uint32_t m);
size_t qk_gemv_peer_scratch_bytes(const QkLayout &L, uint32_t m);
cudaError_t qk_launch_gemv_peer(const QkLayout &L, const uint8_t *tiled, const float *x, uint32_t m,
                                uint64_t ldy, unsigned *status, unsigned char *scratch, int sm_count,
                                cudaStream_t s, const QkPeers *peers);
// Gate and up projection of a feed-forward block in one launch (two matrices of the same
// shape and format): h[i * ldh + j] = silu(gate_j . x_i) * (up_j . x_i).  Scratch as
// qk_gemv_fast_scratch_bytes.
bool qk_gemv_dual_supported(const QkLayout &L, uint32_t m);
cudaError_t qk_launch_gemv_dual(const QkLayout &L, const uint8_t *gate_tiled, const uint8_t *up_tiled, const float *x,
                                float *h, uint32_t m, uint64_t ldh, unsigned *status, unsigned char *scratch,
                                int sm_count, cudaStream_t s);
size_t qk_gemv_fast_scratch_bytes(const QkLayout &L, uint32_t m);
// host_x: x is mapped host memory; it is read once (split by a kernel of its own), not by every CTA.
cudaError_t qk_launch_gemv_fast(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,
                                uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,
                                int sm_count, cudaStream_t s, bool host_x = false);

// Mixture-of-experts projections of a handful of tokens on the decode kernels, all experts hit in one
// launch (qk_gemv_moe.cuh).  The job list is made on the device: one expert and one or two rows each.
#define QK_MOE_MAX 16       // most local experts
#define QK_MOE_DEC_TOKENS 16  // most tokens of such a call
#define QK_MOE_DEC_ROWS 4   // experts with more rows than this go to the tensor cores
#define QK_MOE_JOBS 32      // most jobs: a lane of the warp that deals them out holds one
struct QkMoeJobs {
  uint32_t n, pad[3];
  struct {
    uint32_t expert, rows, slot[2];  // slots = token * top_k + k
  } job[QK_MOE_JOBS];
};
// Most jobs that `slots` routed rows over n_local experts can make (QK_MOE_JOBS at most is served).
static inline size_t qk_moe_dec_jobs(size_t slots, size_t n_local, uint32_t rows_per_job) {
  const size_t all = n_local * ((QK_MOE_DEC_ROWS + rows_per_job - 1) / rows_per_job);
  return slots < all ? slots : all;
}
uint32_t qk_moe_dec_rows(const QkLayout &L);  // rows a job may have: 2, 1, or 0 where the format or shape is not served
size_t qk_moe_dec_image_bytes(const QkLayout &L);  // scratch per split activation row
// plan != null: the same launch also makes the plan (qk_moe_plan.cuh): ids / wts as qk_launch_moe_route,
// big[e] = rows of expert e where these exceed QK_MOE_DEC_ROWS, else 0, lists / pos as qk_launch_moe_lists.
namespace qkmoe { struct PlanArgs; }
cudaError_t qk_launch_moe_dec_split(const QkLayout &L, const float *x, uint32_t rows, unsigned char *img,
                                    const qkmoe::PlanArgs *plan, cudaStream_t s);
// y[slot][row] = w[expert] row . image(slot / div), or with w2 the silu(gate) * up of both.
cudaError_t qk_launch_moe_dec(const QkLayout &L, const uint8_t *const *w, const uint8_t *const *w2, uint32_t n,
                              uint32_t rows_per_job, const QkMoeJobs *jobs, const unsigned char *img, uint32_t div, float *y,
                              uint64_t ldy, unsigned *status, int sm_count, cudaStream_t s);

// Batched matmul on tcgen05 / TMEM (used for m > QK_GEMV_MAX_M).  One call multiplies `n` weight
// matrices of one shape and format, each by its own group of activation rows: n = 1 is the ordinary
// matmul; the projections of a feed-forward block or the experts of a mixture go together.
#define QK_MAX_GROUPS 16
struct QkTcCall {
  const QkLayout *L;                 // of every matrix
  const void *maps[QK_MAX_GROUPS];   // their tensor maps (qk_gemm_tc_map, 128 bytes each)
  const float *rows[QK_MAX_GROUPS];  // and the factors of their rows (qk_gemm_tc_factors)
  bool wide;                         // one of them is marked
  uint32_t n, n_act;                 // matrices; activation groups: matrix e multiplies group e % n_act
  // Activation row i of group e is x row e * xcap + i; with `lists` (device) it is x row
  // lists[e * list_stride + i] / list_div.  x2 != null: the row is silu(x) * x2 instead.
  const float *x, *x2;
  const int *lists;
  uint32_t list_stride, list_div;
  // m rows per group, or (counts != null, on the device) counts[e] of at most m; `expect`: the rows of an average group
  const int *counts;
  uint32_t m, expect, xcap, ycap;
  uint32_t live;                     // with counts: most rows that all groups have together
  float *y;                          // output row i of matrix e: y + (e * ycap + i) * ldy
  uint64_t ldy;
};
bool qk_gemm_tc_supported(const QkLayout &L, uint32_t m);
// The tensor map (128 bytes, 64-byte aligned) through which the kernel fetches a matrix: L.total_bytes and
// this many zeros behind them.
uint64_t qk_gemm_tc_pad_bytes(const QkLayout &L);
cudaError_t qk_gemm_tc_map(const QkLayout &L, uint8_t *tiled, void *map);
// A power of two per row (whole chunks of rows) over which the kernel expands its weights: bytes of the table, 0 where the
// format has none, and its computation from the tiled matrix.  *wide: the matrix has a row whose blocks differ so widely that
// its calls expand another way (the mark).  Waits for the stream.
size_t qk_gemm_tc_factor_bytes(const QkLayout &L);
cudaError_t qk_gemm_tc_factors(const QkLayout &L, const uint8_t *tiled, float *rows, bool *wide, cudaStream_t s);
// Scratch of a call: the fp16 activations (rows in sixteens), their scales and, at their most for every call, the
// partial tiles of a K split (two per CTA): which plan a shape gets does not change what it needs.
size_t qk_gemm_tc_part_bytes(int sm_count);
size_t qk_gemm_tc_scratch_bytes(const QkTcCall &c, int sm_count);
cudaError_t qk_launch_gemm_tc(const QkTcCall &c, unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s);

// Mixture-of-experts glue (routing, token lists, gather, silu * up, weighted scatter-add).
cudaError_t qk_launch_moe_route(const float *logits, uint32_t tokens, uint32_t n_exp, uint32_t top_k,
                                int *ids, float *wts, cudaStream_t s);
// Both for a call whose experts go together, in one launch where the pairs are few enough.
#define QK_MOE_PLAN_SLOTS 16384u
cudaError_t qk_launch_moe_group_plan(const float *logits, uint32_t tokens, uint32_t n_exp, uint32_t top_k,
                                     uint32_t expert_begin, uint32_t n_local, int *ids, float *wts, int *counts,
                                     int *lists, int *pos, cudaStream_t s);
cudaError_t qk_launch_moe_lists(const int *ids, uint32_t tokens, uint32_t top_k, uint32_t expert_begin,
                                uint32_t n_local, int *counts, int *lists, int *pos, cudaStream_t s);
// y[token] = sum in slot order of wts * output row; the rows of expert e lie at o + e * cap (position
// pos inside), or, where `by_slot` is given and big[e] == 0, at by_slot + slot.
cudaError_t qk_launch_moe_combine(const float *o, const float *by_slot, const int *big, const int *ids, const int *pos,
                                  const float *wts, uint32_t tokens, uint32_t top_k, uint32_t expert_begin,
                                  uint32_t n_local, uint32_t cap, uint32_t hidden, float *y, cudaStream_t s);
cudaError_t qk_launch_moe_gather(const float *x, const int *list, uint32_t n, uint32_t top_k,
                                 uint32_t hidden, float *xe, cudaStream_t s);
cudaError_t qk_launch_moe_silu_mul(const float *g, float *u, uint64_t n, cudaStream_t s);
// g <- silu(g) * u (swiglu_inplace of the dense feed-forward block)
cudaError_t qk_launch_swiglu(float *g, const float *u, uint64_t n, cudaStream_t s);
cudaError_t qk_launch_moe_scatter(const float *o, const int *list, const float *wts, uint32_t n,
                                  uint32_t top_k, uint32_t hidden, float *y, cudaStream_t s);
cudaError_t qk_launch_moe_take_rows(const float *x, const int *idx, uint32_t n, uint32_t width, float *out,
                                    cudaStream_t s);
cudaError_t qk_launch_moe_sum_rows(const float *src, const int *idx, uint32_t tokens, uint32_t per_row,
                                   uint32_t width, float *y, cudaStream_t s);

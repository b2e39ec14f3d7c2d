// Definitions shared by the translation units that implement the C ABI.
#pragma once
#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include "../../include/qk_cuda.h"
#include "qk_kernels.h"

struct qk_weights {
  QkLayout L;
  uint8_t *dev;
  int device;
  size_t algo_bytes;
  float *rows = nullptr;  // factors of the rows for the tcgen05 matmul (behind the matrix in `dev`)
  bool wide = false;      // and whether a row's blocks differ widely (qk_gemm_tc_factors)
  alignas(64) unsigned char tmap[128];  // tensor map of `dev` for the tcgen05 matmul (formats it serves)
  uint64_t fp = 0;  // content fingerprint of the host buffer it was uploaded from (host-pointer cache only)
};

// Host calls of up to this many bytes go through the context's own pinned staging: a driver copy from
// or to pageable memory costs more than the memcpy (larger ones are left to the driver, which overlaps).
#define QK_HOST_STAGE ((size_t)256 << 10)

#define QK_UPLOAD_STAGE ((size_t)32 << 20)

// A context starts with scratch for this many bytes of converted activations beside the partial tiles of a
// matmul (128 rows of 4096 columns and their rounding): calls up to there never grow it, so they may be
// captured without a call before.
#define QK_MIN_SCRATCH ((size_t)2 << 20)

struct QkScratch {
  unsigned char *p = nullptr;
  size_t cap = 0;
};

// Images of split activations, one per stream, for the formats whose calls may overlap on different
// streams (Q5_K, Q3_K, Q2_K).  A slot belongs to the stream that first asked for it, by its id (which,
// unlike a handle, is never used again), until the context ends.
#define QK_IMAGES 16
#define QK_IMAGE_BYTES ((size_t)256 << 10)  // above what fits a CTA's shared memory

struct qk_ctx {
  int device;
  int sm_count;
  cudaStream_t stream;
  // Status word raised by device code (bounded waits that ran out, range checks): one word of
  // pinned host memory that the kernels reach through its device mapping, so the host reads
  // it after a stream synchronise without another copy.
  unsigned *status_dev;                  // device-side address, passed to kernels
  volatile unsigned *status_host = nullptr;  // the same word as the host sees it
  // device scratch of the *_dev entry points (split or converted activations, partial tiles); grown on
  // demand, which synchronises: size it once before capturing into a CUDA graph.  The host-pointer entry
  // points have their own: they run on the context's stream, where nothing orders them behind *_dev calls
  // that are still in flight on the caller's.
  QkScratch scratch, host_scratch;
  unsigned char *images = nullptr;  // QK_IMAGES slots, made with the context
  unsigned long long image_of[QK_IMAGES] = {};
  int n_images = 0;
  std::string err;
  std::mutex mu;
  // scratch for the host-pointer entry points
  void *sa = nullptr, *sb = nullptr;
  size_t sa_cap = 0, sb_cap = 0;
  // pinned, device-mapped staging of those calls' activations and results (QK_HOST_STAGE bytes each,
  // made by the first such call)
  unsigned char *hx = nullptr, *hx_dev = nullptr, *hy = nullptr, *hy_dev = nullptr;
  // device buffer through which weights are uploaded (QK_UPLOAD_STAGE bytes, made by the first upload)
  uint8_t *up = nullptr;
  // weight cache for the host-pointer entry points
  typedef std::tuple<const void *, size_t, int, size_t, size_t, uint64_t> Key;
  std::map<Key, qk_weights *> cache;
  size_t cache_bytes = 0, cache_cap = (size_t)64 << 30;
  bool force_simple = false;
  // scratch of qk_moe_ffn_dev (routing tables and per-expert activations); grown on demand
  void *moe = nullptr;
  size_t moe_cap = 0;
  // scratch of qk_ffn_dev (the hidden activations between the projections); grown on demand
  void *ffn = nullptr;
  size_t ffn_cap = 0;
};

// Grows `sc` (with a device synchronise) to twice `need` bytes, if it is smaller than `need`.
int qk_ensure_scratch(qk_ctx *c, QkScratch &sc, size_t need);

// C ABI of the backend (see include/qk_cuda.h): argument checking in the
// reference's order, the context (stream, scratch, weight cache), and the
// choice of kernel for each shape.  Nothing here computes on the CPU: a call
// that cannot reach the GPU returns QK_CUDA_ERROR.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include <vector>

#include "qk_internal.h"
#include "qk_moe_plan.cuh"

#define CK(ctx, call)                                                                     \
  do {                                                                                    \
    cudaError_t e__ = (call);                                                             \
    if (e__ != cudaSuccess) {                                                             \
      (ctx)->err = std::string(#call) + ": " + cudaGetErrorString(e__);                   \
      return QK_CUDA_ERROR;                                                               \
    }                                                                                     \
  } while (0)

static bool type_ok(int t) {
  return t == QK_TYPE_Q4_0 || t == QK_TYPE_Q8_0 || t == QK_TYPE_Q4_K || t == QK_TYPE_Q5_K || t == QK_TYPE_Q6_K ||
         t == QK_TYPE_IQ4_XS || t == QK_TYPE_Q2_K || t == QK_TYPE_Q3_K || t == QK_TYPE_Q8_K;
}

extern "C" size_t qk_block_size(int type) {
  switch (type) {
    case QK_TYPE_Q4_0:
    case QK_TYPE_Q8_0:
      return 32;
    case QK_TYPE_Q2_K:
    case QK_TYPE_Q3_K:
    case QK_TYPE_Q4_K:
    case QK_TYPE_Q5_K:
    case QK_TYPE_Q6_K:
    case QK_TYPE_Q8_K:
    case QK_TYPE_IQ4_XS:
      return 256;
    default:
      return 0;
  }
}

extern "C" size_t qk_block_bytes(int type) {
  switch (type) {
    case QK_TYPE_Q4_0:
      return 18;
    case QK_TYPE_Q8_0:
      return 34;
    case QK_TYPE_Q4_K:
      return 144;
    case QK_TYPE_Q5_K:
      return 176;
    case QK_TYPE_Q2_K:
      return 84;
    case QK_TYPE_Q3_K:
      return 110;
    case QK_TYPE_Q8_K:
      return 292;
    case QK_TYPE_Q6_K:
      return 210;
    case QK_TYPE_IQ4_XS:
      return 136;
    default:
      return 0;
  }
}

extern "C" const char *qk_name(int type) {
  switch (type) {
    case QK_TYPE_Q4_0:
      return "Q4_0";
    case QK_TYPE_Q8_0:
      return "Q8_0";
    case QK_TYPE_Q4_K:
      return "Q4_K";
    case QK_TYPE_Q5_K:
      return "Q5_K";
    case QK_TYPE_Q2_K:
      return "Q2_K";
    case QK_TYPE_Q3_K:
      return "Q3_K";
    case QK_TYPE_Q8_K:
      return "Q8_K";
    case QK_TYPE_Q6_K:
      return "Q6_K";
    case QK_TYPE_IQ4_XS:
      return "IQ4_XS";
    default:
      return nullptr;
  }
}

extern "C" int qk_init(int device, qk_ctx **out) {
  if (!out) return QK_INVALID_ARGUMENT;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) return QK_CUDA_ERROR;
  if (cudaSetDevice(device) != cudaSuccess) return QK_CUDA_ERROR;
  qk_ctx *c = new qk_ctx();
  c->device = device;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess || prop.major != 10) {
    delete c;  // the kernels are sm_100a-only
    return QK_CUDA_ERROR;
  }
  c->sm_count = prop.multiProcessorCount;
  unsigned *sh = nullptr;
  const size_t scratch = QK_MIN_SCRATCH + qk_gemm_tc_part_bytes(c->sm_count);
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaHostAlloc((void **)&sh, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess ||
      cudaHostGetDevicePointer((void **)&c->status_dev, sh, 0) != cudaSuccess ||
      cudaMalloc(&c->scratch.p, scratch) != cudaSuccess ||
      cudaMalloc(&c->host_scratch.p, scratch) != cudaSuccess ||  // (here: the first host call would wait milliseconds for it)
      cudaMalloc(&c->images, QK_IMAGES * QK_IMAGE_BYTES) != cudaSuccess) {
    if (sh) cudaFreeHost(sh);
    if (c->scratch.p) cudaFree(c->scratch.p);
    if (c->host_scratch.p) cudaFree(c->host_scratch.p);
    delete c;
    return QK_CUDA_ERROR;
  }
  *sh = 0;
  c->status_host = sh;
  c->scratch.cap = c->host_scratch.cap = scratch;
  const char *fs = qk_knob("QK_FORCE_SIMPLE");
  c->force_simple = fs && fs[0] == '1';
  *out = c;
  return QK_OK;
}

static void free_weights(qk_weights *h) {
  if (!h) return;
  if (h->dev) cudaFree(h->dev);
  delete h;
}

extern "C" int qk_shutdown(qk_ctx *c) {
  if (!c) return QK_INVALID_ARGUMENT;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  for (auto &kv : c->cache) free_weights(kv.second);
  if (c->sa) cudaFree(c->sa);
  if (c->sb) cudaFree(c->sb);
  cudaFreeHost((void *)c->status_host);
  if (c->hx) cudaFreeHost(c->hx);
  if (c->scratch.p) cudaFree(c->scratch.p);
  if (c->host_scratch.p) cudaFree(c->host_scratch.p);
  cudaFree(c->images);
  if (c->moe) cudaFree(c->moe);
  if (c->ffn) cudaFree(c->ffn);
  if (c->up) cudaFree(c->up);
  cudaStreamDestroy(c->stream);
  delete c;
  return QK_OK;
}

extern "C" int qk_last_error(qk_ctx *c, char *buf, size_t buf_len) {
  if (!c || !buf || buf_len == 0) return QK_INVALID_ARGUMENT;
  snprintf(buf, buf_len, "%s", c->err.c_str());
  return QK_OK;
}

static int grow(qk_ctx *c, void **p, size_t *cap, size_t need) {
  if (need <= *cap) return QK_OK;
  if (*p) {
    CK(c, cudaStreamSynchronize(c->stream));
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
  }
  size_t want = need + need / 4 + 256;
  CK(c, cudaMalloc(p, want));
  *cap = want;
  return QK_OK;
}

static size_t need_bytes(int type, size_t n_rows, size_t n_cols) {
  size_t bs = qk_block_size(type), bb = qk_block_bytes(type);
  return n_rows * ((n_cols + bs - 1) / bs) * bb;
}

// ------------------------------------------------------------ upload
static int upload_impl(qk_ctx *c, int type, const uint8_t *w, size_t n_cols, size_t row_begin,
                       size_t row_end, qk_weights **out) {
  size_t rows = row_end - row_begin;
  qk_weights *h = new qk_weights();
  h->device = c->device;
  h->dev = nullptr;
  if (!qk_make_layout(type, rows, n_cols, &h->L)) {
    delete h;
    return QK_UNSUPPORTED_TYPE;
  }
  h->algo_bytes = need_bytes(type, rows, n_cols);
  size_t row_bytes = (size_t)h->L.nb * h->L.bb;
  size_t tiled = h->L.total_bytes ? h->L.total_bytes + qk_gemm_tc_pad_bytes(h->L) : 16;
  cudaError_t e = cudaMalloc(&h->dev, tiled + qk_gemm_tc_factor_bytes(h->L));  // (tiled is a multiple of 16)
  h->rows = (float *)(h->dev + tiled);
  if (e != cudaSuccess) {
    c->err = std::string("cudaMalloc(weights): ") + cudaGetErrorString(e);
    delete h;
    return QK_CUDA_ERROR;
  }
  if (qk_gemm_tc_supported(h->L, 1) && (e = qk_gemm_tc_map(h->L, h->dev, h->tmap)) != cudaSuccess) {
    c->err = std::string("weights upload: tensor map: ") + cudaGetErrorString(e);
    free_weights(h);
    return QK_CUDA_ERROR;
  }
  // The GGUF bytes pass through the context's upload buffer, whole 8-row chunks at a time (a device
  // allocation and a release per call cost more than the repacking, and now and then many milliseconds);
  // only rows of which it does not hold eight get a buffer of their own.
  int st = QK_OK;
  uint8_t *raw = nullptr;
  do {
    // every byte of a whole chunk is written by the repacking: clear only one with rows missing and what lies behind
    const uint64_t whole = h->L.rows / QK_TILE_ROWS * h->L.chunk_bytes;
    if (whole < tiled && (e = cudaMemsetAsync(h->dev + whole, 0, tiled - whole, c->stream)) != cudaSuccess) break;
    if (h->algo_bytes == 0) break;
    size_t step = QK_UPLOAD_STAGE / (QK_TILE_ROWS * row_bytes) * QK_TILE_ROWS;
    if (step && !c->up && (e = cudaMalloc(&c->up, QK_UPLOAD_STAGE)) != cudaSuccess) break;
    if (!step) {
      step = QK_TILE_ROWS;
      if ((e = cudaMalloc(&raw, step * row_bytes)) != cudaSuccess) break;
    }
    uint8_t *buf = raw ? raw : c->up;
    for (size_t r = 0; r < h->L.rows && e == cudaSuccess; r += step) {
      QkLayout part;
      const size_t n = h->L.rows - r < step ? h->L.rows - r : step;
      qk_make_layout(type, n, n_cols, &part);
      e = cudaMemcpyAsync(buf, w + (row_begin + r) * row_bytes, n * row_bytes, cudaMemcpyHostToDevice, c->stream);
      if (e == cudaSuccess) e = qk_launch_repack(part, buf, h->dev + r / QK_TILE_ROWS * h->L.chunk_bytes, c->stream);
    }
  } while (0);
  if (e == cudaSuccess) e = qk_gemm_tc_factors(h->L, h->dev, h->rows, &h->wide, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  else cudaStreamSynchronize(c->stream);
  if (raw) cudaFree(raw);
  if (e != cudaSuccess) {
    c->err = std::string("weights upload: ") + cudaGetErrorString(e);
    free_weights(h);
    st = QK_CUDA_ERROR;
  } else {
    *out = h;
  }
  return st;
}

extern "C" int qk_weights_upload(qk_ctx *c, int type, const uint8_t *w, size_t w_len, size_t n_rows,
                                 size_t n_cols, size_t row_begin, size_t row_end,
                                 qk_weights **out) {
  if (!c || !out) return QK_INVALID_ARGUMENT;
  *out = nullptr;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  if (row_begin > row_end || row_end > n_rows) return QK_INVALID_ARGUMENT;
  if (n_rows >= (1ull << 31) || n_cols >= (1ull << 31)) return QK_INVALID_ARGUMENT;
  if (w_len < need_bytes(type, n_rows, n_cols)) return QK_BUFFER_TOO_SMALL;
  if (!w && need_bytes(type, n_rows, n_cols) > 0) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  CK(c, cudaSetDevice(c->device));
  return upload_impl(c, type, w, n_cols, row_begin, row_end, out);
}

extern "C" int qk_weights_free(qk_ctx *c, qk_weights *h) {
  if (!c || !h) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  cudaSetDevice(c->device);
  free_weights(h);
  return QK_OK;
}

extern "C" int qk_weights_info(const qk_weights *h, int *type, size_t *rows, size_t *cols,
                               size_t *bytes) {
  if (!h) return QK_INVALID_ARGUMENT;
  if (type) *type = h->L.type;
  if (rows) *rows = h->L.rows;
  if (cols) *cols = h->L.cols;
  if (bytes) *bytes = h->algo_bytes;
  return QK_OK;
}

// Cheap content fingerprint of a host weight buffer: every byte when it is small, else its
// first and last 256 bytes and 64 evenly spread 8-byte samples (about 70 cache lines: the
// check runs on every host-pointer call, and the 2048 samples it once took were a dozen
// microseconds of cache misses per call on weights that do not fit the host's caches).  It
// guards the pointer-keyed cache against a freed buffer's address being reused for other
// weights; it does not detect a few bytes edited in place (qk_weights_cache_evict).
static uint64_t fingerprint(const uint8_t *w, size_t n) {
  uint64_t h = 1469598103934665603ull ^ n;
  auto mix = [&](uint64_t v) { h = (h ^ v) * 1099511628211ull; h ^= h >> 29; };
  if (n <= 4096) {
    size_t i = 0;
    for (; i + 8 <= n; i += 8) { uint64_t v; memcpy(&v, w + i, 8); mix(v); }
    for (; i < n; i++) mix(w[i]);
    return h;
  }
  for (size_t i = 0; i < 256; i += 8) { uint64_t v; memcpy(&v, w + i, 8); mix(v); }
  for (size_t i = n - 256; i + 8 <= n; i += 8) { uint64_t v; memcpy(&v, w + i, 8); mix(v); }
  const size_t step = (n - 8) / 64;
  for (size_t k = 0; k < 64; k++) { uint64_t v; memcpy(&v, w + k * step, 8); mix(v); }
  return h;
}

// Cached device copy for the host-pointer entry points, keyed by (pointer, length, type,
// shape); a hit whose fingerprint no longer matches is uploaded again.
static int cached(qk_ctx *c, int type, const uint8_t *w, size_t w_len, size_t n_rows, size_t n_cols,
                  qk_weights **out) {
  const size_t need = need_bytes(type, n_rows, n_cols);
  const uint64_t fp = fingerprint(w, need);
  qk_ctx::Key k(w, w_len, type, n_rows, n_cols, 0);
  auto it = c->cache.find(k);
  if (it != c->cache.end()) {
    if (it->second->fp == fp) {
      *out = it->second;
      return QK_OK;
    }
    CK(c, cudaStreamSynchronize(c->stream));  // other contents behind the same address: drop the stale copy
    c->cache_bytes -= it->second->algo_bytes;
    free_weights(it->second);
    c->cache.erase(it);
  }
  if (c->cache_bytes + need > c->cache_cap) {  // simplest policy: start over
    CK(c, cudaStreamSynchronize(c->stream));
    for (auto &kv : c->cache) free_weights(kv.second);
    c->cache.clear();
    c->cache_bytes = 0;
  }
  int st = upload_impl(c, type, w, n_cols, 0, n_rows, out);
  if (st == QK_OK) {
    (*out)->fp = fp;
    c->cache[k] = *out;
    c->cache_bytes += need;
  }
  return st;
}

extern "C" int qk_weights_cache_evict(qk_ctx *c, const uint8_t *w) {
  if (!c) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  for (auto it = c->cache.begin(); it != c->cache.end();) {
    if (!w || std::get<0>(it->first) == (const void *)w) {
      c->cache_bytes -= it->second->algo_bytes;
      free_weights(it->second);
      it = c->cache.erase(it);
    } else {
      ++it;
    }
  }
  return QK_OK;
}

// ------------------------------------------------------------ device entry points
int qk_ensure_scratch(qk_ctx *c, QkScratch &sc, size_t need) {
  if (need <= sc.cap) return QK_OK;
  CK(c, cudaDeviceSynchronize());
  cudaFree(sc.p);
  sc.p = nullptr, sc.cap = 0;
  CK(c, cudaMalloc(&sc.p, need * 2));
  sc.cap = need * 2;
  return QK_OK;
}

// Where a decode call of m rows leaves its split activations, if it has to.  Formats with a tensor-core
// matmul share the context's scratch; the others, which have no other scratch, take a slot of the call's
// stream, or none: in a capture (the graph may run beside the stream it was captured from) and when all
// slots are taken.  (Without a slot every CTA splits: Q5_K 4096 x 14336, four rows 40.8 us against 33.4.)
static int split_image(qk_ctx *c, QkScratch &sc, const QkLayout &L, size_t m, cudaStream_t s, unsigned char **img) {
  *img = nullptr;
  if (qk_gemm_tc_supported(L, 1) || &sc == &c->host_scratch) {
    int st = qk_ensure_scratch(c, sc, qk_gemv_fast_scratch_bytes(L, (uint32_t)m));
    *img = sc.p;
    return st;
  }
  if (m * L.nb * L.bs <= QK_SPLIT_IN_CTA) return QK_OK;
  cudaStreamCaptureStatus cap;
  unsigned long long id;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone || cudaStreamGetId(s, &id) != cudaSuccess) {
    (void)cudaGetLastError();
    return QK_OK;
  }
  int i = 0;
  while (i < c->n_images && c->image_of[i] != id) i++;
  if (i == QK_IMAGES) return QK_OK;
  if (i == c->n_images) c->image_of[c->n_images++] = id;
  *img = c->images + i * QK_IMAGE_BYTES;
  return QK_OK;
}

static int tc_call(qk_ctx *c, QkScratch &sc, const QkTcCall &call, cudaStream_t s) {
  int st = qk_ensure_scratch(c, sc, qk_gemm_tc_scratch_bytes(call, c->sm_count));
  if (st) return st;
  CK(c, qk_launch_gemm_tc(call, c->status_dev, sc.p, c->sm_count, s));
  return QK_OK;
}

// Whether m > 4 rows of a format without a tensor-core matmul take less time as pieces of `step` rows on the
// decode kernels than on the generic kernel, which decodes a weight once per eight rows in one launch: it wins
// where the matrix is too small to repay a launch per piece (Q2_K 8 x 256 by 1024: 21 against 1440 us; Q5_K 1024 x
// 4096 by 256: 1516 against 343).  Microseconds of both: over 222 shapes (8 x 256 .. 4096 x 4096, 5 .. 1024
// rows) the choice takes 1.001 times the faster one's time in the mean, 1.16 at worst.
static bool pieces_pay(const QkLayout &L, size_t m, size_t step) {
  const double cols = L.cols, elems = cols * L.rows, eights = (double)((m + 7) / 8), pieces = (double)((m + step - 1) / step);
  const double chain = 0.031 * cols * ceil(eights / 64), all = 1.1e-5 * elems * eights;  // a warp's row; all weights on all SMs
  const double generic = 5 + (L.type == QK_TYPE_Q3_K ? 1.25 : 1.0) * (chain > all ? chain : all);
  const double acts = step * cols;  // (Q5_K: the more there are, the fewer weight tiles fit beside them)
  const double split = L.type == QK_TYPE_Q5_K ? (1e-4 + 1e-9 * acts) * acts : 1.8e-4 * acts;
  return pieces * (3.2 + split + 2.5e-4 * L.rows + 1.9e-7 * elems) <= generic;
}

static int gemm_dispatch(qk_ctx *c, QkScratch &sc, const qk_weights *h, const float *x, float *y, size_t m,
                         size_t ldy, cudaStream_t s) {
  if (h->L.rows == 0 || m == 0) return QK_OK;
  if (h->L.cols == 0) {  // empty dot products
    CK(c, cudaMemset2DAsync(y, ldy * sizeof(float), 0, h->L.rows * sizeof(float), m, s));
    return QK_OK;
  }
  // Formats without a tensor-core matmul (Q5_K, Q3_K, Q2_K) take a batch on the decode kernels too, as many
  // rows at a time as these take: the weights are streamed once per four rows (or two), where the generic
  // kernel decodes them byte by byte once per eight.
  const bool tc = qk_gemm_tc_supported(h->L, 1);
  if (!c->force_simple && qk_gemv_fast_supported(h->L, 1) && (m <= QK_GEMV_MAX_M || !tc)) {
    size_t step = m < QK_GEMV_MAX_M ? m : QK_GEMV_MAX_M;
    while (step > 1 && !qk_gemv_fast_supported(h->L, (uint32_t)step)) step--;
    if (step == m || (!tc && (m <= QK_GEMV_MAX_M || pieces_pay(h->L, m, step)))) {
      unsigned char *img;
      int st = split_image(c, sc, h->L, step, s, &img);
      if (st) return st;
      for (size_t i = 0; i < m; i += step) {
        const uint32_t k = (uint32_t)(m - i < step ? m - i : step);
        CK(c, qk_launch_gemv_fast(h->L, h->dev, x + i * h->L.cols, y + i * ldy, k, ldy, c->status_dev, img, c->sm_count, s));
      }
      return QK_OK;
    }
  }
  // The tensor-core path rounds its operands to fp16; what the decode kernels take keeps f32-grade
  // activations.  Two to four rows that they do not take go to the tensor cores as well: three and four of
  // Q6_K (registers), and rows whose split does not fit the shared memory beside the tiles (four of Q4_K and
  // Q4_0 from 10240 columns, of IQ4_XS from 10496, of Q8_0 from 7680; two of Q8_0 from 12288, of Q6_K from 12544, of
  // Q4_K and Q4_0 from 16640, of IQ4_XS from 17408).  One row too long for them, and a K that is not a multiple
  // of 256, go to the generic kernel below.
  const bool tc_small = m <= QK_GEMV_MAX_M && m > 1 && qk_gemv_fast_supported(h->L, 1);
  if (!c->force_simple && (m > QK_GEMV_MAX_M || tc_small) && m < (1u << 30) &&
      qk_gemm_tc_supported(h->L, (uint32_t)m)) {
    QkTcCall call = {};
    call.L = &h->L, call.maps[0] = h->tmap, call.rows[0] = h->rows, call.wide = h->wide, call.n = call.n_act = 1;
    call.x = x, call.m = (uint32_t)m, call.y = y, call.ldy = ldy;
    return tc_call(c, sc, call, s);
  }
  CK(c, qk_launch_gemm_simple(h->L, h->dev, x, y, (uint32_t)m, ldy, s));
  return QK_OK;
}

extern "C" int qk_gemv_dev(qk_ctx *c, const qk_weights *h, const float *x_dev, float *y_dev,
                           void *stream) {
  if (!c || !h || !x_dev || !y_dev) return QK_INVALID_ARGUMENT;
  if (h->device != c->device) return QK_INVALID_ARGUMENT;
  return gemm_dispatch(c, c->scratch, h, x_dev, y_dev, 1, h->L.rows, (cudaStream_t)stream);
}

extern "C" int qk_gemm_dev(qk_ctx *c, const qk_weights *h, const float *x_dev, float *y_dev,
                           size_t m, size_t ldy, void *stream) {
  if (!c || !h || !x_dev || !y_dev) return QK_INVALID_ARGUMENT;
  if (h->device != c->device) return QK_INVALID_ARGUMENT;
  if (ldy < h->L.rows) return QK_DIMENSION_MISMATCH;
  return gemm_dispatch(c, c->scratch, h, x_dev, y_dev, m, ldy, (cudaStream_t)stream);
}

extern "C" int qk_moe_route_dev(qk_ctx *c, const float *logits_dev, size_t tokens, size_t n_exp,
                                size_t top_k, int *ids_dev, float *wts_dev, void *stream) {
  if (!c || !logits_dev || !ids_dev || !wts_dev) return QK_INVALID_ARGUMENT;
  if (n_exp == 0 || top_k == 0 || n_exp > 4096) return QK_INVALID_ARGUMENT;
  CK(c, qk_launch_moe_route(logits_dev, (uint32_t)tokens, (uint32_t)n_exp, (uint32_t)top_k, ids_dev, wts_dev,
                            (cudaStream_t)stream));
  return QK_OK;
}

extern "C" int qk_moe_take_rows_dev(qk_ctx *c, const float *x_dev, const int *idx_dev, size_t n, size_t width,
                                    float *out_dev, void *stream) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (n == 0 || width == 0) return QK_OK;
  if (!x_dev || !idx_dev || !out_dev || n > 0x7fffffffu || width > 0x7fffffffu) return QK_INVALID_ARGUMENT;
  CK(c, qk_launch_moe_take_rows(x_dev, idx_dev, (uint32_t)n, (uint32_t)width, out_dev, (cudaStream_t)stream));
  return QK_OK;
}

extern "C" int qk_moe_sum_rows_dev(qk_ctx *c, const float *src_dev, const int *idx_dev, size_t tokens,
                                   size_t per_row, size_t width, float *y_dev, void *stream) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (tokens == 0 || width == 0) return QK_OK;
  if (!y_dev || (per_row && (!src_dev || !idx_dev)) || tokens > 0x7fffffffu || per_row > 0x7fffffffu ||
      width > 0x7fffffffu)
    return QK_INVALID_ARGUMENT;
  CK(c, qk_launch_moe_sum_rows(src_dev, idx_dev, (uint32_t)tokens, (uint32_t)per_row, (uint32_t)width, y_dev,
                               (cudaStream_t)stream));
  return QK_OK;
}

extern "C" int qk_moe_ffn_dev(qk_ctx *c, const qk_weights *const *gate, const qk_weights *const *up,
                              const qk_weights *const *down, size_t n_local, size_t expert_begin,
                              size_t n_exp, const float *logits_dev, const float *x_dev, float *y_dev,
                              size_t tokens, size_t top_k, void *stream) {
  if (!c || !logits_dev || !x_dev || !y_dev || (n_local && (!gate || !up || !down))) return QK_INVALID_ARGUMENT;
  if (n_exp == 0 || top_k == 0 || n_exp > 4096 || expert_begin + n_local > n_exp) return QK_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  size_t hidden = 0, inter = 0;
  for (size_t e = 0; e < n_local; e++) {
    if (!gate[e] || !up[e] || !down[e]) return QK_INVALID_ARGUMENT;
    if (gate[e]->device != c->device || up[e]->device != c->device || down[e]->device != c->device)
      return QK_INVALID_ARGUMENT;
    if (e == 0) hidden = gate[e]->L.cols, inter = gate[e]->L.rows;
    if (gate[e]->L.cols != hidden || gate[e]->L.rows != inter || up[e]->L.cols != hidden ||
        up[e]->L.rows != inter || down[e]->L.cols != inter || down[e]->L.rows != hidden)
      return QK_DIMENSION_MISMATCH;
  }
  if (n_local == 0 || tokens == 0) return QK_OK;
  const size_t slots = tokens * top_k;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  auto grow_moe = [&](size_t need) -> int {
    if (need > c->moe_cap) {
      CK(c, cudaDeviceSynchronize());
      if (c->moe) cudaFree(c->moe);
      c->moe = nullptr, c->moe_cap = 0;
      CK(c, cudaMalloc(&c->moe, need));
      c->moe_cap = need;
    }
    return QK_OK;
  };

  // Experts of one format (per projection) that the tensor-core kernel takes go together, every
  // projection in one launch over all local experts; the token counts stay on the device and nothing is
  // read back, so the whole call is a fixed sequence of launches with no host synchronisation.
  bool grouped = !c->force_simple && n_local <= QK_MAX_GROUPS && n_local <= QK_MOE_MAX && hidden > 0 && inter > 0;
  for (size_t e = 0; e < n_local && grouped; e++)
    grouped = gate[e]->L.type == gate[0]->L.type && up[e]->L.type == gate[0]->L.type &&
              down[e]->L.type == down[0]->L.type && qk_gemm_tc_supported(gate[e]->L, 1) &&
              qk_gemm_tc_supported(down[e]->L, 1);
  // gate / up / down of the experts' rows in `lists` (counts in cnt) on the tensor cores: outputs at o,
  // `cap` rows apart per expert (an expert may receive every token; only the live rows are touched)
  const size_t cap = tokens, rows = n_local * cap;
  auto on_tensor_cores = [&](const int *cnt, const int *lists, float *g, float *o) -> int {
    float *u = g + rows * inter;
    QkTcCall gu = {};
    gu.L = &gate[0]->L, gu.n_act = (uint32_t)n_local, gu.counts = cnt, gu.m = (uint32_t)tokens;
    gu.expect = (uint32_t)((slots + n_exp - 1) / n_exp), gu.xcap = gu.ycap = (uint32_t)cap;
    gu.live = (uint32_t)slots;
    gu.x = x_dev, gu.lists = lists, gu.list_stride = (uint32_t)slots, gu.list_div = (uint32_t)top_k;
    gu.y = g, gu.ldy = inter;
    // gate and up as 2 n groups over n activation groups (groups n .. 2 n - 1 write u, behind g)
    const bool one_launch = 2 * n_local <= QK_MAX_GROUPS;
    for (size_t e = 0; e < n_local; e++) gu.maps[e] = gate[e]->tmap, gu.rows[e] = gate[e]->rows, gu.wide |= gate[e]->wide;
    if (one_launch)
      for (size_t e = 0; e < n_local; e++) gu.maps[n_local + e] = up[e]->tmap, gu.rows[n_local + e] = up[e]->rows, gu.wide |= up[e]->wide;
    gu.n = (uint32_t)(one_launch ? 2 * n_local : n_local);
    int st = tc_call(c, c->scratch, gu, s);
    if (st) return st;
    if (!one_launch) {
      gu.wide = false;
      for (size_t e = 0; e < n_local; e++) gu.maps[e] = up[e]->tmap, gu.rows[e] = up[e]->rows, gu.wide |= up[e]->wide;
      gu.y = u;
      if ((st = tc_call(c, c->scratch, gu, s))) return st;
    }
    // silu(g) * u is formed where the down projection's activations are converted
    QkTcCall dn = {};
    dn.L = &down[0]->L, dn.n = dn.n_act = (uint32_t)n_local, dn.counts = cnt, dn.m = (uint32_t)tokens, dn.expect = gu.expect, dn.live = gu.live;
    dn.xcap = dn.ycap = (uint32_t)cap, dn.x = g, dn.x2 = u, dn.y = o, dn.ldy = hidden;
    for (size_t e = 0; e < n_local; e++) dn.maps[e] = down[e]->tmap, dn.rows[e] = down[e]->rows, dn.wide |= down[e]->wide;
    return tc_call(c, c->scratch, dn, s);
  };

  if (grouped && tokens > QK_MOE_DEC_TOKENS) {
    const size_t o_ids = 0, o_wts = o_ids + al(slots * 4), o_cnt = o_wts + al(slots * 4);
    const size_t o_lists = o_cnt + al(n_local * 4), o_pos = o_lists + al(n_local * slots * 4);
    const size_t o_g = o_pos + al(slots * 4), o_o = o_g + al(2 * rows * inter * 4), need = o_o + al(rows * hidden * 4);
    int st = grow_moe(need);
    if (st) return st;
    unsigned char *base = (unsigned char *)c->moe;
    int *ids = (int *)(base + o_ids), *cnt = (int *)(base + o_cnt), *lists = (int *)(base + o_lists);
    int *pos = (int *)(base + o_pos);
    float *wts = (float *)(base + o_wts), *g = (float *)(base + o_g), *o = (float *)(base + o_o);
    CK(c, qk_launch_moe_group_plan(logits_dev, (uint32_t)tokens, (uint32_t)n_exp, (uint32_t)top_k, (uint32_t)expert_begin,
                                   (uint32_t)n_local, ids, wts, cnt, lists, pos, s));
    if ((st = on_tensor_cores(cnt, lists, g, o))) return st;
    CK(c, qk_launch_moe_combine(o, nullptr, nullptr, ids, pos, wts, (uint32_t)tokens, (uint32_t)top_k, (uint32_t)expert_begin,
                                (uint32_t)n_local, (uint32_t)cap, (uint32_t)hidden, y_dev, s));
    return QK_OK;
  }

  // A handful of tokens: the experts with up to QK_MOE_DEC_ROWS rows on the decode kernels (f32-grade
  // sums, as a plain matmul of that many rows), any others on the tensor cores beside them.  Where K is so
  // long that a job holds one row only (Q8_0 from 12032 columns), nine experts and up can make more jobs
  // than the list takes: such a call goes expert by expert.
  const uint32_t rg = grouped ? qk_moe_dec_rows(gate[0]->L) : 0, rd = grouped ? qk_moe_dec_rows(down[0]->L) : 0;
  const uint32_t per_job = rg < rd ? rg : rd;
  if (grouped && per_job && qk_moe_dec_jobs(slots, n_local, per_job) <= QK_MOE_JOBS) {
    const bool big_too = tokens > QK_MOE_DEC_ROWS;
    const size_t ig = qk_moe_dec_image_bytes(gate[0]->L), id = qk_moe_dec_image_bytes(down[0]->L);
    const size_t o_jobs = 0, o_ids = al(sizeof(QkMoeJobs)), o_wts = o_ids + al(slots * 4), o_big = o_wts + al(slots * 4);
    const size_t o_lists = o_big + al(n_local * 4), o_pos = o_lists + al(n_local * slots * 4), o_ig = o_pos + al(slots * 4);
    const size_t o_h = o_ig + al(tokens * ig), o_id = o_h + al(slots * inter * 4), o_o = o_id + al(slots * id);
    const size_t o_g = o_o + al(slots * hidden * 4), o_ob = o_g + (big_too ? al(2 * rows * inter * 4) : 0);
    int st = grow_moe(o_ob + (big_too ? al(rows * hidden * 4) : 0));
    if (st) return st;
    unsigned char *base = (unsigned char *)c->moe;
    QkMoeJobs *jobs = (QkMoeJobs *)(base + o_jobs);
    int *ids = (int *)(base + o_ids), *big = (int *)(base + o_big), *lists = (int *)(base + o_lists), *pos = (int *)(base + o_pos);
    float *wts = (float *)(base + o_wts), *h = (float *)(base + o_h), *o = (float *)(base + o_o), *ob = (float *)(base + o_ob);
    const uint8_t *wg[QK_MOE_MAX], *wu[QK_MOE_MAX], *wd[QK_MOE_MAX];
    for (size_t e = 0; e < n_local; e++) wg[e] = gate[e]->dev, wu[e] = up[e]->dev, wd[e] = down[e]->dev;
    const qkmoe::PlanArgs plan = {logits_dev, (uint32_t)tokens, (uint32_t)n_exp, (uint32_t)top_k, (uint32_t)expert_begin,
                                  (uint32_t)n_local, per_job, ids, wts, big, lists, pos, jobs};
    CK(c, qk_launch_moe_dec_split(gate[0]->L, x_dev, (uint32_t)tokens, base + o_ig, &plan, s));
    CK(c, qk_launch_moe_dec(gate[0]->L, wg, wu, (uint32_t)n_local, per_job, jobs, base + o_ig, (uint32_t)top_k, h, inter,
                            c->status_dev, c->sm_count, s));
    CK(c, qk_launch_moe_dec_split(down[0]->L, h, (uint32_t)slots, base + o_id, nullptr, s));
    CK(c, qk_launch_moe_dec(down[0]->L, wd, nullptr, (uint32_t)n_local, per_job, jobs, base + o_id, 1, o, hidden, c->status_dev,
                            c->sm_count, s));
    if (big_too && (st = on_tensor_cores(big, lists, (float *)(base + o_g), ob))) return st;
    CK(c, qk_launch_moe_combine(ob, o, big, ids, pos, wts, (uint32_t)tokens, (uint32_t)top_k, (uint32_t)expert_begin,
                                (uint32_t)n_local, (uint32_t)cap, (uint32_t)hidden, y_dev, s));
    return QK_OK;
  }

  // Other formats, mixed formats, more experts: one after the other, sized by the token counts read back.
  // scratch: ids, wts, counts, lists, then the per-expert activations (sized for every token)
  const size_t o_ids = 0, o_wts = o_ids + al(slots * 4), o_cnt = o_wts + al(slots * 4);
  const size_t o_lists = o_cnt + al(n_local * 4), o_xe = o_lists + al(n_local * slots * 4);
  const size_t o_g = o_xe + al(tokens * hidden * 4), o_u = o_g + al(tokens * inter * 4);
  const size_t o_o = o_u + al(tokens * inter * 4), need = o_o + al(tokens * hidden * 4);
  {
    int st = grow_moe(need);
    if (st) return st;
  }
  unsigned char *base = (unsigned char *)c->moe;
  int *ids = (int *)(base + o_ids), *cnt = (int *)(base + o_cnt), *lists = (int *)(base + o_lists);
  float *wts = (float *)(base + o_wts), *xe = (float *)(base + o_xe), *g = (float *)(base + o_g);
  float *u = (float *)(base + o_u), *o = (float *)(base + o_o);

  CK(c, cudaMemsetAsync(y_dev, 0, tokens * hidden * sizeof(float), s));
  CK(c, qk_launch_moe_route(logits_dev, (uint32_t)tokens, (uint32_t)n_exp, (uint32_t)top_k, ids, wts, s));
  CK(c, qk_launch_moe_lists(ids, (uint32_t)tokens, (uint32_t)top_k, (uint32_t)expert_begin, (uint32_t)n_local,
                            cnt, lists, nullptr, s));
  // the token counts size the per-expert matmuls: one small copy and a stream synchronise
  std::vector<int> counts(n_local);
  CK(c, cudaMemcpyAsync(counts.data(), cnt, n_local * sizeof(int), cudaMemcpyDeviceToHost, s));
  CK(c, cudaStreamSynchronize(s));
  for (size_t e = 0; e < n_local; e++) {
    const size_t m = (size_t)counts[e];
    if (m == 0) continue;
    const int *list = lists + e * slots;
    CK(c, qk_launch_moe_gather(x_dev, list, (uint32_t)m, (uint32_t)top_k, (uint32_t)hidden, xe, s));
    int st = gemm_dispatch(c, c->scratch, gate[e], xe, g, m, inter, s);
    if (st) return st;
    st = gemm_dispatch(c, c->scratch, up[e], xe, u, m, inter, s);
    if (st) return st;
    CK(c, qk_launch_moe_silu_mul(g, u, (uint64_t)m * inter, s));
    st = gemm_dispatch(c, c->scratch, down[e], u, o, m, hidden, s);
    if (st) return st;
    CK(c, qk_launch_moe_scatter(o, list, wts, (uint32_t)m, (uint32_t)top_k, (uint32_t)hidden, y_dev, s));
  }
  return QK_OK;
}

// ------------------------------------------------------------ feed-forward block
// FFN(x) = down(silu(gate x) * up x): the dense branch of feed_forward
// (crates/oxillama-arch/src/llama/model.rs:281-310) with swiglu_inplace
// (crates/oxillama-arch/src/common/swiglu.rs:15-21).
extern "C" int qk_ffn_dev(qk_ctx *c, const qk_weights *gate, const qk_weights *up, const qk_weights *down,
                          const float *x_dev, float *y_dev, size_t m, void *stream) {
  if (!c || !gate || !up || !down || !x_dev || !y_dev) return QK_INVALID_ARGUMENT;
  if (gate->device != c->device || up->device != c->device || down->device != c->device) return QK_INVALID_ARGUMENT;
  const size_t hidden = gate->L.cols, inter = gate->L.rows;
  if (up->L.cols != hidden || up->L.rows != inter || down->L.cols != inter) return QK_DIMENSION_MISMATCH;
  if (m == 0 || down->L.rows == 0) return QK_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // scratch: h (and, on the unfused route, the up projection) [m x inter] each
  const size_t need = 2 * m * (inter ? inter : 1) * sizeof(float);
  if (need > c->ffn_cap) {
    CK(c, cudaDeviceSynchronize());
    if (c->ffn) cudaFree(c->ffn);
    c->ffn = nullptr, c->ffn_cap = 0;
    CK(c, cudaMalloc(&c->ffn, need));
    c->ffn_cap = need;
  }
  float *h = (float *)c->ffn, *u = h + m * inter;
  const bool fused = !c->force_simple && gate->L.type == up->L.type && hidden > 0 && inter > 0 && m <= QK_GEMV_MAX_M && qk_gemv_dual_supported(gate->L, (uint32_t)m);
  if (fused) {
    // gate and up in one launch (they share the split activations), silu(g) * u in its reducer
    unsigned char *img;
    int st = split_image(c, c->scratch, gate->L, m, s, &img);
    if (st) return st;
    CK(c, qk_launch_gemv_dual(gate->L, gate->dev, up->dev, x_dev, h, (uint32_t)m, inter, c->status_dev, img,
                              c->sm_count, s));
  } else if (!c->force_simple && m > QK_GEMV_MAX_M && m < (1u << 30) && hidden > 0 && inter > 0 && gate->L.type == up->L.type &&
             qk_gemm_tc_supported(gate->L, (uint32_t)m) && qk_gemm_tc_supported(down->L, (uint32_t)m)) {
    // Batches: gate and up as one tensor-core launch over the activations converted once, and
    // silu(g) * u formed where the down projection's activations are converted.
    QkTcCall gu = {};
    gu.L = &gate->L, gu.maps[0] = gate->tmap, gu.maps[1] = up->tmap, gu.rows[0] = gate->rows, gu.rows[1] = up->rows, gu.wide = gate->wide || up->wide, gu.n = 2, gu.n_act = 1;
    gu.x = x_dev, gu.m = (uint32_t)m, gu.xcap = gu.ycap = (uint32_t)m, gu.y = h, gu.ldy = inter;
    int st = tc_call(c, c->scratch, gu, s);
    if (st) return st;
    QkTcCall dn = {};
    dn.L = &down->L, dn.maps[0] = down->tmap, dn.rows[0] = down->rows, dn.wide = down->wide, dn.n = dn.n_act = 1;
    dn.x = h, dn.x2 = u, dn.m = (uint32_t)m, dn.y = y_dev, dn.ldy = down->L.rows;
    return tc_call(c, c->scratch, dn, s);
  } else {
    int st = gemm_dispatch(c, c->scratch, gate, x_dev, h, m, inter, s);
    if (st) return st;
    if ((st = gemm_dispatch(c, c->scratch, up, x_dev, u, m, inter, s))) return st;
    CK(c, qk_launch_swiglu(h, u, (uint64_t)m * inter, s));
  }
  return gemm_dispatch(c, c->scratch, down, h, y_dev, m, down->L.rows, s);
}

extern "C" int qk_dequant_dev(qk_ctx *c, const qk_weights *h, float *out_dev, void *stream) {
  if (!c || !h || !out_dev) return QK_INVALID_ARGUMENT;
  CK(c, qk_launch_dequant(h->L, h->dev, out_dev, (cudaStream_t)stream));
  return QK_OK;
}

extern "C" int qk_matvec_q8_fused_dev(qk_ctx *c, const qk_weights *h, const uint8_t *acts_q8_dev,
                                      float *out_dev, void *stream) {
  if (!c || !h || !acts_q8_dev || !out_dev) return QK_INVALID_ARGUMENT;
  CK(c, qk_launch_fused_simple(h->L, h->dev, acts_q8_dev, out_dev, (cudaStream_t)stream));
  return QK_OK;
}

extern "C" int qk_quantize_q8_0_dev(qk_ctx *c, const float *x_dev, size_t n, uint8_t *out_dev,
                                    void *stream) {
  if (!c || (n && (!x_dev || !out_dev))) return QK_INVALID_ARGUMENT;
  if (n % 32 != 0) return QK_DIMENSION_MISMATCH;
  CK(c, qk_launch_quantize_q8_0(x_dev, n, out_dev, (cudaStream_t)stream));
  return QK_OK;
}

// Reads and clears the status word; the stream that ran the kernels must have been synchronised.
static int take_device_status(qk_ctx *c) {
  const unsigned v = *c->status_host;
  if (!v) return QK_OK;
  *c->status_host = 0;
  c->err = (v & QK_DEV_TIMEOUT) ? "device-side wait ran out" : "device-side range check tripped";
  return (v & QK_DEV_TIMEOUT) ? QK_TIMEOUT : QK_KERNEL_ERROR;
}

extern "C" int qk_check_device_status(qk_ctx *c, void *stream) {
  if (!c) return QK_INVALID_ARGUMENT;
  CK(c, cudaStreamSynchronize((cudaStream_t)stream));
  return take_device_status(c);
}

// ------------------------------------------------------------ host-pointer entry points
extern "C" int qk_dequant_block(qk_ctx *c, int type, const uint8_t *block, size_t block_len,
                                float *out, size_t out_len) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  size_t bs = qk_block_size(type), bb = qk_block_bytes(type);
  if (block_len < bb) return QK_BUFFER_TOO_SMALL;
  if (out_len < bs) return QK_BUFFER_TOO_SMALL;
  if (!block || !out) return QK_INVALID_ARGUMENT;
  return qk_dequant_matrix(c, type, block, bb, 1, bs, out, bs);
}

extern "C" int qk_dequant_matrix(qk_ctx *c, int type, const uint8_t *w, size_t w_len, size_t n_rows,
                                 size_t n_cols, float *out, size_t out_len) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  if (w_len < need_bytes(type, n_rows, n_cols)) return QK_BUFFER_TOO_SMALL;
  if (out_len < n_rows * n_cols) return QK_BUFFER_TOO_SMALL;
  if (n_rows * n_cols == 0) return QK_OK;
  if (!w || !out) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  CK(c, cudaSetDevice(c->device));
  qk_weights *h = nullptr;
  int st = upload_impl(c, type, w, n_cols, 0, n_rows, &h);  // not cached: one-shot
  if (st) return st;
  size_t nbytes = n_rows * n_cols * sizeof(float);
  st = grow(c, &c->sb, &c->sb_cap, nbytes);
  if (st == QK_OK) {
    cudaError_t e = qk_launch_dequant(h->L, h->dev, (float *)c->sb, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, c->sb, nbytes, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
      c->err = std::string("dequant: ") + cudaGetErrorString(e);
      st = QK_CUDA_ERROR;
    }
  }
  free_weights(h);
  return st;
}

static int host_stage(qk_ctx *c) {
  if (c->hx) return QK_OK;
  unsigned char *p = nullptr, *d = nullptr;
  CK(c, cudaHostAlloc((void **)&p, 2 * QK_HOST_STAGE, cudaHostAllocMapped | cudaHostAllocPortable));
  cudaError_t e = cudaHostGetDevicePointer((void **)&d, p, 0);
  if (e != cudaSuccess) {
    cudaFreeHost(p);
    CK(c, e);
  }
  c->hx = p, c->hx_dev = d, c->hy = p + QK_HOST_STAGE, c->hy_dev = d + QK_HOST_STAGE;
  return QK_OK;
}

static int host_gemm(qk_ctx *c, int type, const uint8_t *w, size_t w_len, size_t n, size_t k,
                     const float *x, float *y, size_t m) {
  std::lock_guard<std::mutex> g(c->mu);
  CK(c, cudaSetDevice(c->device));
  qk_weights *h = nullptr;
  int st = cached(c, type, w, w_len, n, k, &h);
  if (st) return st;
  const size_t xb = m * k * sizeof(float), yb = m * n * sizeof(float);
  const bool stage_x = xb <= QK_HOST_STAGE, stage_y = yb <= QK_HOST_STAGE;
  if ((stage_x || stage_y) && (st = host_stage(c))) return st;
  // Decode-sized calls: the kernels that serve M <= 4 split the activations once, before the matvec,
  // straight out of the mapped staging (a copy and its hand-over to the kernel drop out), and store y
  // (a few KB, 32 contiguous bytes per 8-row chunk) straight through the mapping, into the caller's
  // buffer if that is pinned, else into the staging.
  const bool decode = m <= QK_GEMV_MAX_M && k > 0 && !c->force_simple && qk_gemv_fast_supported(h->L, (uint32_t)m);
  float *ydev = nullptr;
  bool direct = false;
  if (decode) {
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, y) == cudaSuccess && pa.type == cudaMemoryTypeHost && pa.devicePointer)
      ydev = (float *)pa.devicePointer, direct = true;
    else
      (void)cudaGetLastError();
    if (!direct && stage_y) ydev = (float *)c->hy_dev;
  }
  if (!ydev) {
    if ((st = grow(c, &c->sb, &c->sb_cap, yb ? yb : 4))) return st;
    ydev = (float *)c->sb;
  }
  if (stage_x) memcpy(c->hx, x, xb);
  if (decode && stage_x) {
    if ((st = qk_ensure_scratch(c, c->host_scratch, qk_gemv_fast_scratch_bytes(h->L, (uint32_t)m)))) return st;
    CK(c, qk_launch_gemv_fast(h->L, h->dev, (const float *)c->hx_dev, ydev, (uint32_t)m, n, c->status_dev,
                              c->host_scratch.p, c->sm_count, c->stream, true));
  } else {
    if ((st = grow(c, &c->sa, &c->sa_cap, xb ? xb : 4))) return st;
    if (xb) CK(c, cudaMemcpyAsync(c->sa, stage_x ? (const void *)c->hx : x, xb, cudaMemcpyHostToDevice, c->stream));
    if ((st = gemm_dispatch(c, c->host_scratch, h, (const float *)c->sa, ydev, m, n, c->stream))) return st;
  }
  const bool from_dev = ydev == (float *)c->sb;
  if (from_dev) CK(c, cudaMemcpyAsync(stage_y ? (void *)c->hy : y, c->sb, yb, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  if (!direct && stage_y) memcpy(y, c->hy, yb);
  return take_device_status(c);  // a bounded wait that ran out leaves y invalid: say so
}

extern "C" int qk_gemv(qk_ctx *c, int type, const uint8_t *w, size_t w_len, size_t n_rows,
                       size_t n_cols, const float *x, size_t x_len, float *y, size_t y_len) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  if (x_len < n_cols) return QK_DIMENSION_MISMATCH;  // order as reference/q4_k.rs:117-128
  if (y_len < n_rows) return QK_DIMENSION_MISMATCH;
  if (w_len < need_bytes(type, n_rows, n_cols)) return QK_BUFFER_TOO_SMALL;
  if (n_rows == 0) return QK_OK;
  if (!w || !y || (n_cols && !x)) return QK_INVALID_ARGUMENT;
  return host_gemm(c, type, w, w_len, n_rows, n_cols, x, y, 1);
}

extern "C" int qk_gemm(qk_ctx *c, int type, const uint8_t *w, size_t w_len, const float *x,
                       size_t x_len, float *y, size_t y_len, size_t m, size_t n, size_t k) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  if (x_len < m * k) return QK_DIMENSION_MISMATCH;
  if (y_len < m * n) return QK_DIMENSION_MISMATCH;
  if (w_len < need_bytes(type, n, k)) return QK_BUFFER_TOO_SMALL;
  if (m == 0 || n == 0) return QK_OK;
  if (!w || !y || (k && !x)) return QK_INVALID_ARGUMENT;
  return host_gemm(c, type, w, w_len, n, k, x, y, m);
}

// ------------------------------------------------------------ GpuKernel-shaped entry points
// crates/oxillama-gpu/src/kernels/mod.rs:91-106 (e.g. kernels/q4_k.rs:170-195): raw weight
// bytes and dimensions instead of a QuantTensor; checks in that implementation's order, every
// failed size check being its GpuError::BufferSize { expected, got } (text in qk_last_error).
static int buffer_size(qk_ctx *c, size_t expected, size_t got) {
  c->err = "Buffer size mismatch: expected " + std::to_string(expected) + ", got " + std::to_string(got);
  return QK_BUFFER_TOO_SMALL;
}

extern "C" int qk_gpu_gemv(qk_ctx *c, int type, const uint8_t *weight_bytes, size_t weight_len,
                           const float *input, size_t input_len, float *output, size_t output_len,
                           size_t rows, size_t cols) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) {
    c->err = "Unsupported quant type for GPU: type id " + std::to_string(type);
    return QK_UNSUPPORTED_TYPE;
  }
  if (output_len < rows) return buffer_size(c, rows, output_len);
  if (input_len < cols) return buffer_size(c, cols, input_len);
  if (weight_len < need_bytes(type, rows, cols)) return buffer_size(c, need_bytes(type, rows, cols), weight_len);
  if (rows == 0) return QK_OK;
  if (!weight_bytes && need_bytes(type, rows, cols)) return QK_INVALID_ARGUMENT;
  if (!output || (cols && !input)) return QK_INVALID_ARGUMENT;
  return host_gemm(c, type, weight_bytes, weight_len, rows, cols, input, output, 1);
}

// Y[b][r] = sum_c A[r][c] X[b][c]: kernels/batched_gemv.rs:36-50 with the matrix still
// quantised (that function takes it dequantised to f32; its callers dequantise first).
extern "C" int qk_gpu_gemv_batched(qk_ctx *c, int type, const uint8_t *weight_bytes, size_t weight_len,
                                   const float *vectors, size_t vectors_len, float *output, size_t output_len,
                                   size_t rows, size_t cols, size_t batch_size) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) {
    c->err = "Unsupported quant type for GPU: type id " + std::to_string(type);
    return QK_UNSUPPORTED_TYPE;
  }
  if (weight_len < need_bytes(type, rows, cols)) return buffer_size(c, need_bytes(type, rows, cols), weight_len);
  if (vectors_len != batch_size * cols) return buffer_size(c, batch_size * cols, vectors_len);  // exact, as there
  if (output_len < batch_size * rows) return buffer_size(c, batch_size * rows, output_len);
  if (rows == 0 || batch_size == 0) return QK_OK;
  if (!output) return QK_INVALID_ARGUMENT;
  if (cols == 0) {  // batched_gemv.rs:88-90: zeros
    memset(output, 0, batch_size * rows * sizeof(float));
    return QK_OK;
  }
  if (!weight_bytes || !vectors) return QK_INVALID_ARGUMENT;
  return host_gemm(c, type, weight_bytes, weight_len, rows, cols, vectors, output, batch_size);
}

extern "C" int qk_matvec_q8_fused(qk_ctx *c, int type, const uint8_t *w, size_t w_len,
                                  const uint8_t *acts_q8, size_t acts_len, float *out,
                                  size_t out_len, size_t n_rows, size_t n_cols) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (!type_ok(type)) return QK_UNSUPPORTED_TYPE;
  if (out_len < n_rows) return QK_DIMENSION_MISMATCH;  // order as reference/q4_k.rs:226-250
  size_t bs = qk_block_size(type);
  size_t acts_needed = ((n_cols + bs - 1) / bs) * (bs / 32) * 34;
  if (w_len < need_bytes(type, n_rows, n_cols)) return QK_BUFFER_TOO_SMALL;
  if (acts_len < acts_needed) return QK_BUFFER_TOO_SMALL;
  if (n_rows == 0 || n_cols == 0) return QK_OK;
  if (!w || !acts_q8 || !out) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  CK(c, cudaSetDevice(c->device));
  qk_weights *h = nullptr;
  int st = cached(c, type, w, w_len, n_rows, n_cols, &h);
  if (st) return st;
  if ((st = grow(c, &c->sa, &c->sa_cap, acts_needed))) return st;
  if ((st = grow(c, &c->sb, &c->sb_cap, n_rows * sizeof(float)))) return st;
  CK(c, cudaMemcpyAsync(c->sa, acts_q8, acts_needed, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->sb, out, n_rows * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  CK(c, qk_launch_fused_simple(h->L, h->dev, (const uint8_t *)c->sa, (float *)c->sb, c->stream));
  CK(c, cudaMemcpyAsync(out, c->sb, n_rows * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return QK_OK;
}

extern "C" int qk_quantize_q8_0(qk_ctx *c, const float *x, size_t n, uint8_t *out, size_t out_len) {
  if (!c) return QK_INVALID_ARGUMENT;
  if (n % 32 != 0) return QK_DIMENSION_MISMATCH;  // quantize.rs:59-64
  if (out_len < n / 32 * 34) return QK_BUFFER_TOO_SMALL;
  if (n == 0) return QK_OK;
  if (!x || !out) return QK_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(c->mu);
  CK(c, cudaSetDevice(c->device));
  int st;
  if ((st = grow(c, &c->sa, &c->sa_cap, n * sizeof(float)))) return st;
  if ((st = grow(c, &c->sb, &c->sb_cap, n / 32 * 34))) return st;
  CK(c, cudaMemcpyAsync(c->sa, x, n * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  CK(c, qk_launch_quantize_q8_0((const float *)c->sa, n, (uint8_t *)c->sb, c->stream));
  CK(c, cudaMemcpyAsync(out, c->sb, n / 32 * 34, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return QK_OK;
}

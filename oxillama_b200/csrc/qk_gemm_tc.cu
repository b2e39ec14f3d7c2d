// Host side of the tensor-core matmul (qk_gemm_tc.cuh): tensor maps, the choice of tiles, the
// per-format dispatch.
#include "qk_gemm_tc.cuh"

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

bool fmt_ok(int t) {
  return t == QK_T_Q4_K || t == QK_T_Q8_0 || t == QK_T_Q4_0 || t == QK_T_Q6_K || t == QK_T_IQ4_XS;
}

}  // namespace

namespace qktc {

// Shared memory for accumulator halves of `hn` tokens.  The weight ring has an even number of stages:
// a stage then always belongs to the same set of expanding warps, which is never more than one phase
// ahead of its barrier (with an odd number a set could find the barrier of a stage that the other set
// has not been given yet, two phases back, and take that for its own).  Narrow tiles are bound by the
// weight stream and give it what they can; tiles of more than 128 tokens need four activation stages first (a
// stage is refilled only after the MMAs that read it have retired).
static bool plan_smem(uint32_t bn, uint32_t hn, uint32_t cg, uint32_t cs, uint32_t w_stage, uint32_t lut, TcSmem *S, uint32_t *total) {
  TcSmem s;
  uint32_t off = 0;
  s.w_full = off, off += MAX_WST * 8;
  s.w_empty = off, off += MAX_WST * 8;
  s.b_full = off, off += MAX_BST * 8;
  s.b_empty = off, off += MAX_BST * 8;
  s.a_full = off, off += 24;
  s.a_empty = off, off += 24;
  s.d_full = off, off += 16;
  s.d_empty = off, off += 16;
  s.drain = off, off += 8;
  s.tmem_slot = off, off += 8;
  s.pre = off, off += (QK_MAX_GROUPS + 1) * 4;
  s.sched = off, off += (uint32_t)sizeof(Sched);
  off = (off + 15u) & ~15u;
  s.scales = off, off += 4 * 512 + 16;  // a copy of a half's token scales per epilogue warp, and one word
  if (off > LUT_OFF) return false;
  off = LUT_OFF + lut;
  s.red = off, off += cs > 1 ? cs * ((hn + cs - 1) / cs) * BM * 4 : 0;  // the cluster's partial sums of this CTA's tokens
  off = (off + 1023u) & ~1023u;
  s.w_stage = w_stage, s.b_stage = (hn / cg) * 512u;  // this CTA's tokens, a super-block's four steps
  const uint32_t room = SMEM_BUDGET - off;
  auto fits = [&](uint32_t w, uint32_t b) { return w * s.w_stage + b * s.b_stage <= room; };
  if (!fits(2, 2)) return false;
  uint32_t nb = 2, nw = 2;
  const uint32_t enough = bn <= 128 ? 3u : 4u;
  while (nb < enough && fits(bn <= 128 ? 4 : 2, nb + 1)) nb++;
  while (nw < (uint32_t)MAX_WST && fits(nw + 2, nb)) nw += 2;
  while (nb < (uint32_t)MAX_BST && hn > 64 && fits(nw, nb + 1)) nb++;
  s.b_stages = nb, s.w_stages = nw;
  s.b = off, off += nb * s.b_stage;  // 1024-byte aligned: the swizzle repeats every 8 rows of 128 bytes
  s.w = off, off += nw * s.w_stage;
  *S = s, *total = off;
  return true;
}

static uint32_t round_up(uint32_t v, uint32_t to) { return (v + to - 1) / to * to; }

// Form of the kernel, token-tile width and K split by predicted time: cycles of the slowest CTA.  The constants are a
// fit to 96 shapes (256 x 12288 .. 28672 x 4096, 8 .. 2048 tokens, Q4_K, Q6_K, Q8_0, IQ4_XS), each timed with every tile
// width and split; the expansion's (one for all but Q6_K), the cluster's and the one for Q8_0 were then fitted to 1076
// calls with the weights from HBM (16 shapes 1024 x 1024 .. 28672 x 4096, 300 x 8192 .. 4096 x 14336, the same tokens and
// formats; rows of gate and up together are such shapes too): the form it picks was 1.1 % slower than the fastest in the
// mean, 19 % at worst.  Q4_K and Q6_K since expand faster (WFmt): with 870 and 1130 for 1000 and 1170 the 315 and 52 calls of
// another sweep (15 and 4 shapes, 5 .. 1024 tokens) take 0.995 and 0.997 of the time in the mean (8192 x 4096 by 8 to 24
// 13.4 -> 10.7 us; 5120 x 5120 by 80 15.4 -> 16.3); 900 and 930 gained less.  A super-block takes as long as its expansion or its MMAs, or in a pair the
// round of hand-overs (expanding warps -> issuer -> tensor pipe -> back).  A tile whose partials go through the
// workspace costs some 7000 cycles and 40 per token (writing them out, the fence, the counter, reading them back);
// through the cluster 4300 and 17 per token (with 4600 for any width IQ4_XS 2048 x 2048 by 64 took 9.5 us in clusters, 8.1
// without).  4200 for Q6_K: with 4300, and super-blocks that expand faster, its rows of six by up to 16 tokens went to a CTA a tile
// (1536 x 1536 by 8 6.66 us, in clusters 6.15; no other of 400 shapes changes).
bool make_plan(const QkTcCall &c, int sm_count, TcPlan *P) {
  const QkLayout &L = *c.L;
  const uint32_t w_stage = 16u * 8u * L.bb * (256u / L.bs), lut = L.type == QK_T_IQ4_XS ? WFmt<QK_T_IQ4_XS>::LUT : 0u;
  TcPlan p;
  p.nsb = (L.cols + 255u) / 256u, p.cs = 1;
  auto half_of = [&](uint32_t bn) { return bn <= 128 ? bn : round_up((bn + 1) / 2, 16); };
  if (c.counts) {
    // Counts on the device: tiles wide enough for a group somewhat above the average, so that most
    // groups take one (the MMA covers only a tile's live tokens, rounded up to 16).
    uint32_t bn = round_up(c.expect + c.expect / 2, 32);
    const uint32_t all = round_up(c.m, 32);
    if (bn > all) bn = all;
    if (bn > 128) bn = MAX_BN;  // two whole halves
    p.cg = bn <= 64 ? 1 : 2;
    p.bn = bn, p.min_run = 4;
    p.tok_blocks = (c.m + bn - 1) / bn;
    p.row_blocks = (L.rows + p.cg * BM - 1) / (p.cg * BM);
    p.grid = (uint32_t)sm_count / p.cg;
  } else {
    // (with a marked matrix as before)
    const float expand = L.type == QK_T_Q6_K ? (c.wide ? 1170.f : 1130.f) : L.type == QK_T_Q4_K && !c.wide ? 870.f : 1000.f;
    float best = FLT_MAX;
    auto take = [&](float t, uint32_t cg, uint32_t cs, uint32_t bn, uint32_t tbr, uint32_t rbs, uint32_t run, uint32_t grid) {
      if (t < best) best = t, p.cg = cg, p.cs = cs, p.bn = bn, p.tok_blocks = tbr, p.row_blocks = rbs, p.min_run = run, p.grid = grid;
    };
    const uint32_t tb0 = (c.m + MAX_BN - 1) / MAX_BN;
    // Every token block reads the weights again, from L2 at best: 1.5 % for twice as many blocks as needed.  (Three blocks
    // instead of two can still be the faster form, from HBM too: Q4_K 28672 x 4096 by 512 108 against 120 us, 112 row
    // blocks being 3.03 rounds of 74 pairs in two and 4.54 in three; 14336 x 4096 by 512 65.5 against 59.4.)
    // (A pair only where its second CTA has rows: Q4_0 64 x 1280 by 2048 tokens 26.4 -> 14.0 us.)
    for (uint32_t cg = 1; cg <= (L.rows > BM ? 2u : 1u); cg++) {
      const uint32_t units = (uint32_t)sm_count / cg, rbs = (L.rows + cg * BM - 1) / (cg * BM);
      for (uint32_t k = 0; k < 10; k++) {
        const uint32_t tb = tb0 << (k >> 1), tbk = (k & 1) ? tb + (tb + 1) / 2 : tb;  // 1, 1.5, 2, 3, 4, 6, .. times the fewest
        const uint32_t bn = round_up((c.m + tbk - 1) / tbk, 16);
        if (k && bn < 32) break;
        if (cg == 1 && bn > 64) continue;
        const uint32_t tbr = (c.m + bn - 1) / bn;
        float sb = cg == 1 ? expand : fmaxf(fmaxf(expand + 125.f, 980.f + 2.f * bn), 9.f * bn);
        const float out = bn * 59.f;
        // Beside Q8_0's four stages of weights there is room for two of such a tile's activations (plan_smem): 4096 x
        // 14336 by 512 76.6 us in tiles of 128, 71.2 of 176.
        if (L.type == QK_T_Q8_0 && bn > 112 && bn <= 128) sb += 60.f;
        const uint64_t tiles = (uint64_t)c.n * rbs * tbr;
        for (uint32_t run = 1; run <= 16; run <<= 1) {
          const uint32_t R = (uint32_t)(tiles % units), total = R * p.nsb;
          float t = (float)(tiles / units) * (p.nsb * sb + (bn > 128 ? 9000.f : 70.f + 38.f * bn)) + out;
          uint32_t grid = units;
          if (R) {
            uint32_t sk = total / run;
            sk = sk < 1 ? 1 : sk > units ? units : sk;
            if (tiles < units) {
              if (sk < R) sk = R;
              grid = sk;
            }
            const float len = (float)((total + sk - 1) / sk), contrib = (float)sk / R;
            t += len * sb;
            if (contrib > 1.01f) t += 7200.f + bn * (36.f + 3.5f * contrib);
          }
          if (tb0 > 1) t *= 1.f + 0.015f * log2f((float)tbr / tb0);
          take(t, cg, 1, bn, tbr, rbs, run, grid);
        }
        // One tile per cluster of cs CTAs.  At most as many as fit at a time: 32 clusters of four, 14 of eight on
        // 148 SMs (1024 x 4096 by 37: 8.5 us as 8 clusters of eight, 12.8 as 16).  Clusters of two are never the fastest.
        if (cg == 1 && c.n == 1)
          for (uint32_t cs = 4; cs <= 8 && cs <= p.nsb; cs <<= 1)
            if (tiles * cs <= (uint32_t)sm_count * (cs == 4 ? 14u : 12u) / 16u)
              take((float)((p.nsb + cs - 1) / cs) * sb + (L.type == QK_T_Q6_K ? 4200.f : 4300.f) + 17.f * bn + out, 1, cs, bn, tbr, rbs, 1, (uint32_t)tiles * cs);
      }
    }
  }
  p.hn = half_of(p.bn);
  if (!plan_smem(p.bn, p.hn, p.cg, p.cs, w_stage, lut, &p.S, &p.smem)) return false;
  // The rows that the MMAs cover, whatever the tiles: a wider box of the last token block ends outside the tensor map,
  // and the copy unit fills it with zeros (381 calls whose tiles cover more rows, timed both ways: no difference).
  p.xrows = c.counts || c.n_act > 1 ? c.n_act * c.xcap : round_up(c.m, 16);
  const size_t Kp = (size_t)p.nsb * 256u;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  p.o_scale = al((size_t)p.xrows * Kp * 2);
  p.o_cnt = al(p.o_scale + (size_t)(p.xrows + MAX_BN) * 4);
  p.o_part = al(p.o_cnt + (size_t)sm_count * 2 * 4);
  p.grid *= p.cg;
  p.bytes = p.o_part + qk_gemm_tc_part_bytes(sm_count);  // (whatever this plan uses of them)
  *P = p;
  return true;
}

// The fp16 activations [xrows][Kp] as boxes [4 steps][rows][64 columns]: a box lands as four swizzled
// operand tiles.
bool x_map(CUtensorMap *m, __half *x16, uint32_t xrows, uint32_t Kp, uint32_t rows) {
  EncodeTiledFn enc = encode_fn();
  cuuint64_t dims[3] = {64, xrows, Kp / 64};
  cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, 128};
  cuuint32_t box[3] = {64, rows, 4};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc && enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, x16, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace qktc

bool qk_gemm_tc_supported(const QkLayout &L, uint32_t m) { return fmt_ok(L.type) && m >= 1 && L.rows >= 1 && L.nb >= 1; }

// Zeroed chunks behind the matrix that fill up its last box of 128 rows.  A box that ends outside the matrix is slow
// when many CTAs fetch it at a time (Q8_0 8 x 1280 by 2048 tokens: 37.5 us with the rows filled in by the copy unit,
// 16.6 with zeros in memory).  Where K is so long that they would be many bytes the copy unit fills them in.
uint64_t qk_gemm_tc_pad_bytes(const QkLayout &L) {
  if (!qk_gemm_tc_supported(L, 1)) return 0;
  const uint64_t pad = (16 - L.chunks % 16) % 16 * L.chunk_bytes;
  return pad <= (16ull << 20) ? pad : 0;
}

cudaError_t qk_gemm_tc_map(const QkLayout &L, uint8_t *tiled, void *map) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  // [chunks][blocks of a row][8 rows of one block, as 64-bit words]
  cuuint64_t dims[3] = {L.bb, L.nb, L.chunks + qk_gemm_tc_pad_bytes(L) / L.chunk_bytes};
  cuuint64_t strides[2] = {8ull * L.bb, L.chunk_bytes};
  cuuint32_t box[3] = {L.bb, 256u / L.bs, 16};
  cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap m;
  if (enc(&m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, tiled, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  memcpy(map, &m, sizeof(m));
  return cudaSuccess;
}

// (four bytes a row, and the mark)
size_t qk_gemm_tc_factor_bytes(const QkLayout &L) {
  return L.chunks && (L.type == QK_T_Q4_K || L.type == QK_T_Q6_K) ? (size_t)L.chunks * QK_TILE_ROWS * sizeof(float) + 16 : 0;
}

namespace {
__device__ __forceinline__ uint32_t max_byte(uint32_t v) {
  v = __vmaxu4(v, v >> 16);
  return max(v & 0xFFu, (v >> 8) & 0xFFu);
}
__device__ __forceinline__ float abs_half(uint32_t bits) { return fabsf(__half2float(__ushort_as_half((unsigned short)bits))); }

// The power of two over which 2^24 b is at most 0.998 of 2^16, about fp16's largest (2^-6 at least: 2^30 is what the kernel takes)
__device__ __forceinline__ float factor_over(float b) {
  int e = 0;
  const float f = frexpf(b, &e);  // b = f * 2^e, f in [0.5, 1)
  return b > 0.f ? ldexpf(1.f, max(e + 8 + (f > 0.998f ? 1 : 0), -6)) : 1.f;
}

// A warp per row.  Its factor is that of the largest scale that its blocks can have by their d (Q4_K: 63 |d|, |dmin|; Q6_K: 128
// |d|), which keeps the results of such matrices, bit for bit, what they are for any sub-scales; where that is more than 8 times the
// factor of the largest scale in use (|d sc|, |d|, |dmin|; Q6_K: |d sc|, |d|), or with `in_use`, the latter.  Scales that are not
// finite do not count (their blocks stay not finite), a row of zeros has factor 1.  `mark` is set where what a block of the row
// reaches is below 2^-10 of the factor in use or 2^-12 of its own (see WFmt): 63 * 15 d of Q4_K (6-bit scales are made with the
// largest of a block 63; if all are 0, 63 dmin), 32 |d sc| of Q6_K.
__global__ void __launch_bounds__(256) qk_row_factor_kernel(QkLayout L, const uint8_t *__restrict__ tiled, float *__restrict__ rows, unsigned *__restrict__ mark, bool in_use) {
  const uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= L.chunks * QK_TILE_ROWS) return;
  float b = 0.f, top = 0.f, least = FLT_MAX;
  if (row < L.rows)
    for (uint32_t k = lane; k < L.nb; k += 32) {
      if (L.type == QK_T_Q4_K) {
        const uint4 h = *reinterpret_cast<const uint4 *>(tiled + qk_byte_offset(L, row, k, 0, 0));
        const uint32_t sc = max_byte(__vmaxu4(h.y & 0x3F3F3F3Fu, (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u)));
        const uint32_t mn = max_byte(__vmaxu4(h.z & 0x3F3F3F3Fu, ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u)));
        const float d = abs_half(h.x), dmin = abs_half(h.x >> 16);
        if (d <= FLT_MAX) b = fmaxf(b, d * (float)max(sc, 1u)), top = fmaxf(top, 63.f * d);
        if (dmin <= FLT_MAX) b = fmaxf(b, dmin), top = fmaxf(top, dmin);
        if (sc && d > 0.f && d <= FLT_MAX) least = fminf(least, 945.f * d);
        else if (mn && dmin > 0.f && dmin <= FLT_MAX) least = fminf(least, 63.f * dmin);
      } else {
        const uint4 s = *reinterpret_cast<const uint4 *>(tiled + qk_byte_offset(L, row, k, 1, 0));
        const uint32_t sc = max_byte(__vmaxu4(__vmaxu4(__vabs4(s.x), __vabs4(s.y)), __vmaxu4(__vabs4(s.z), __vabs4(s.w))));
        const float d = abs_half(*reinterpret_cast<const uint16_t *>(tiled + qk_byte_offset(L, row, k, 2, 0)));
        if (d <= FLT_MAX) b = fmaxf(b, d * (float)max(sc, 1u)), top = fmaxf(top, 128.f * d);
        if (sc && d > 0.f && d <= FLT_MAX) least = fminf(least, 32.f * d * (float)sc);
      }
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o)), top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
  }
  if (lane == 0) {
    const float used = factor_over(b), by_d = factor_over(top), factor = in_use || by_d > 8.f * used ? used : by_d;
    rows[row] = factor;
    if (least < fmaxf(used * 0x1p-10f, factor * 0x1p-12f)) atomicOr(mark, 1u);
  }
}
}  // namespace

cudaError_t qk_gemm_tc_factors(const QkLayout &L, const uint8_t *tiled, float *rows, bool *wide, cudaStream_t s) {
  *wide = false;
  if (!qk_gemm_tc_factor_bytes(L)) return cudaSuccess;
  unsigned *mark = reinterpret_cast<unsigned *>(rows + (size_t)L.chunks * QK_TILE_ROWS), m = 0;
  cudaError_t e = cudaMemsetAsync(mark, 0, sizeof(m), s);
  if (e != cudaSuccess) return e;
  qk_row_factor_kernel<<<L.chunks, 256, 0, s>>>(L, tiled, rows, mark, false);
  if ((e = cudaGetLastError()) == cudaSuccess) e = cudaMemcpyAsync(&m, mark, sizeof(m), cudaMemcpyDeviceToHost, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess && m) {  // (the other expansion reaches 2^16 down from the largest scale in use)
    qk_row_factor_kernel<<<L.chunks, 256, 0, s>>>(L, tiled, rows, mark, true);
    e = cudaGetLastError(), e2 = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = e2;
  }
  *wide = e == cudaSuccess && m != 0;
  return e;
}

size_t qk_gemm_tc_part_bytes(int sm_count) { return (size_t)sm_count * 2 * qktc::MAX_BN * qktc::BM * 4; }

size_t qk_gemm_tc_scratch_bytes(const QkTcCall &c, int sm_count) {
  qktc::TcPlan P;
  return qktc::make_plan(c, sm_count, &P) ? P.bytes : 0;
}

#define QK_TC_DECLARE(NAME) \
  cudaError_t qk_tc_##NAME##_launch(const QkTcCall &c, unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s);
QK_TC_DECLARE(q4k)
QK_TC_DECLARE(q80)
QK_TC_DECLARE(q40)
QK_TC_DECLARE(q6k)
QK_TC_DECLARE(iq4xs)

cudaError_t qk_launch_gemm_tc(const QkTcCall &c, unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s) {
  if (c.n == 0 || c.n > QK_MAX_GROUPS || c.n_act == 0 || c.n % c.n_act || c.m == 0 || !qk_gemm_tc_supported(*c.L, 1))
    return cudaErrorInvalidValue;
  switch (c.L->type) {
    case QK_T_Q4_K:
      return qk_tc_q4k_launch(c, status, scratch, sm_count, s);
    case QK_T_Q8_0:
      return qk_tc_q80_launch(c, status, scratch, sm_count, s);
    case QK_T_Q4_0:
      return qk_tc_q40_launch(c, status, scratch, sm_count, s);
    case QK_T_Q6_K:
      return qk_tc_q6k_launch(c, status, scratch, sm_count, s);
    case QK_T_IQ4_XS:
      return qk_tc_iq4xs_launch(c, status, scratch, sm_count, s);
    default:
      return cudaErrorInvalidValue;
  }
}

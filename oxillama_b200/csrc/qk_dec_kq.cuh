// Q5_K, Q3_K and Q2_K policies of the decode kernel (qk_gemv_skel.cuh).
//
//   Q5_K  the Q4_K super-block with a fifth bit per weight: k = 32 of the MMA is one sub-block; A
//         rows 0-7 = the eight weight rows of sub-block 2p (5-bit values), rows 8-15 = the same rows
//         of sub-block 2p + 1, as in the Q8_0 policy.
//   Q3_K, Q2_K  16-column scales, so the two groups of an MMA are the two 16-column strips of one
//         32-column block, as in the Q6_K policy.  Six and four words per lane hold a 256-column
//         span: a word of 2-bit fields serves the four 32-column blocks of its 128-column half.
//
// Their generic kernel decoded every weight byte by byte from global memory (14336 x 4096 Q5_K at one
// row: 570 us); here they stream at the rate of the tuned formats.
//
// A 256-column span of a tile, 8 rows, block-major:
//   Q5_K  [8 rows x 16 header | 8 rows x 32 qh | 4 groups x 8 rows x 32 nibble bytes]        = 1408
//   Q3_K  [2 x 8 rows x 16 hmask | 4 x 8 rows x 16 qs | 3 x 8 rows x 4 scales | 8 x f16 d]   = 880
//   Q2_K  [8 rows x 16 scales | 4 x 8 rows x 16 qs | 8 rows x (f16 d, f16 dmin)]             = 672
#pragma once
#include "qk_dec_fmts.cuh"

namespace qkdec {

// ---------------------------------------------------------------------------- Q5_K
// reference/q5_k.rs:66-108: low nibbles of group g = sub-block 2 g with bit g of qh[l] on top, high
// nibbles = sub-block 2 g + 1 with bit g + 4.
struct DecQ5K {
  static constexpr uint32_t COLB = 1408, XSB = 8;
  static constexpr int MAX_M = 4;
  static constexpr bool HAS_DUAL = true, HAS_PEER = false;
  static constexpr bool ANY_DEPTH = false;  // ring depths that are no multiple of the groups (ring_is_deep)
  static constexpr uint32_t PAIR_COLS = 12288;  // fewest columns of which a pair of CTAs takes half each (pair_pays)
  static constexpr bool PAIR_FULL = true;  // pairs also where every one has a single chunk (pair_pays)
  static constexpr uint32_t BY_TILE_M = 4;  // most rows with which the stages of long chunks are handed back one by one
  static constexpr uint32_t SHORT_M = 1u << 3;  // rows (bit m) with which matrices of a single k-tile have a kernel of their own (launch_mma)
  static constexpr bool OWN_SPLIT = true;  // any number of rows may have to be split by every CTA itself (no scratch in a capture)
  static constexpr uint32_t XCH = 0;       // shared memory per compute warp for what its lanes exchange
  static constexpr bool HAS_ONE = false;   // a variant of the policy for one row
  __device__ static __forceinline__ void store_digits(unsigned char *row_img, uint32_t PS, uint32_t e0, uint32_t w0,
                                                      uint32_t w1, uint32_t w2) {
    store_digits_natural(row_img, PS, e0, w0, w1, w2);
  }
  __device__ static __forceinline__ void store_xs(unsigned char *tab, size_t blk, float sx, float s32, float, float) {
    *reinterpret_cast<float2 *>(tab + blk * 8) = make_float2(sx, s32);
  }
  template <int M>
  struct Data {
    uint4 h;
    uint2 qh, w[4];
    float4 xs[M];
    uint2 b[M][4];
  };
  struct Lane : LaneCommon {
    bool hi_half;
    uint32_t m1, m2, sel0, sel1, hl, ql;
    __device__ __forceinline__ void init(uint32_t lane, uint32_t wl, uint32_t ximg, uint32_t PS, uint32_t xs_off,
                                         uint32_t Kp) {
      init_common(lane, wl, ximg, PS, xs_off, Kp);
      const uint32_t g = lane >> 2, tig = lane & 3;
      hi_half = tig >= 2;  // the lane unpacks sub-blocks 2 tig, 2 tig + 1 of the header
      m1 = hi_half ? 0x0F0F0F0Fu : 0x3F3F3F3Fu, m2 = hi_half ? 0x30303030u : 0u;
      sel0 = 0x7540u | (2u * (tig & 1u)), sel1 = sel0 + 1u;
      hl = wl * COLB + g * 16, ql = wl * COLB + 128 + g * 32 + tig * 8;
    }
  };
  struct Base {
    uint32_t h, q, x, xs;
  };
  __device__ static __forceinline__ Base base(const Lane &LN, uint32_t tile, uint32_t kt) {
    return {tile + LN.hl, tile + LN.ql, LN.xl + kt * (QK_TILE_ELEMS / 32) * 32, LN.xsl + kt * (QK_TILE_ELEMS / 32) * 8};
  }
  template <int M, int J, int WG>
  __device__ static __forceinline__ void load(Data<M> &D, const Base &B, const Lane &LN) {
    D.h = lds128o<J * WG * (int)COLB>(B.h);
    D.qh = lds64o<J * WG * (int)COLB>(B.q);
    static_for<0, 4>([&](auto gq) { D.w[decltype(gq)::value] = lds64o<J * WG * (int)COLB + 256 + decltype(gq)::value * 256>(B.q); });
    load_x_common<M, J, WG>(D, B, LN);
  }
  template <int M>
  __device__ static __forceinline__ void compute(const Data<M> &D, const Lane &LN, float (&acc)[M][3]) {
    const uint4 h = D.h;  // d, dmin, 6-bit scales and mins: as Q4_K
    const float d = h2f_bits(h.x), dmin = h2f_bits(h.x >> 16);
    const uint32_t scw = ((LN.hi_half ? h.w : h.y) & LN.m1) | ((h.y >> 2) & LN.m2);
    const uint32_t mnw = ((LN.hi_half ? (h.w >> 4) : h.z) & LN.m1) | ((h.z >> 2) & LN.m2);
    const float ds0 = d * (__int_as_float(__byte_perm(scw, 0x4B000000u, LN.sel0)) - 8388608.f);
    const float ds1 = d * (__int_as_float(__byte_perm(scw, 0x4B000000u, LN.sel1)) - 8388608.f);
    const float dm0 = dmin * (__int_as_float(__byte_perm(mnw, 0x4B000000u, LN.sel0)) - 8388608.f);
    const float dm1 = dmin * (__int_as_float(__byte_perm(mnw, 0x4B000000u, LN.sel1)) - 8388608.f);
    uint32_t a[4][4];
#pragma unroll
    for (int g = 0; g < 4; g++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint32_t w = i ? D.w[g].y : D.w[g].x, q = i ? D.qh.y : D.qh.x;
        const uint32_t hi = g == 0 ? q : q >> g;  // bit g + 4 of every byte at bit 4
        a[g][2 * i] = (w & 0x0F0F0F0Fu) | ((q << (4 - g)) & 0x10101010u);
        a[g][2 * i + 1] = ((w >> 4) & 0x0F0F0F0Fu) | (hi & 0x10101010u);
      }
#pragma unroll
    for (int m = 0; m < M; m++) {
      const float tx = ds0 * D.xs[m].x, ty = ds1 * D.xs[m].z;
      acc[m][2] = fmaf(dm0, D.xs[m].y, acc[m][2]);
      acc[m][2] = fmaf(dm1, D.xs[m].w, acc[m][2]);
      float c[4][4];
#pragma unroll
      for (int gq = 0; gq < 4; gq++)
        mma_u8s8(c[gq], a[gq][0], a[gq][1], a[gq][2], a[gq][3], D.b[m][gq].x, D.b[m][gq].y);
#pragma unroll
      for (int gq = 0; gq < 4; gq++) {
        acc[m][0] = fmaf(__shfl_sync(0xffffffffu, tx, gq, 4), c[gq][0] - MMA_BIAS, acc[m][0]);
        acc[m][1] = fmaf(__shfl_sync(0xffffffffu, ty, gq, 4), c[gq][3] - MMA_BIAS, acc[m][1]);
      }
    }
  }
  __device__ static __forceinline__ float finish(const float (&a)[3], const Lane &LN) {
    return LN.kD * (a[0] + a[1]) - a[2];
  }
};

// ---------------------------------------------------------------------------- 16-column scales
// What Q3_K and Q2_K share: digits of the strips (as in the Q6_K policy), the MMAs, the scaling.
struct LaneStrips {
  float kD;
  uint32_t xl, xsl, xm, xsm, m0, m1;
  __device__ __forceinline__ void init_strips(uint32_t lane, uint32_t wl, uint32_t ximg, uint32_t PS, uint32_t xs_off,
                                              uint32_t Kp) {
    const uint32_t g = lane >> 2, tig = lane & 3;
    kD = digit_weight(tig);
    // B column g: digit g / 2 of strip g & 1 (columns 6, 7 unused): four bytes of the natural-order plane
    xl = ximg + (g < 6 ? (g >> 1) : 2u) * PS + (g & 1u) * 16u + tig * 4 + wl * 256;
    xsl = ximg + xs_off + (wl * 8 + 2 * tig) * 16;
    xm = 3 * PS, xsm = (Kp / 32) * 16;
    m0 = (g & 1u) ? 0u : 0xFFFFFFFFu, m1 = ~m0;  // an even column is zero in k-slots 16-31, an odd one in 0-15
  }
};
template <int M, int J, int WG, class D, class B, class LN>
__device__ __forceinline__ void load_x_strips(D &d, const B &b, const LN &ln) {
#pragma unroll
  for (int m = 0; m < M; m++) {
    d.xs[m][0] = lds128fo<J * WG * 128>(b.xs + m * ln.xsm);
    d.xs[m][1] = lds128fo<J * WG * 128 + 16>(b.xs + m * ln.xsm);
    const uint32_t xb = b.x + m * ln.xm;
    static_for<0, 8>([&](auto iq) { d.b[m][decltype(iq)::value] = lds32o<J * WG * 256 + decltype(iq)::value * 32>(xb); });
  }
}
// a[4 G + k][strip]: the A fragments; ds: the lane's four scales, index 4 tig + j = 8 G + 2 k + strip
// with G = tig / 2, k = 2 (tig & 1) + j / 2; off: what comes off per unit of the strip's sum of x.
template <int M, class D, class LN>
__device__ __forceinline__ void mma_strips(const D &d, const LN &ln, const uint32_t (&a)[8][2], const float (&ds)[4],
                                           const float (&off)[4], float (&acc)[M][3]) {
#pragma unroll
  for (int m = 0; m < M; m++) {
    const float4 x0 = d.xs[m][0], x1 = d.xs[m][1];
    const float t[4] = {ds[0] * x0.x, ds[1] * x0.x, ds[2] * x1.x, ds[3] * x1.x};
    float z = off[0] * x0.z;
    z = fmaf(off[1], x0.w, z), z = fmaf(off[2], x1.z, z), z = fmaf(off[3], x1.w, z);
    acc[m][2] += z;
    float c[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++) mma_u8s8(c[i], a[i][0], 0u, a[i][1], 0u, d.b[m][i] & ln.m0, d.b[m][i] & ln.m1);
#pragma unroll
    for (int i = 0; i < 8; i++) {  // block i = 4 G + k: its scales live in lane 2 G + k / 2 of the quad, entries 2 (k & 1), + 1
      acc[m][0] = fmaf(__shfl_sync(0xffffffffu, t[2 * (i & 1)], i >> 1, 4), c[i][0] - MMA_BIAS, acc[m][0]);
      acc[m][1] = fmaf(__shfl_sync(0xffffffffu, t[2 * (i & 1) + 1], i >> 1, 4), c[i][1] - MMA_BIAS, acc[m][1]);
    }
  }
}

// ---------------------------------------------------------------------------- Q3_K
// reference/q3_k.rs:29-59, 79-118.  Element (half G, shift k, strip n, l): column 128 G + 32 k + 16 n + l,
// q = (qs[32 G + 16 n + l] >> 2 k & 3) + 4 (bit 4 G + k of hmask[16 n + l]), value d (sc - 32) (q - 4).
struct DecQ3K {
  static constexpr uint32_t COLB = 880, XSB = 16;
  static constexpr int MAX_M = 2;  // three rows and up spill, as with Q6_K
  static constexpr bool HAS_DUAL = true, HAS_PEER = false;
  static constexpr bool ANY_DEPTH = false;  // ring depths that are no multiple of the groups (ring_is_deep)
  static constexpr uint32_t PAIR_COLS = 11008;  // fewest columns of which a pair of CTAs takes half each (pair_pays)
  static constexpr bool PAIR_FULL = true;  // pairs also where every one has a single chunk (pair_pays)
  static constexpr uint32_t BY_TILE_M = 4;  // most rows with which the stages of long chunks are handed back one by one
  static constexpr uint32_t SHORT_M = 1u << 2;  // rows (bit m) with which matrices of a single k-tile have a kernel of their own (launch_mma)
  static constexpr bool OWN_SPLIT = true;  // any number of rows may have to be split by every CTA itself (no scratch in a capture)
  static constexpr uint32_t XCH = 0;       // shared memory per compute warp for what its lanes exchange
  static constexpr bool HAS_ONE = false;   // a variant of the policy for one row
  __device__ static __forceinline__ void store_digits(unsigned char *row_img, uint32_t PS, uint32_t e0, uint32_t w0,
                                                      uint32_t w1, uint32_t w2) {
    store_digits_natural(row_img, PS, e0, w0, w1, w2);
  }
  __device__ static __forceinline__ void store_xs(unsigned char *tab, size_t blk, float sx, float s32, float s16a,
                                                  float s16b) {
    *reinterpret_cast<float4 *>(tab + blk * 16) = make_float4(sx, s32, s16a, s16b);
  }
  template <int M>
  struct Data {
    uint32_t hm[2], qs[4], s[2], dd;  // qs[2 G + n]; s: scale bytes 0-3 or 4-7 (by the lane), bytes 8-11
    float4 xs[M][2];
    uint32_t b[M][8];
  };
  struct Lane : LaneStrips {
    uint32_t wl0, sl0, sl2, dl, shl, mlo, mhi;
    __device__ __forceinline__ void init(uint32_t lane, uint32_t wl, uint32_t ximg, uint32_t PS, uint32_t xs_off,
                                         uint32_t Kp) {
      init_strips(lane, wl, ximg, PS, xs_off, Kp);
      const uint32_t g = lane >> 2, tig = lane & 3;
      wl0 = wl * COLB + g * 16 + tig * 4;
      sl0 = wl * COLB + 768 + (tig & 1u) * 32 + g * 4, sl2 = wl * COLB + 768 + 64 + g * 4;
      dl = wl * COLB + 864 + 2 * g;
      // scales 0-7: the low six bits of bytes 0-7; 8-15: a nibble of bytes 8-11 under the top two bits of bytes 0-7
      shl = tig == 3 ? 4 : 0, mlo = tig < 2 ? 0x3F3F3F3Fu : 0u, mhi = tig < 2 ? 0u : 0x30303030u;
    }
  };
  struct Base {
    uint32_t w, s, s2, d, x, xs;
  };
  __device__ static __forceinline__ Base base(const Lane &LN, uint32_t tile, uint32_t kt) {
    return {tile + LN.wl0, tile + LN.sl0, tile + LN.sl2, tile + LN.dl, LN.xl + kt * (QK_TILE_ELEMS / 32) * 32,
            LN.xsl + kt * (QK_TILE_ELEMS / 32) * 16};
  }
  template <int M, int J, int WG>
  __device__ static __forceinline__ void load(Data<M> &D, const Base &B, const Lane &LN) {
    constexpr int C0 = J * WG * (int)COLB;
    D.hm[0] = lds32o<C0>(B.w), D.hm[1] = lds32o<C0 + 128>(B.w);
    static_for<0, 4>([&](auto iq) { D.qs[decltype(iq)::value] = lds32o<C0 + 256 + decltype(iq)::value * 128>(B.w); });
    D.s[0] = lds32o<C0>(B.s), D.s[1] = lds32o<C0>(B.s2), D.dd = lds16o<C0>(B.d);
    load_x_strips<M, J, WG>(D, B, LN);
  }
  template <int M>
  __device__ static __forceinline__ void compute(const Data<M> &D, const Lane &LN, float (&acc)[M][3]) {
    const float d = h2f_bits(D.dd);
    const uint32_t sc = (D.s[0] & LN.mlo) | ((D.s[0] >> 2) & LN.mhi) | ((D.s[1] >> LN.shl) & (LN.mhi ? 0x0F0F0F0Fu : 0u));
    float ds[4], off[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      ds[j] = d * (float)((int)((sc >> (8 * j)) & 0xFFu) - 32);
      off[j] = 4.f * ds[j];
    }
    uint32_t a[8][2];
#pragma unroll
    for (int G = 0; G < 2; G++)
#pragma unroll
      for (int k = 0; k < 4; k++)
#pragma unroll
        for (int n = 0; n < 2; n++) {
          const int bit = 4 * G + k;
          const uint32_t hm = bit < 2 ? D.hm[n] << (2 - bit) : D.hm[n] >> (bit - 2);
          a[bit][n] = ((D.qs[2 * G + n] >> (2 * k)) & 0x03030303u) | (hm & 0x04040404u);
        }
    mma_strips<M>(D, LN, a, ds, off, acc);
  }
  __device__ static __forceinline__ float finish(const float (&a)[3], const Lane &LN) {
    return LN.kD * (a[0] + a[1]) - a[2];
  }
};

// ---------------------------------------------------------------------------- Q2_K
// reference/q2_k.rs:42-79: strip is = 8 G + 2 k + n, q = qs[32 G + 16 n + l] >> 2 k & 3, value
// d (s & 15) q - dmin (s >> 4) with s = scales[is].
struct DecQ2K {
  static constexpr uint32_t COLB = 672, XSB = 16;
  static constexpr int MAX_M = 2;  // as Q3_K
  static constexpr bool HAS_DUAL = true, HAS_PEER = false;
  static constexpr bool ANY_DEPTH = false;  // ring depths that are no multiple of the groups (ring_is_deep)
  static constexpr uint32_t PAIR_COLS = 0;  // fewest columns of which a pair of CTAs takes half each (pair_pays)
  static constexpr bool PAIR_FULL = true;  // pairs also where every one has a single chunk (pair_pays)
  static constexpr uint32_t BY_TILE_M = 4;  // most rows with which the stages of long chunks are handed back one by one
  static constexpr uint32_t SHORT_M = 1u << 2;  // rows (bit m) with which matrices of a single k-tile have a kernel of their own (launch_mma)
  static constexpr bool OWN_SPLIT = true;  // any number of rows may have to be split by every CTA itself (no scratch in a capture)
  static constexpr uint32_t XCH = 0;       // shared memory per compute warp for what its lanes exchange
  static constexpr bool HAS_ONE = false;   // a variant of the policy for one row
  __device__ static __forceinline__ void store_digits(unsigned char *row_img, uint32_t PS, uint32_t e0, uint32_t w0,
                                                      uint32_t w1, uint32_t w2) {
    store_digits_natural(row_img, PS, e0, w0, w1, w2);
  }
  __device__ static __forceinline__ void store_xs(unsigned char *tab, size_t blk, float sx, float s32, float s16a,
                                                  float s16b) {
    *reinterpret_cast<float4 *>(tab + blk * 16) = make_float4(sx, s32, s16a, s16b);
  }
  template <int M>
  struct Data {
    uint32_t sc, qs[4], dm;  // scale bytes 4 tig .. + 3; qs[2 G + n]; d | dmin << 16
    float4 xs[M][2];
    uint32_t b[M][8];
  };
  struct Lane : LaneStrips {
    uint32_t wl0, dl;
    __device__ __forceinline__ void init(uint32_t lane, uint32_t wl, uint32_t ximg, uint32_t PS, uint32_t xs_off,
                                         uint32_t Kp) {
      init_strips(lane, wl, ximg, PS, xs_off, Kp);
      const uint32_t g = lane >> 2, tig = lane & 3;
      wl0 = wl * COLB + g * 16 + tig * 4;
      dl = wl * COLB + 640 + 4 * g;
    }
  };
  struct Base {
    uint32_t w, d, x, xs;
  };
  __device__ static __forceinline__ Base base(const Lane &LN, uint32_t tile, uint32_t kt) {
    return {tile + LN.wl0, tile + LN.dl, LN.xl + kt * (QK_TILE_ELEMS / 32) * 32, LN.xsl + kt * (QK_TILE_ELEMS / 32) * 16};
  }
  template <int M, int J, int WG>
  __device__ static __forceinline__ void load(Data<M> &D, const Base &B, const Lane &LN) {
    constexpr int C0 = J * WG * (int)COLB;
    D.sc = lds32o<C0>(B.w);
    static_for<0, 4>([&](auto iq) { D.qs[decltype(iq)::value] = lds32o<C0 + 128 + decltype(iq)::value * 128>(B.w); });
    D.dm = lds32o<C0>(B.d);
    load_x_strips<M, J, WG>(D, B, LN);
  }
  template <int M>
  __device__ static __forceinline__ void compute(const Data<M> &D, const Lane &LN, float (&acc)[M][3]) {
    const float d = h2f_bits(D.dm), dmin = h2f_bits(D.dm >> 16);
    float ds[4], off[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      ds[j] = d * (float)((D.sc >> (8 * j)) & 0x0Fu);
      off[j] = dmin * (float)((D.sc >> (8 * j + 4)) & 0x0Fu);
    }
    uint32_t a[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int n = 0; n < 2; n++) a[i][n] = (D.qs[2 * (i >> 2) + n] >> (2 * (i & 3))) & 0x03030303u;
    mma_strips<M>(D, LN, a, ds, off, acc);
  }
  __device__ static __forceinline__ float finish(const float (&a)[3], const Lane &LN) {
    return LN.kD * (a[0] + a[1]) - a[2];
  }
};

}  // namespace qkdec

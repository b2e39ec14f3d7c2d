// Decode-path dequant-dot (1..4 activation rows) on the integer tensor-core MMA: the part
// that is the same for every weight format.  A format's policy F (qk_dec_*.cuh) says how one
// 256-column span of eight weight rows lies in a tile, which registers hold it, how it is
// loaded and what the MMAs and the scaling are; everything else is here.
//
// The matvec is HBM-bound; what limits a CUDA-core version on this part is the
// issue rate of the per-weight multiply (dp4a runs at a quarter of the FP32
// rate here).  So the multiply-accumulate of every 32-weight group is handed to
// mma.sync.m16n8k32 (8-bit x s8 -> s32) and the CUDA cores only unpack weight bits and
// apply one scale per group.  The matrix is NOT reshaped into a GEMM: each MMA still
// computes plain row dot products, eight weight rows at a time.
//
// Activations are split per 32-column block as x ~= sx (D0 + D1/254 + D2/254^2)
// with |D| <= 127 (error <= amax * 6.1e-8), so the integer dots are exact and
// the result carries f32-grade accuracy.  The B operand's eight columns hold the three
// digits of two 32-weight groups (even columns one group, odd columns the other), so each
// lane of an MMA quad owns digit j = lane % 4 of both groups in fixed registers.
//
// qk_gemv_imma_kernel, persistent, one CTA per SM: a producer warp streams 8-row
// tiles into a ring of shared-memory stages with cp.async.bulk (mbarrier completion);
// the compute warps (16, in four groups or fewer) first split x
// into the digit planes and scale table in shared memory, then a group takes every
// G-th chunk, each warp its share of the tile's 256-column spans, and leaves its row
// partials in a small ring; the producer warp sums a chunk's partials, writes the outputs
// (into y, or as tagged words into every rank's slots for a row-sharded layer) and refills
// the chunk's stages.  No CTA-wide barrier and no compute warp ever waits for another in
// steady state.  When M * K is too large for every CTA to redo the split, qk_xsplit_kernel
// does it once into a scratch image in global memory, which each CTA brings in with one
// more bulk copy.
// Both kernels use programmatic dependent launch: call i+1 is resident and has its first
// weight tiles (weights are immutable) under way before call i has finished;
// griddepcontrol.wait orders everything that touches x, y or the scratch image, and the
// rest of the ring is issued behind the activation loads, not ahead of them.  Every wait on an
// mbarrier is bounded: when one runs out the warp stops, QK_DEV_TIMEOUT is
// raised in the status word, and the other warps run into their own bounds.
#pragma once
#include <cfloat>
#include <cstdlib>
#include <type_traits>

#include "qk_formats.cuh"
#include "qk_kernels.h"
#include "qk_peer.cuh"
#include "qk_pipe.cuh"

#ifdef QK_TRACE
// Developer build only: block 0 timestamps its pipeline into a global buffer.
extern __device__ unsigned long long *qk_trace_buf;
#define QK_STAMP(cond, idx)                                                        \
  do {                                                                             \
    if ((cond) && qk_trace_buf && blockIdx.x == 0 && (threadIdx.x & 31) == 0) {    \
      unsigned long long t__;                                                      \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t__));                     \
      qk_trace_buf[idx] = t__;                                                     \
    }                                                                              \
  } while (0)
#else
#define QK_STAMP(cond, idx) do {} while (0)
#endif

namespace qkdec {

using namespace qkpipe;

constexpr int MAX_CW = 16;                      // compute warps (+ one or two producer / reducer warps)
constexpr uint32_t NBT = QK_TILE_ELEMS / 256;   // super-blocks per full k-tile (16)
constexpr int MAX_STAGE = 12;
constexpr int MAX_SLOT = MAX_STAGE + 1;
constexpr uint32_t PAIR_CHUNKS = 32;            // most chunks of a pair of CTAs

struct SmemMma {
  uint32_t full, redfull, xbar;  // mbarriers (8 B each)
  uint32_t empty;                // chunks of several k-tiles: a stage's tile has been used (one arrival per warp of the group)
  uint32_t prog;                 // chunks the reducer warp has read so far (one word, polled by the producer warp)
  uint32_t issued;               // DEEP: tiles issued so far (one word, polled by the compute warps)
  uint32_t xch;                  // F::XCH bytes per compute warp
  uint32_t pbar, pair;           // PAIR: per chunk, the mbarrier and the 8 x M sums that the other CTA sends
  uint32_t red, ximg, stage;
  uint32_t PS;         // digit plane stride, bytes
  uint32_t xs_off;     // offset of the (sx, Sx) table inside the x image
  uint32_t ximg_bytes;
};

// Loads at a compile-time byte offset from a register base: the offset rides in the
// instruction, where an address built in C++ costs an integer add per load.
template <int OFF>
__device__ __forceinline__ uint2 lds64o(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint4 lds128o(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ float4 lds128fo(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4+%5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr), "n"(OFF));
  return v;
}
template <int I, int N, typename Fn>
__device__ __forceinline__ void static_for(Fn &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The accumulators start at the bit pattern of 1.5 * 2^23, so the integer sums (|v| < 2^22: at most 32 x
// 255 x 127) come out as the floats 12582912 + v: one subtraction, or the difference of two of them,
// gives the exact sum on a full-rate pipe where an int-to-float conversion runs at half rate.
constexpr float MMA_BIAS = 12582912.f;
__device__ __forceinline__ void mma_u8s8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  int r[4];
  asm(  // a pure function of its operands: left free for the scheduler to interleave
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000));
#pragma unroll
  for (int i = 0; i < 4; i++) c[i] = __int_as_float(r[i]);
}

__device__ __forceinline__ void mma_u8s8_k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  int r[4];
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"(a0), "r"(a1), "r"(b0), "r"(0x4B400000));
#pragma unroll
  for (int i = 0; i < 4; i++) c[i] = __int_as_float(r[i]);
}
__device__ __forceinline__ uint32_t word(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Four activations of one 32-column block -> their three balanced base-254 digits, one
// packed word per digit plane: x ~ (amax / 127) (d0 + d1 / 254 + d2 / 254^2).  Adding
// 1.5 * 2^23 rounds to the nearest integer and leaves it, as two's complement, in the low
// mantissa byte; with |v| <= amax every digit lies in [-127, 127] without a clamp.  (Values
// that are not finite give arbitrary digits: digit_scale marks their block.)
__device__ __forceinline__ void split_quad(const float (&v)[4], float inv, uint32_t &w0, uint32_t &w1,
                                           uint32_t &w2) {
  constexpr float MAGIC = 12582912.f;
  uint32_t b0[4], b1[4], b2[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float t0 = fmaf(v[i], inv, MAGIC);
    const float r1 = fmaf(v[i], inv, -(t0 - MAGIC));  // exact residual of the first digit
    const float t1 = fmaf(r1, 254.f, MAGIC);
    const float r2 = fmaf(r1, 254.f, -(t1 - MAGIC));
    const float t2 = fmaf(r2, 254.f, MAGIC);
    b0[i] = __float_as_uint(t0), b1[i] = __float_as_uint(t1), b2[i] = __float_as_uint(t2);
  }
  w0 = __byte_perm(__byte_perm(b0[0], b0[1], 0x0040), __byte_perm(b0[2], b0[3], 0x0040), 0x5410);
  w1 = __byte_perm(__byte_perm(b1[0], b1[1], 0x0040), __byte_perm(b1[2], b1[3], 0x0040), 0x5410);
  w2 = __byte_perm(__byte_perm(b2[0], b2[1], 0x0040), __byte_perm(b2[2], b2[3], 0x0040), 0x5410);
}

// 127 / amax, finite whatever the block holds: a block whose largest magnitude is below 1e-36 keeps the
// grid of 1e-36 (last digit 1.2e-43), and up to FLT_MAX the divisor stays below the 2^126 from which
// __fdividef gives 0.
__device__ __forceinline__ float digit_inv(float &amax) {
  amax = fmaxf(amax, 1e-36f);
  return __fdividef(127.f / 16.f, amax * (1.f / 16.f));
}
// The scale that goes with it.  A block with an infinity or a NaN in it (s32: the sum of its columns) has
// no digits: its scale is NaN, and so is every result that it is part of.
__device__ __forceinline__ float digit_scale(float amax, float s32) {
  return amax > FLT_MAX || s32 != s32 ? __int_as_float(0x7FFFFFFF) : amax * (1.f / 127.f);
}

// Waits (bounded) until more than `item` tiles have been issued: from then on the barrier of the item's stage
// is in the item's phase.  A stage goes from group to group of the compute warps, so a group could come to it
// while the tile before, another group's, is still on its way, two phases back, and take that barrier for its
// own.  That the phases before are over reaches this group through the count alone: published with a release
// behind the waits that saw it, read with an acquire.  `seen`: the count as last read.
__device__ __forceinline__ bool wait_issued(uint32_t word_addr, uint32_t item, uint32_t &seen) {
  if (seen > item) return true;
  unsigned long long t0 = 0;
  for (uint32_t polls = 1;; polls++) {
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(seen) : "r"(word_addr) : "memory");
    if (seen > item) return true;
    if ((polls & 1023u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (!t0) t0 = t;
      if (t - t0 > 250000000ull) return false;
    }
  }
}

// Waits (bounded) until the reducer has read `chunks` chunks.
__device__ __forceinline__ bool wait_read(const volatile uint32_t *prog, uint32_t chunks) {
  unsigned long long t0 = 0;
  for (uint32_t polls = 1; *prog < chunks; polls++) {
    if ((polls & 1023u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (!t0) t0 = t;
      if (t - t0 > 250000000ull) return false;
    }
  }
  return true;
}

__device__ __forceinline__ void tell_issued(uint32_t word_addr, uint32_t items) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(word_addr), "r"(items) : "memory");
}

// Activations e0 .. e0 + 3 of one row out of the tagged slots of a gathered buffer (columns
// past `cols` read as zero); false if a slot's tag did not arrive within the wait's bound.
__device__ __forceinline__ bool load_quad_slots(const unsigned long long *row, unsigned want, uint32_t e0,
                                                uint32_t cols, float (&v)[4]) {
  if (e0 + 4 <= cols) return qkpeer::slot_wait4(row + e0, want, v);
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[i] = 0.f;
    if (e0 + i < cols) ok &= qkpeer::slot_wait(row + e0 + i, want, v[i]);
  }
  return ok;
}

// A float into the same place of the other CTA's shared memory, counted by the mbarrier there.
__device__ __forceinline__ void st_async_other(uint32_t addr, uint32_t bar, uint32_t rank, float v) {
  asm volatile(
      "{\n\t.reg .b32 a, b;\n\tmapa.shared::cluster.u32 a, %0, %2;\n\tmapa.shared::cluster.u32 b, %1, %2;\n\t"
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [a], %3, [b];\n\t}" ::"r"(addr),
      "r"(bar), "r"(rank), "r"(__float_as_uint(v))
      : "memory");
}
__device__ __forceinline__ float lds32f(uint32_t addr) { return __uint_as_float(lds32(addr)); }
// Blocks of a row in its first half: whole spans of 256 columns, the longer half where they are odd.
__host__ __device__ __forceinline__ uint32_t half_blocks(const QkLayout &L) { return (L.nb * L.bs / 256u + 1u) / 2u * (256u / L.bs); }

// ---------------------------------------------------------------- x image
// [M][3 digit planes of PS bytes, columns in the format's order F::store_digits][M][Kp/32] scale entries
// of F::XSB bytes: (sx, sum over the 32 columns) and, for formats with 16-column scales, the two half sums
template <class F>
__global__ void __launch_bounds__(256)
    qk_xsplit_kernel(const float *__restrict__ x, uint32_t m_rows, uint32_t cols, uint32_t Kp,
                     uint32_t PS, uint32_t xs_off, unsigned char *__restrict__ img,
                     const unsigned long long *wait_slots, const unsigned *wait_epoch, uint64_t wait_ld,
                     unsigned *status) {
  pdl_launch_dependents();
  pdl_wait();  // x may be the previous kernel's output; the image may still be in use by it
  const uint32_t quads = Kp / 4, total = m_rows * quads;
  const uint32_t it = blockIdx.x * 256 + threadIdx.x;
  if (it >= total) return;  // warp-uniform: total is a multiple of 64
  const uint32_t m = it / quads, e0 = (it % quads) * 4;
  float v[4];
  if (wait_slots) {  // x is gathered from other GPUs: read it from the tagged slots as it arrives
    if (!load_quad_slots(wait_slots + (uint64_t)m * wait_ld, *wait_epoch, e0, cols, v)) atomicOr(status, QK_DEV_TIMEOUT);
  } else {
    const float *xr = x + (uint64_t)m * cols + e0;
    if ((cols & 3u) == 0 && ((uintptr_t)x & 15u) == 0 && e0 + 4 <= cols) {
      const float4 q = __ldg(reinterpret_cast<const float4 *>(xr));
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) v[i] = (e0 + i < cols) ? __ldg(xr + i) : 0.f;
    }
  }
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  float s4 = (v[0] + v[1]) + (v[2] + v[3]);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1)  // the 8 threads of one 32-column block
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
  s4 += __shfl_xor_sync(0xffffffffu, s4, 2);  // this thread's 16-column half
  const float other = __shfl_xor_sync(0xffffffffu, s4, 4);
  const float inv = digit_inv(amax);
  uint32_t w0, w1, w2;
  split_quad(v, inv, w0, w1, w2);
  F::store_digits(img + (size_t)m * 3 * PS, PS, e0, w0, w1, w2);
  if ((threadIdx.x & 7) == 0)
    F::store_xs(img + xs_off, (size_t)m * (Kp / 32) + e0 / 32, digit_scale(amax, s4 + other), s4 + other, s4, other);
}

// ---------------------------------------------------------------- main kernel
// The same split as qk_xsplit_kernel, done by the compute warps straight into the
// CTA's shared-memory x image (used when x is small enough that every CTA
// redoing it is cheaper than a second kernel and a copy).
// x: M rows of `cols` columns, ldx apart (PAIR: a CTA's half of the columns).
template <class F, int M, int CW, bool PEER, bool PAIR>
__device__ void xsplit_in_cta(const float *__restrict__ x, uint32_t cols, uint32_t ldx, uint32_t Kp,
                              unsigned char *img, uint32_t PS, uint32_t xs_off, bool tell_producer,
                              const QkPeers &peers, unsigned *status) {
  constexpr int CT = CW * 32;  // compute threads
  const uint32_t quads = Kp / 4, total = (uint32_t)M * quads;
  // Every CTA of the grid reads the same few KB of x at the same moment: each starts at
  // a different 32-column block (whole blocks, so the 8 threads of a block stay together)
  // to spread the requests over the L2 slices, and loads 16 bytes at a time when it can.
  const uint32_t rot = (blockIdx.x * 40u) % total;  // a multiple of 8 quads
  const bool vec = (ldx & 3u) == 0 && ((uintptr_t)x & 15u) == 0;
  const bool from_slots = PEER && peers.wait_slots != nullptr;
  const unsigned want = from_slots ? *peers.wait_epoch : 0u;
  bool arrived = true;  // false once a slot has failed to arrive in time: this thread waits no more
  constexpr int U = !PAIR && (M * 4096 / 4 + CT - 1) / CT < 4 ? (M * 4096 / 4 + CT - 1) / CT : 4;  // quads in flight per thread
  for (uint32_t base = 0; base < total; base += CT * U) {
    float v[U][4];
    uint32_t qidx[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
      const uint32_t it0 = base + j * CT + threadIdx.x;
      uint32_t it = it0 + rot;
      if (it >= total) it -= total;
      qidx[j] = it0 < total ? it : 0xFFFFFFFFu;
      const uint32_t m = M == 1 ? 0u : it / quads, e0 = (M == 1 ? it : it % quads) * 4;
      if (from_slots) {  // gathered activations: straight from the tagged slots, as they arrive
        v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
        if (it0 < total && arrived &&
            !load_quad_slots(peers.wait_slots + (uint64_t)m * peers.wait_ld, want, e0, cols, v[j])) {
          arrived = false;
          atomicOr(status, QK_DEV_TIMEOUT);
        }
      } else if (it0 < total && vec && e0 + 4 <= cols) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(x + (uint64_t)m * ldx + e0));
        v[j][0] = q.x, v[j][1] = q.y, v[j][2] = q.z, v[j][3] = q.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
          v[j][i] = (it0 < total && e0 + i < cols) ? __ldg(x + (uint64_t)m * ldx + e0 + i) : 0.f;
      }
    }
    // This thread's first activation loads are on their way: the producer may send the rest
    // of the ring behind them.
    if (tell_producer && base == 0) asm volatile("bar.arrive 2, %0;" ::"n"((CW + 1) * 32) : "memory");
#pragma unroll
    for (int j = 0; j < U; j++) {
      const uint32_t it = qidx[j];
      if (it == 0xFFFFFFFFu) continue;  // warp-uniform: total and CT are multiples of 32
      const uint32_t m = M == 1 ? 0u : it / quads, e0 = (M == 1 ? it : it % quads) * 4;
      float amax = fmaxf(fmaxf(fabsf(v[j][0]), fabsf(v[j][1])), fmaxf(fabsf(v[j][2]), fabsf(v[j][3])));
      float s4 = (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
      s4 += __shfl_xor_sync(0xffffffffu, s4, 2);  // this thread's 16-column half
      const float other = __shfl_xor_sync(0xffffffffu, s4, 4);
      QK_STAMP(threadIdx.x == 0 && j == 0 && amax >= 0.f, 122);
      const float inv = digit_inv(amax);
      uint32_t w0, w1, w2;
      split_quad(v[j], inv, w0, w1, w2);
      F::store_digits(img + (size_t)m * 3 * PS, PS, e0, w0, w1, w2);
      if ((threadIdx.x & 7) == 0)
        F::store_xs(img + xs_off, (size_t)m * (Kp / 32) + e0 / 32, digit_scale(amax, s4 + other), s4 + other, s4, other);
    }
  }
}

// The previous sharded call's gathered result, from its tagged slots into its plain buffer:
// the calling warps of all CTAs share the slots, eight loads in flight per lane; a slot whose
// tag has not arrived yet is waited for (bounded).
__device__ __forceinline__ void unpack_slots(const QkPeers &peers, unsigned uwant, uint32_t lane, unsigned *status) {
  const uint64_t stride = (uint64_t)gridDim.x * 32;
  bool arrived = true;
  for (uint64_t base = (uint64_t)blockIdx.x * 32 + lane; base < peers.unpack_n; base += 8 * stride) {
    unsigned long long w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint64_t i = base + j * stride;
      w[j] = i < peers.unpack_n ? qkpeer::slot_load(peers.unpack_slots + i) : 0ull;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint64_t i = base + j * stride;
      if (i >= peers.unpack_n) break;
      float v = __uint_as_float((unsigned)w[j]);
      if ((unsigned)(w[j] >> 32) != uwant) {  // not there yet: the bounded wait
        if (arrived && !qkpeer::slot_wait(peers.unpack_slots + i, uwant, v)) {
          arrived = false;
          atomicOr(status, QK_DEV_TIMEOUT);
        }
        if (!arrived) v = 0.f;
      }
      peers.unpack_out[i] = v;
    }
  }
}

// PEER: the variant that can store its results into every rank's tagged slots and read
// gathered activations out of slots (kept out of the single-GPU variant, whose speed is
// sensitive to its code size).
// F: the weight format's policy (tile geometry, register image of one 256-column span,
// its loads and its arithmetic; see qk_dec_*.cuh).
// MODE: 0 = one matrix, results into y; 1 = the same with the sharded-layer fan-out (the
// old PEER: results as tagged words into every rank's slots, activations optionally out of
// slots); 2 = two matrices of the same shape and format at once, W as the gate and W2 as the
// up projection of a feed-forward block: a CTA's chunks alternate (gate rows 8 i .., up rows
// 8 i ..), both see the same split activations, and the reducer writes
// silu(gate) * up (crates/oxillama-arch/src/common/swiglu.rs:15-21) where a plain matvec
// writes its dot products.
// 3 = one matrix, each chunk by the two CTAs of a cluster, either half of K (see pair_pays); the reducer of the CTA that
// does not own the chunk (they take turns) sends its sums into the other's shared memory.
// DEEP: the ring has every stage that fits, not a multiple of the groups' (see make_plan_mma).
// LONG: the variant that can hand stages back one by one (see the producer and launch_mma).
template <class F, int M, bool INCTA, int CW, int G, int MODE, bool DEEP, bool LONG>
__global__ void __launch_bounds__((CW + 2 + (MODE == 1 ? 1 : 0)) * 32, 1)
    qk_gemv_imma_kernel(QkLayout L, const uint8_t *__restrict__ W, const uint8_t *__restrict__ W2,
                           const float *__restrict__ x,
                           const unsigned char *__restrict__ ximg_g, float *__restrict__ y,
                           uint64_t ldy, unsigned *status, int nstage, int nslot,
                           uint32_t stage_bytes, SmemMma S, uint32_t Kp, QkPeers peers, int npre) {
  constexpr int WG = CW / G;  // warps per group; a group owns every G-th chunk
  constexpr int XW = CW + 2;  // first warp behind the compute, reducer and producer warps
  constexpr bool PEER = MODE == 1, DUAL = MODE == 2, PAIR = MODE == 3;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  // chunks of this CTA (pair), in the order it takes them; with two matrices every 8-row group counts twice
  const uint32_t rank = PAIR ? blockIdx.x & 1u : 0u, first = PAIR ? blockIdx.x >> 1 : blockIdx.x, step = PAIR ? gridDim.x >> 1 : gridDim.x;
  const uint32_t my_chunks = (first < L.chunks ? (L.chunks - first + step - 1) / step : 0) * (DUAL ? 2u : 1u);
  // its blocks of a row: from block b0 on, nb of them
  const uint32_t nb0 = PAIR ? half_blocks(L) : 0u, b0 = rank ? nb0 : 0u, nb = !PAIR ? L.nb : rank ? L.nb - nb0 : nb0;
  const uint32_t ktiles = PAIR ? (nb + L.nbt - 1) / L.nbt : L.ktiles;
  auto tile_blocks = [&](uint32_t kt) { return min(nb - kt * L.nbt, L.nbt); };
  const uint32_t my_items = my_chunks * ktiles;
  const bool by_tile = LONG && ktiles > 1 && my_items > (uint32_t)nstage;  // stages are handed back one by one (see the producer)

  QK_STAMP(warp == 0, 0);
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < nstage; s++) mbar_init(sbase + S.full + s * 8, 1);
    for (int s = 0; s < nslot; s++) mbar_init(sbase + S.redfull + s * 8, WG);
    mbar_init(sbase + S.xbar, 1);
    *reinterpret_cast<volatile uint32_t *>(smem + S.prog) = 0u, *reinterpret_cast<volatile uint32_t *>(smem + S.issued) = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (by_tile && warp == 2 && lane < (uint32_t)nstage) {
    mbar_init(sbase + S.empty + lane * 8, WG);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (PAIR && warp == 1 && lane < my_chunks && (lane & 1u) == rank) {  // (PAIR_CHUNKS = 32: a lane each)
    mbar_init(sbase + S.pbar + lane * 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(sbase + S.pbar + lane * 8, 8 * M * 4);
  }
  __syncthreads();
  if (PAIR) asm volatile("barrier.cluster.arrive.release;" ::: "memory");  // (the reducers wait for it, and alone come to the second one)

  // tile issue state and helpers of whichever warp streams the tiles
  uint32_t pc = 0, pkt = 0, pst = 0;  // chunk ordinal, k-tile and stage of the next item
  const uint64_t policy = stream_policy();
  uint32_t lead = 0;                  // the lane that issues, in the warp that does
  auto issue = [&]() {                // the whole warp
    const uint32_t chunk = first + (DUAL ? pc >> 1 : pc) * step;
    const uint8_t *Wc = (DUAL && (pc & 1u)) ? W2 : W;
    const uint32_t bytes = QK_TILE_ROWS * tile_blocks(pkt) * L.bb;
    const uint32_t bar = sbase + S.full + pst * 8;
    // (a chunk is its blocks one after the other, eight rows each)
    const uint64_t at = qk_tile_offset(L, chunk, pkt) + (PAIR ? QK_TILE_ROWS * b0 * L.bb : 0u);
    stream_tile(sbase + S.stage + pst * stage_bytes, Wc + at, bytes, bar, policy, lead);
    if (++pkt == ktiles) pkt = 0, pc++;
    if (++pst == (uint32_t)nstage) pst = 0;
  };
  uint32_t item = 0;  // items issued so far; kept in step by every lane
  auto issue_upto = [&](uint32_t limit) {
    const uint32_t end = limit < my_items ? limit : my_items;
    for (; item < end;) {
      issue();
      item++;
      if (DEEP && lead) tell_issued(sbase + S.issued, item);
    }
  };
  if (warp == CW + 1) {
    lead = elect_lead();
    // ================= producer warp =================
    // It streams the tiles: the first ring fill, then the k-tiles of chunk c + (ring depth)
    // as soon as the compute warps have handed chunk c over (they are done with its stages
    // then).  A warp of its own, because a copy instruction does not return until the copy
    // unit has room for it -- a third of a microsecond and more under a saturated stream --
    // and behind the reducer's sums the refills went out up to 1.7 us late, leaving the
    // stream idle between the first ring fill and the refills (IQ4_XS 14336 x 4096: 11.3 -> 10.95 us;
    // Q6_K 4096 x 4096 5.13 -> 4.99, 14336 x 4096 10.21 -> 9.95).  The producer stays at most
    // one chunk ahead of the reducer (S.prog), which is what makes the ring of `nslot`
    // partial buffers safe: chunk c + nslot cannot be computed, let alone handed over,
    // before the reducer has read chunk c.
    issue_upto((uint32_t)npre);  // weights are immutable: their prefetch need not wait for the previous kernel
    pdl_wait();                  // the x image belongs to the previous kernel until it has finished
    if (!INCTA && lane == 0) {
      mbar_expect_tx(sbase + S.xbar, S.ximg_bytes);
      bulk_g2s(sbase + S.ximg, ximg_g, S.ximg_bytes, sbase + S.xbar);
    }
    if (npre < nstage) {
      // The rest of the first ring fill goes out once the compute warps' activation loads
      // have landed (named barrier 2), so that those loads do not queue behind a whole
      // ring of weight tiles from every CTA: measured 11.1 -> 9.7 us per launch at 14336 x 4096.
      if (INCTA) asm volatile("bar.sync 2, %0;" ::"n"((CW + 1) * 32) : "memory");
      issue_upto((uint32_t)nstage);
    }
    const volatile uint32_t *prog = reinterpret_cast<const volatile uint32_t *>(smem + S.prog);
    bool alive = true;
    if (!by_tile) {
      uint32_t slot = 0, sph = 0;
      for (uint32_t c = 0; c < my_chunks && item < my_items; c++) {
        alive = mbar_wait_bounded(sbase + S.redfull + slot * 8, sph)  // chunk c handed over
                && wait_read(prog, c);                                // the reducer has read the chunks before c
        if (!alive) break;
        issue_upto(item + ktiles);
        if (++slot == (uint32_t)nslot) slot = 0, sph ^= 1;
      }
    } else {
      // Chunks of several k-tiles: a stage is filled again as soon as its own tile has been used, not when the whole chunk
      // has been handed over (us: Q4_K 4096 x 14336 by one 10.4 -> 9.7, by two 14.3 -> 12.8, 8192 x 14336 17.1 -> 14.3; Q6_K
      // 16384 x 12288 32.9 -> 27.6; Q5_K 4096 x 14336 by four 41.5 -> 34.9); the first tile of a chunk once the reducer has read the one whose slot it takes.
      uint32_t est = 0, eph = 0;
      while (alive && item < my_items) {
        alive = mbar_wait_bounded(sbase + S.empty + est * 8, eph) && (pkt || pc < (uint32_t)nslot || wait_read(prog, pc + 1 - nslot));
        if (!alive) break;
        issue_upto(item + 1);
        if (++est == (uint32_t)nstage) est = 0, eph ^= 1;
      }
    }
    if (!alive && lane == 0) atomicOr(status, QK_DEV_TIMEOUT);
    return;
  }

  if (warp == CW) {
    // ================= reducer warp =================
    // When a chunk's partials are complete the warp sums them and writes the 8 x M outputs
    // (or stores them into every rank's slots), then says so in S.prog.
    pdl_wait();  // the x image and y belong to the previous kernel until it has finished
    QK_STAMP(true, 120);
    // Sharded output: this call's tag is the object's call count + 1.  Lane 0 reads the
    // count, then counts this CTA in (the add carries a dependency on the value read, so it
    // cannot overtake the read); the CTA that is counted in last knows that every CTA of the
    // launch has read the count and moves it on.  The round trips run while the compute
    // warps load the activations; nothing of this sits at the end of the kernel.
    unsigned e_count = 0, uwant = 0;
    if (PEER && peers.unpack_n)  // needed further down; asked for now, together with the count
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(uwant) : "l"(peers.unpack_epoch) : "memory");
    if (PEER && peers.n && lane == 0) {
      unsigned one;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(e_count) : "l"(peers.epoch) : "memory");
      asm volatile("and.b32 %0, %1, 0;\n\tadd.u32 %0, %0, 1;" : "=r"(one) : "r"(e_count));
      if (atomicAdd(peers.counter, one) == gridDim.x - 1) {
        *reinterpret_cast<volatile unsigned *>(peers.counter) = 0;
        *reinterpret_cast<volatile unsigned *>(peers.epoch) = e_count + 1u;
      }
    }
    const unsigned tag = (PEER && peers.n) ? __shfl_sync(0xffffffffu, e_count, 0) + 1u : 0u;
    // this lane's two destination ranks (lane / 8 and lane / 8 + 4), held in registers: an
    // indexed read of the kernel parameters per chunk costs a constant-cache miss each time
    unsigned long long *slots_a = nullptr, *slots_b = nullptr;
    if (PEER && peers.n) {
      const uint32_t q = lane >> 3;
#pragma unroll
      for (uint32_t p = 0; p < QK_MAX_PEERS; p++) {
        if (p == q && p < peers.n) slots_a = peers.slots[p];
        if (p == q + 4 && p < peers.n) slots_b = peers.slots[p];
      }
    }
    // In passing: the previous sharded call's gathered result goes from its slots into its
    // plain buffer -- by a warp of its own when the launch has one (see below), else here,
    // where this warp has nothing else to do until the first chunk is reduced.
    if (PEER && peers.unpack_n && blockDim.x == XW * 32) unpack_slots(peers, uwant, lane, status);
    if (PAIR) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // the other CTA runs, its barriers are initialised
    uint32_t slot = 0, sph = 0;
    bool dead = false;   // (a lane's) a wait for the other CTA's sums ran out
    float gate_v = 0.f;  // two matrices: the gate chunk's sum, kept until the up chunk's arrives
    for (uint32_t c = 0; c < my_chunks; c++) {
      if (!mbar_wait_bounded(sbase + S.redfull + slot * 8, sph)) {
        if (lane == 0) atomicOr(status, QK_DEV_TIMEOUT);
        dead = true;
        break;
      }
      const float *red = reinterpret_cast<const float *>(smem + S.red) + slot * (WG * M * 8);
      float v = 0.f;
      if (PEER && M == 1 && peers.n) {
        // One activation row, sharded output: every lane sums the row it stores (lane (q, r):
        // row r, for ranks q and q + 4), so that no shuffle sits between the sums and the
        // stores -- the last chunks of a CTA are reduced one after the other, and what each
        // costs here is the tail of the launch.
        const uint32_t r = lane & 7u, row = (blockIdx.x + c * gridDim.x) * 8 + r;
#pragma unroll
        for (int wv = 0; wv < WG; wv++) v += red[wv * 8 + r];
        if (row < L.rows) {
          if (slots_a) qkpeer::slot_store(slots_a + row, v, tag);
          if (slots_b) qkpeer::slot_store(slots_b + row, v, tag);
        }
      } else if (lane < 8 * M) {
        const uint32_t m = lane >> 3, r = lane & 7u;
#pragma unroll
        for (int wv = 0; wv < WG; wv++) v += red[(wv * M + m) * 8 + r];
        const uint32_t row = (first + (DUAL ? c >> 1 : c) * step) * 8 + r;
        if (PAIR) {
          const uint32_t at = sbase + S.pair + (c * 8 * M + lane) * 4, bar = sbase + S.pbar + c * 8;
          if ((c & 1u) != rank) {
            st_async_other(at, bar, rank ^ 1u, v);
          } else if (!mbar_wait_bounded(bar, 0)) {
            dead = true;
          } else if (row < L.rows) {
            y[(uint64_t)m * ldy + row] = v + lds32f(at);
          }
        } else if (DUAL) {
          if ((c & 1u) == 0) {
            gate_v = v;
          } else if (row < L.rows) {
            // swiglu_inplace: sigmoid = 1 / (1 + exp(-g)); g * sigmoid * u, each step rounded
            const float sg = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-gate_v)));
            y[(uint64_t)m * ldy + row] = __fmul_rn(__fmul_rn(gate_v, sg), v);
          }
        } else if (!(PEER && peers.n) && row < L.rows) {
          y[(uint64_t)m * ldy + row] = v;
        }
      }
      if (PEER && peers.n && M > 1) {
        // The same (value, tag) word into the slot of every rank: lane (q, r) stores row r
        // to ranks q, q + 4 (eight consecutive slots = 64 bytes per rank and activation row).
        const uint32_t r = lane & 7u, row = (blockIdx.x + c * gridDim.x) * 8 + r;
#pragma unroll
        for (int m = 0; m < M; m++) {
          const float vm = __shfl_sync(0xffffffffu, v, m * 8 + (int)r);
          if (row < L.rows) {
            if (slots_a) qkpeer::slot_store(slots_a + (uint64_t)m * ldy + row, vm, tag);
            if (slots_b) qkpeer::slot_store(slots_b + (uint64_t)m * ldy + row, vm, tag);
          }
        }
      }
      if (PAIR && __any_sync(0xffffffffu, dead)) {
        if (lane == 0) atomicOr(status, QK_DEV_TIMEOUT);
        break;
      }
      __syncwarp();
      if (lane == 0) *reinterpret_cast<volatile uint32_t *>(smem + S.prog) = c + 1u;  // read: its slot may be written again
      QK_STAMP(c < 30, 64 + c);
      if (++slot == (uint32_t)nslot) slot = 0, sph ^= 1;
    }
    // No CTA ends while the other may still send into its memory: the reducers meet (threads that have ended do not count).
    if (PAIR) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    return;
  }

  if (PEER && warp == XW) {
    // ================= unpack warp (launched only when there is something to unpack) =================
    // On the producer / reducer warp the unpacking (two or three rounds of slot loads, about
    // a microsecond each) held up the first reductions; a warp of its own runs beside them.
    pdl_wait();
    if (peers.unpack_n) {
      unsigned uwant;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(uwant) : "l"(peers.unpack_epoch) : "memory");
      unpack_slots(peers, uwant, lane, status);
    }
    return;
  }

  // ================= compute warps =================
  const uint32_t group = warp / WG, wl = warp % WG;
  const uint32_t g = lane >> 2, tig = lane & 3;
  typename F::Lane LN;  // this lane's constants: which bytes, digits and scales it handles
  LN.init(lane, wl, sbase + S.ximg, S.PS, S.xs_off, Kp);
  if constexpr (F::XCH != 0) LN.set_exchange(sbase + S.xch + warp * F::XCH, lane);

  pdl_wait();  // x may be the previous kernel's output; y may be read or written by it
  QK_STAMP(warp == 0, 121);
  bool dead = false;
  if (INCTA) {
    const uint32_t c0 = b0 * L.bs;  // (PAIR: the second half begins inside the row)
    xsplit_in_cta<F, M, CW, PEER, PAIR>(x + c0, PAIR && !rank ? min(nb0 * L.bs, L.cols) : L.cols - c0, L.cols, Kp, smem + S.ximg, S.PS, S.xs_off,
                                        npre < nstage, peers, status);
    QK_STAMP(warp == 0, 123);
    asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");  // compute warps only
  } else if (!mbar_wait_bounded(sbase + S.xbar, 0)) {
    dead = true;
  }
  float acc[M][3];  // per activation row: the format's running sums (see F::compute / F::finish)
#pragma unroll
  for (int m = 0; m < M; m++) acc[m][0] = acc[m][1] = acc[m][2] = 0.f;
  using Data = typename F::template Data<M>;

  QK_STAMP(warp == 0, 1);
  // loop state kept as counters: no integer division on the critical path
  uint32_t st = 0, fph = 0, slot = 0, seen = 0;
  auto advance_stage = [&](uint32_t n) {
    st += n;
    while (st >= (uint32_t)nstage) st -= nstage, fph ^= 1;
  };
  advance_stage(group * ktiles);
  slot = group % nslot;
  uint32_t tstamp = 0;
  for (uint32_t c = group; c < my_chunks && !dead; c += G) {
    for (uint32_t kt = 0; kt < ktiles; kt++) {
      const uint32_t nbt = tile_blocks(kt) * L.bs / 256u;  // 256-column spans in this tile
      const uint32_t tile = sbase + S.stage + st * stage_bytes;
      // (in the ring's first round there is no tile before)
      const uint32_t it = c * ktiles + kt;
      if ((DEEP && it >= (uint32_t)nstage && !wait_issued(sbase + S.issued, it, seen)) || !mbar_wait_bounded(sbase + S.full + st * 8, fph)) {
        dead = true;
        break;
      }
      QK_STAMP(warp == 0 && tstamp < 30, 2 + 2 * tstamp);
      // One column at a time (fully unrolled): four warps per scheduler hide the latencies.  (Eight warps
      // with the next column's loads in a second register buffer left a scheduler two warps to choose
      // from: 14336 x 4096, 8.0 us at one row, 12.7 at two, 23.5 at four, against 7.9, 11.5, 17.7.)  A full
      // tile (all but the last k-tile of a K that is not a multiple of the tile width) runs without the
      // per-column bound checks.
      // every shared-memory load of a column is a compile-time offset from these per-tile bases
      const typename F::Base B = F::base(LN, tile, kt);
      auto load_sb = [&](Data &D, auto jt) { F::template load<M, decltype(jt)::value, WG>(D, B, LN); };
      auto compute_sb = [&](const Data &D) { F::template compute<M>(D, LN, acc); };
      auto tile_body = [&](auto full_tag) {
        constexpr bool FULL = decltype(full_tag)::value;
        constexpr int NSB = NBT / WG;  // columns of a full tile per warp
        static_for<0, NSB>([&](auto jt) {
          if (FULL || wl + decltype(jt)::value * WG < nbt) {
            Data D;
            load_sb(D, jt);
            compute_sb(D);
          }
        });
      };
      if (nbt == NBT)
        tile_body(std::true_type{});
      else
        tile_body(std::false_type{});
      QK_STAMP(warp == 0 && tstamp < 30, 3 + 2 * tstamp);
      tstamp++;
      if (by_tile) {
        __syncwarp();
        if (lane == 0) mbar_arrive(sbase + S.empty + st * 8);
      }
      advance_stage(1);
    }
    if (dead) break;
    // chunk finished: leave the row partials for the reducer
    float *red = reinterpret_cast<float *>(smem + S.red) + slot * (WG * M * 8);
#pragma unroll
    for (int m = 0; m < M; m++) {
      float v = F::finish(acc[m], LN);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (tig == 0) red[(wl * M + m) * 8 + g] = v;
      acc[m][0] = acc[m][1] = acc[m][2] = 0.f;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(sbase + S.redfull + slot * 8);
    slot += G;
    while (slot >= (uint32_t)nslot) slot -= nslot;
    advance_stage((G - 1) * ktiles);
  }
  if (dead) atomicOr(status, QK_DEV_TIMEOUT);  // a bounded wait ran out: results are invalid
  QK_STAMP(warp == 0, 100);
}

struct PlanMma {
  SmemMma S;
  uint32_t Kp, stage_bytes, total;
  int nstage, nslot, groups;
  int deep;  // stages that fit
};

// xsb: bytes per 32-column block in the activation scale table (F::XSB).  pair: for CTAs that take half of K each.
// xch: bytes per compute warp for what its lanes exchange.
inline bool make_plan_mma(const QkLayout &full, uint32_t m, PlanMma *P, uint32_t xsb, bool pair = false, uint32_t xch = 0) {
  if (full.nb == 0 || full.chunks == 0) return false;  // nothing to stream: the callers handle empty shapes
  if (full.nb * full.bs % 256u) return false;          // the kernels walk K in spans of 256 columns
  QkLayout L = full;
  if (pair) {
    L.nb = half_blocks(full);
    L.ktiles = (L.nb + L.nbt - 1) / L.nbt;
    // (both halves in as many tiles: the ring's depth is a multiple of theirs)
    if (L.nb == full.nb || (full.nb - L.nb + L.nbt - 1) / L.nbt != L.ktiles) return false;
  }
  uint32_t Kp = L.nb * L.bs;
  uint32_t nbt_max = L.nb < L.nbt ? L.nb : L.nbt;
  uint32_t stage_bytes = QK_TILE_ROWS * nbt_max * L.bb;
  stage_bytes = (stage_bytes + 127u) & ~127u;
  SmemMma S;
  uint32_t off = 0;
  S.full = off, off += MAX_STAGE * 8;
  S.empty = off, off += MAX_STAGE * 8;
  S.redfull = off, off += MAX_SLOT * 8;
  S.xbar = off, off += 8;
  S.prog = off, off += 4;
  S.issued = off, off += 4;
  S.pbar = S.pair = off;
  if (pair) off += PAIR_CHUNKS * 8, S.pair = off, off += PAIR_CHUNKS * 8 * m * 4;
  off = (off + 127u) & ~127u;
  S.xch = off, off += MAX_CW * xch;
  S.red = off, off += MAX_SLOT * MAX_CW * m * 8 * 4;
  off = (off + 127u) & ~127u;
  S.PS = Kp + 64;
  S.xs_off = m * 3 * S.PS;
  S.ximg_bytes = S.xs_off + m * (Kp / 32) * xsb;  // multiple of 16: PS and Kp/32*8 both are
  S.ximg = off, off += S.ximg_bytes;
  off = (off + 127u) & ~127u;
  S.stage = off;
  const uint32_t budget = 227u * 1024u - 1024u;
  if (off + 2 * stage_bytes > budget) return false;
  int nstage = (int)((budget - off) / stage_bytes);
  if (nstage > MAX_STAGE) nstage = MAX_STAGE;
  if (const char *e = qk_knob("QK_NSTAGE")) {  // developer knob: shallower ring
    int v = atoi(e);
    if (v >= 2 && v < nstage) nstage = v;
  }
  // a chunk's stages are refilled only once the whole chunk is reduced: its k-tiles
  // must all fit in the ring with room to prefetch the next chunk
  if ((uint32_t)nstage < L.ktiles + 1) return false;
  // Largest group count whose G * ktiles divides a ring depth we can afford.  A stage must always be consumed by
  // the same group (a waiter on an mbarrier may be at most one phase ahead of it), so the depth is a multiple of
  // G * ktiles -- but where ring_is_deep says so.
  const int deep = nstage;
  int groups = 1;
  const char *ge = qk_knob("QK_GROUPS");
  const int gmax = ge ? atoi(ge) : 4;
  for (int gtry = 4; gtry >= 2; gtry >>= 1) {
    const int unit = gtry * (int)L.ktiles;
    if (gtry <= gmax && (nstage / unit) * unit >= (int)L.ktiles + 1) {
      groups = gtry;
      nstage = (nstage / unit) * unit;
      break;
    }
  }
  P->S = S, P->Kp = Kp, P->stage_bytes = stage_bytes, P->nstage = nstage, P->nslot = nstage + 1, P->groups = groups;
  P->deep = deep;
  P->total = off + nstage * stage_bytes;
  return true;
}

// Whether a launch takes every stage that fits and counts the tiles issued (wait_issued): formats with F::ANY_DEPTH,
// where a CTA has more tiles than the multiple holds.  Q6_K, four or seven stages at 4096 columns (us, graph):
// 32000 rows 22.6 -> 19.3, 14336 11.2 -> 10.2, 8192 (seven tiles) 7.8 -> 7.2; but 4096 (four) 5.1 -> 5.4,
// 1024 (one) 3.4 -> 3.55: the further stages stay empty and the count costs.  Q4_K, eight or eleven, 14336 rows
// 7.5 -> 8.2.
template <class F>
inline bool ring_is_deep(const QkLayout &L, const PlanMma &P, int sm_count, bool dual, bool pair = false) {
  const uint32_t most = (uint32_t)sm_count / (pair ? 2u : 1u), grid = L.chunks < most ? L.chunks : most;
  const uint32_t ktiles = pair ? (half_blocks(L) + L.nbt - 1) / L.nbt : L.ktiles;
  return F::ANY_DEPTH && P.deep > P.nstage && (L.chunks + grid - 1) / grid * ktiles * (dual ? 2u : 1u) > (uint32_t)P.nstage;
}

template <class F, int M, bool INCTA, int CW, int G, int MODE, bool DEEP, bool LONG>
cudaError_t launch_mma_kernel(const QkLayout &L, const uint8_t *W, const float *x, float *y, uint64_t ldy,
                              unsigned *status, unsigned char *ximg, int sm_count, const PlanMma &P,
                              cudaStream_t s, const QkPeers *peers, const uint8_t *W2) {
  auto kern = qk_gemv_imma_kernel<F, M, INCTA, CW, G, MODE, DEEP, LONG>;
  static QkPerDevice attr_set;
  if (attr_set.first()) {
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return attr_set.reset(), e;
  }
  static int use_pdl = -1;
  if (use_pdl < 0) {
    const char *e = qk_knob("QK_PDL");
    use_pdl = (e && e[0] == '0') ? 0 : 1;
  }
  cudaLaunchAttribute at[2];
  unsigned n_at = 0;
  if (use_pdl) at[n_at].id = cudaLaunchAttributeProgrammaticStreamSerialization, at[n_at++].val.programmaticStreamSerializationAllowed = 1;

  if (!INCTA) {
    const uint32_t quads = (uint32_t)M * P.Kp / 4;
    cudaLaunchConfig_t c0 = {};
    c0.gridDim = dim3((quads + 255) / 256), c0.blockDim = dim3(256), c0.stream = s;
    c0.attrs = at, c0.numAttrs = n_at;
    cudaError_t e = cudaLaunchKernelEx(&c0, qk_xsplit_kernel<F>, x, (uint32_t)M, L.cols, P.Kp,
                                       P.S.PS, P.S.xs_off, ximg, peers ? peers->wait_slots : nullptr,
                                       peers ? peers->wait_epoch : nullptr, peers ? peers->wait_ld : (uint64_t)0, status);
    if (e != cudaSuccess) return e;
  }
  static int ctas = -1;  // developer knob: persistent CTAs per SM (they must fit: see QK_NSTAGE)
  if (ctas < 0) {
    const char *e = qk_knob("QK_CTAS");
    ctas = (e && atoi(e) == 2) ? 2 : 1;
  }
  uint32_t grid = (uint32_t)sm_count * (uint32_t)ctas;  // persistent
  if (MODE == 3) grid = (uint32_t)sm_count / 2;         // pairs
  if (grid > L.chunks) grid = L.chunks;
  if (MODE == 3) grid *= 2;
  const int nstage = DEEP ? P.deep : P.nstage;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid), cfg.blockDim = dim3((CW + 2 + ((MODE == 1 && peers && peers->unpack_n) ? 1 : 0)) * 32);
  cfg.dynamicSmemBytes = P.total + (uint32_t)(nstage - P.nstage) * P.stage_bytes, cfg.stream = s;
  if (MODE == 3) {
    at[n_at].id = cudaLaunchAttributeClusterDimension;
    at[n_at].val.clusterDim.x = 2, at[n_at].val.clusterDim.y = 1, at[n_at].val.clusterDim.z = 1, n_at++;
  }
  cfg.attrs = at, cfg.numAttrs = n_at;
  QkPeers pv = {};
  if (peers) pv = *peers;
  // Weight tiles issued before the wait on the previous kernel; the rest of the ring follows
  // the activation loads.  Measured at Q4_K 14336 x 4096: M = 1 1 tile 8.09 us, 2 7.88, 3 8.12; M = 2
  // 1 tile 11.2 us, 3 11.5, 4 11.7 (Q8_0 4096^2: 6.4, 7.0, 7.3): the more activations there are to
  // bring in, the more a tile ahead of them costs.
  // QK_PRE overrides (developer knob).
  static int npre_env = -1;
  if (npre_env < 0) {
    const char *e = qk_knob("QK_PRE");
    npre_env = e ? atoi(e) : 0;
  }
  int npre = npre_env > 0 ? npre_env : (M == 1 ? 2 : 1);
  if (npre > nstage) npre = nstage;
  return cudaLaunchKernelEx(&cfg, kern, L, W, W2, x, (const unsigned char *)ximg, y, ldy, status,
                            nstage, nstage + 1, P.stage_bytes, P.S, P.Kp, pv, npre);
}

// The variant of the kernel.  Where stages can be handed back one by one, that is a condition inside the loop over the tiles,
// and it moves the compiler's allocation at the cap of 96 registers one way or the other, also for rows of a single k-tile, which
// never come to it.  F::SHORT_M names the numbers of rows (bit m) where those are faster with a kernel that has no such
// condition (us, with it / without: Q4_0 by three 896 x 3584 4.9 / 4.35, 3072 x 3072 6.4 / 5.9, Q4_K by three 320 x 1280 3.9 /
// 3.6, a feed-forward block of 1024 x 2816 11.0 / 10.4; Q2_K by three, as two and one, 896 x 3584 10.5 / 9.7, Q3_K 11.7 / 10.9; Q5_K by three
// 9600 x 512 5.3 / 5.1, a feed-forward block of 1024 x 2816 11.4 / 11.0; but Q4_K by four 3072 x 3072 6.5 / 6.9, Q8_0 by four 4096 x
// 4096 9.1 / 9.4, Q6_K by two 14336 x 4096 14.8 / 15.7; all other numbers of rows within 1 to 3 % either way).
template <class F, int M, bool INCTA, int CW, int G, int MODE = 0, bool DEEP = false>
cudaError_t launch_mma(const QkLayout &L, const uint8_t *W, const float *x, float *y, uint64_t ldy,
                       unsigned *status, unsigned char *ximg, int sm_count, const PlanMma &P,
                       cudaStream_t s, const QkPeers *peers = nullptr, const uint8_t *W2 = nullptr) {
  constexpr bool SHORT = M > (int)F::BY_TILE_M || (F::SHORT_M >> M & 1u) != 0;  // rows of a single k-tile have a variant of their own
  // (several rows of more than one k-tile are split by a launch of their own, but in formats with OWN_SPLIT)
  if constexpr (M <= (int)F::BY_TILE_M && (!SHORT || M == 1 || !INCTA || F::OWN_SPLIT)) {
    const uint32_t ktiles = MODE == 3 ? (half_blocks(L) + L.nbt - 1) / L.nbt : L.ktiles;
    if (!SHORT || ktiles > 1)
      return launch_mma_kernel<F, M, INCTA, CW, G, MODE, DEEP, true>(L, W, x, y, ldy, status, ximg, sm_count, P, s, peers, W2);
  }
  if constexpr (SHORT) return launch_mma_kernel<F, M, INCTA, CW, G, MODE, DEEP, false>(L, W, x, y, ldy, status, ximg, sm_count, P, s, peers, W2);
  return cudaErrorInvalidConfiguration;
}

// Every CTA redoing the split costs ~M*K/512 quads per thread; past this size the
// separate split kernel plus one bulk copy of its image is cheaper.
inline bool split_in_cta(const PlanMma &P, uint32_t m) {
  static int force = -2;
  if (force == -2) {
    const char *e = qk_knob("QK_XSPLIT");
    force = e ? atoi(e) : -1;  // 0: always the split kernel, 1: always in-CTA
  }
  if (force >= 0) return force == 1;
  return m * P.Kp <= QK_SPLIT_IN_CTA;
}

// Whether one row's matvec goes to pairs of CTAs, each streaming half of a chunk's K and splitting that half of the
// activations itself: where the SMs' shares of chunks are so uneven that half chunks are a shorter longest share, and K so
// long (F::PAIR_COLS; 0: never) that what drops out is worth the meeting of the pair: the launch that splits the activations,
// and an image of them that leaves the ring few stages.  us, whole chunks / halves, a feed-forward block with this matrix last
// (4096 rows: 4 chunks / 7 halves a CTA): Q6_K 14336 columns 27.4 / 26.1, 12288 23.1 / 23.4, 11008 22.0 / 22.4; Q5_K 26.0 /
// 24.9, 12288 22.0 / 22.0, 11008 20.5 / 21.0; Q3_K 27.4 / 26.4, 11008 23.4 / 22.6; IQ4_XS 34.3 / 34.4,
// 13824 34.2 / 33.5, 13312 32.6 / 33.1, with 5120 rows of 13824 41.7 / 39.4; Q8_0 33.8 / 33.7.  The matvec alone: Q6_K 13.0 / 12.9,
// Q5_K 13.1 / 11.2, Q3_K 14.6 / 12.7, IQ4_XS 14.1 / 13.1.  Q4_K and Q4_0 have rings that are long enough; even shares gain little or
// lose (Q6_K, 1024 rows: one chunk or two halves, 6.1 / 6.7), two rows and more mostly lose (Q4_K 1024 x 14336 6.2 / 8.5).
// With one chunk a pair the next launch becomes resident on the SMs that are left; where none are, the gain is small, and IQ4_XS,
// bound by issue, loses (14336 columns, 400, 480 and 592 rows 6.0 / 5.6, 6.1 / 5.9, 6.0 / 6.7; Q5_K 6.3 / 5.1, 6.3 / 5.3, 6.2 / 5.9; Q3_K 7.1 / 5.8,
// 7.1 / 6.0, 7.0 / 6.9; as the last of a block IQ4_XS by 512 rows of 13824 15.3 / 15.5):
// F::PAIR_FULL.
template <class F>
inline bool pair_pays(const QkLayout &L, int sm_count, PlanMma *P) {
  const uint32_t sms = (uint32_t)sm_count, pairs = sms / 2;
  return L.nb * L.bs >= F::PAIR_COLS && L.chunks <= PAIR_CHUNKS * pairs && 2 * ((L.chunks + sms - 1) / sms) > (L.chunks + pairs - 1) / pairs &&
         (F::PAIR_FULL || L.chunks > pairs || L.chunks * 4 <= pairs * 3) && make_plan_mma(L, 1, P, F::XSB, true, F::XCH);
}

template <class F, int M>
cudaError_t launch_mma_m(const QkLayout &L, const uint8_t *W, const float *x, float *y,
                         uint64_t ldy, unsigned *status, unsigned char *ximg, int sm_count,
                         const PlanMma &P, cudaStream_t s, const QkPeers *peers, const uint8_t *W2, bool host_x) {
  // Warp groups: a group owns every G-th chunk (P.groups was chosen with the ring's depth, see make_plan_mma).
  const bool peer = peers != nullptr, deep = ring_is_deep<F>(L, P, sm_count, W2 != nullptr);
  if constexpr (M == 1 && F::PAIR_COLS != 0) {
    PlanMma H;
    if (!peer && !W2 && !host_x && pair_pays<F>(L, sm_count, &H)) {
#define QK_PAIR(GV, DV) return launch_mma<F, M, true, MAX_CW, GV, 3, DV>(L, W, x, y, ldy, status, ximg, sm_count, H, s)
      if constexpr (F::ANY_DEPTH)
        if (ring_is_deep<F>(L, H, sm_count, false, true)) {
          if (H.groups == 4) QK_PAIR(4, true);
          if (H.groups == 2) QK_PAIR(2, true);
        }
      if (H.groups == 4) QK_PAIR(4, false);
      if (H.groups == 2) QK_PAIR(2, false);
      QK_PAIR(1, false);
#undef QK_PAIR
    }
  }
#define QK_LAUNCH2(CWV, GV, PV, DV)                                                                               \
  return !host_x && (!ximg || split_in_cta(P, M))                                                                 \
             ? launch_mma<F, M, true, CWV, GV, PV, DV>(L, W, x, y, ldy, status, ximg, sm_count, P, s, peers, W2)  \
             : launch_mma<F, M, false, CWV, GV, PV, DV>(L, W, x, y, ldy, status, ximg, sm_count, P, s, peers, W2)
#define QK_LAUNCH1(CWV, GV, PV)                            \
  do {                                                     \
    if constexpr (F::ANY_DEPTH && GV > 1) {                \
      if (deep) {                                          \
        QK_LAUNCH2(CWV, GV, PV, true);                     \
      }                                                    \
    }                                                      \
    QK_LAUNCH2(CWV, GV, PV, false);                        \
  } while (0)
#define QK_LAUNCH(CWV, GV)                \
  do {                                    \
    if constexpr (F::HAS_DUAL) {          \
      if (W2) {                           \
        QK_LAUNCH1(CWV, GV, 2);           \
      }                                   \
    }                                     \
    if constexpr (F::HAS_PEER) {          \
      if (peer) {                         \
        QK_LAUNCH1(CWV, GV, 1);           \
      }                                   \
    }                                     \
    QK_LAUNCH1(CWV, GV, 0);               \
  } while (0)
  switch (P.groups) {
    case 4:
      QK_LAUNCH(MAX_CW, 4);
    case 2:
      QK_LAUNCH(MAX_CW, 2);
    default:
      QK_LAUNCH(MAX_CW, 1);
  }
#undef QK_LAUNCH2
#undef QK_LAUNCH1
#undef QK_LAUNCH
}


// Whether one row goes to the format's variant for it: where every CTA splits the activations itself.
template <class F>
inline bool one_pays(const QkLayout &L, int sm_count, PlanMma *P) {
  using O = typename F::One;
  PlanMma pair;
  return (L.nb * L.bs <= QK_SPLIT_IN_CTA || pair_pays<O>(L, sm_count, &pair)) && make_plan_mma(L, 1, P, O::XSB, false, O::XCH);
}

// The public faces of one format's kernels.
template <class F>
bool supported(const QkLayout &L, uint32_t m) {
  if (m < 1 || m > (uint32_t)F::MAX_M) return false;
  PlanMma P;
  return make_plan_mma(L, m, &P, F::XSB);
}

template <class F>
size_t scratch_bytes(const QkLayout &L, uint32_t m) {
  PlanMma P;
  return make_plan_mma(L, m, &P, F::XSB) ? P.S.ximg_bytes : 0;
}

// tiled2 != nullptr: the two-matrix (feed-forward gate and up) mode, formats with F::HAS_DUAL only.
template <class F>
cudaError_t launch(const QkLayout &L, const uint8_t *tiled, const float *x, float *y, uint32_t m, uint64_t ldy,
                   unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s, const QkPeers *peers,
                   const uint8_t *tiled2 = nullptr, bool host_x = false) {
  PlanMma P;
  if constexpr (F::HAS_ONE) {
    if (m == 1 && !peers && !tiled2 && !host_x && one_pays<F>(L, sm_count, &P))
      return launch_mma_m<typename F::One, 1>(L, tiled, x, y, ldy, status, scratch, sm_count, P, s, nullptr, nullptr, false);
  }
  if (!make_plan_mma(L, m, &P, F::XSB)) return cudaErrorInvalidConfiguration;
  if (m < 1 || m > (uint32_t)F::MAX_M) return cudaErrorInvalidConfiguration;
  if ((tiled2 && (!F::HAS_DUAL || peers)) || (peers && !F::HAS_PEER)) return cudaErrorInvalidConfiguration;
  if (m == 1) return launch_mma_m<F, 1>(L, tiled, x, y, ldy, status, scratch, sm_count, P, s, peers, tiled2, host_x);
  if constexpr (F::MAX_M >= 2)
    if (m == 2) return launch_mma_m<F, 2>(L, tiled, x, y, ldy, status, scratch, sm_count, P, s, peers, tiled2, host_x);
  if constexpr (F::MAX_M >= 3)
    if (m == 3) return launch_mma_m<F, 3>(L, tiled, x, y, ldy, status, scratch, sm_count, P, s, peers, tiled2, host_x);
  if constexpr (F::MAX_M >= 4)
    if (m == 4) return launch_mma_m<F, 4>(L, tiled, x, y, ldy, status, scratch, sm_count, P, s, peers, tiled2, host_x);
  return cudaErrorInvalidConfiguration;
}

}  // namespace qkdec

// One translation unit per format instantiates its kernels and exports these three.
#define QK_DEC_DEFINE(NAME, F)                                                                                  \
  bool qk_dec_##NAME##_supported(const QkLayout &L, uint32_t m) { return qkdec::supported<F>(L, m); }           \
  size_t qk_dec_##NAME##_scratch(const QkLayout &L, uint32_t m) { return qkdec::scratch_bytes<F>(L, m); }       \
  cudaError_t qk_dec_##NAME##_launch(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,         \
                                     uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,        \
                                     int sm_count, cudaStream_t s, const QkPeers *peers, const uint8_t *tiled2, bool host_x) { \
    return qkdec::launch<F>(L, tiled, x, y, m, ldy, status, scratch, sm_count, s, peers, tiled2, host_x);       \
  }
#define QK_DEC_DECLARE(NAME)                                                                                    \
  bool qk_dec_##NAME##_supported(const QkLayout &L, uint32_t m);                                                \
  size_t qk_dec_##NAME##_scratch(const QkLayout &L, uint32_t m);                                                \
  cudaError_t qk_dec_##NAME##_launch(const QkLayout &L, const uint8_t *tiled, const float *x, float *y,         \
                                     uint32_t m, uint64_t ldy, unsigned *status, unsigned char *scratch,        \
                                     int sm_count, cudaStream_t s, const QkPeers *peers, const uint8_t *tiled2, bool host_x);

// Batched dequant-matmul (more than four activation rows) on the 5th-generation tensor cores.
//
//   y[t][n] = sum_k  w(n, k) * x[t][k]          w as the format's dequant_block gives it, rounded to fp16 (Q4_K and Q6_K: over a
//                                               power of two of the row, see WFmt)
//
// A real dense contraction, so it goes to tcgen05.mma: 128 weight rows are the MMA's M, up to
// 256 activation rows (tokens) its N, fp16 operands, f32 accumulation in tensor memory.
//
// Both the accumulator and the expanded weights live in tensor memory: a thread that owns a
// weight row expands its columns in registers and stores them with tcgen05.st straight into the
// lane and columns from which the MMA reads its A operand.  Nothing of the weights passes through
// shared memory a second time: no proxy fence, no swizzled stores, and the MMA reads only the
// activations from there.  (Measured: with A in tensor memory an MMA takes max(12, N / 2) cycles,
// with A in shared memory 47 at least; issued by a warp that walks the loop together, the MMA
// predicated on one lane -- a lone thread behind lane == 0 needs 98 cycles per MMA.)
//
// Two forms of the kernel.  CG = 1: one CTA works on 128 rows, for tiles of up to 64 tokens, where
// the expansion is the bound and the hand-overs inside one SM are the shortest.  CG = 2: a pair of
// CTAs (the two SMs of a TPC) works on 256 rows with cta_group::2, each loading half of the tokens:
// at 256 tokens one SM alone would have to load 64 bytes a cycle of activations, which L2 does not
// deliver to all SMs (measured: 53 at 2700 cycles per 256 columns instead of 2048).
//
// Persistent; the work of a CTA (pair) is a list of segments (output tile, run of 256-column
// super-blocks):
//   warp 0      MMA issuer (of both CTAs, in the first of a pair)
//   warp 1      activation producer: TMA tiles (128-byte swizzle) of the fp16 activations
//   warp 2      weight producer: one TMA box per super-block brings the packed bytes of 128 rows
//               (16 chunks x 8 rows) into a ring; it starts before the previous kernel has ended
//   warp 3      allocates and frees the tensor memory
//   warps 4-19  two sets of eight warps that take the super-blocks in turn, one thread per row and
//               128 columns
//   warps 20-23 epilogue: accumulator -> y (or the workspace of a split tile)
// Tensor memory, 512 columns: tiles of more than 128 tokens have two accumulator halves of up to 128
// and two super-blocks of expanded weights; up to 128 tokens one accumulator and three super-blocks
// (a second accumulator would only hide the writing out of one tile under the next one's MMAs, the third
// super-block shortens every round of hand-overs: Q4_K 4096 x 4096 by 512 22.6 -> 21.6 us); up to 64 tokens two
// accumulators of 64, alternating from tile to tile, and three super-blocks.  An SM stores 32 bytes a
// cycle, so writing out a half takes the time of about 32 of its MMAs: at the ends of a wide tile the two
// super-blocks there are issued first half
// by first half, then second half by second half, so that one half is written out under the MMAs of
// the other and the tensor pipe does not wait.
//
// Tiles are dealt out in whole waves; the remainder that would leave SMs idle is cut along K into
// equal runs of super-blocks over all CTAs (pairs).  A tile cut this way has several contributors: each
// leaves its f32 partial in a workspace and counts itself in, and whoever comes last adds the
// partials in a fixed order (so the result does not depend on who that is: the same bits on every
// run) and writes y.  Nobody waits for another CTA.  Where the tiles are so few that each can have a
// cluster of four or eight CTAs, its CTAs take one run each and store their partials straight into the
// shared memory of the CTA that adds up the token (Q4_K 1024 x 4096 by 8 tokens: 8.3 -> 6.6 us; the fence,
// the counter and the loads of the other way cost 4).
//
// The activations are converted to fp16 once per call by qk_x16_kernel, the columns of every
// 64-group in the order in which the packed words yield their weights (both operands use the same
// order, so the sum is unchanged).  fp16 operands put the result at ~5e-4 of the output's
// inf-norm against the f32 reference (its stated tolerance is 1e-3).
//
// Every mbarrier wait is time-bounded; a wait that runs out raises QK_DEV_TIMEOUT and the CTA
// falls through to the common exit, which lets the copies in flight land and frees its tensor
// memory.
#pragma once
#include <cuda.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "qk_kernels.h"
#include "qk_pipe.cuh"

namespace qktc {

using namespace qkpipe;

constexpr uint32_t BM = 128;       // weight rows per CTA
constexpr int QK_TC_WIDE = 0x100;  // or-ed to a format: its expansion for rows whose blocks differ widely (see WFmt)
constexpr int FIRST_DW = 4;        // first expanding warp
constexpr int NDW = 16;            // expanding warps: two sets of eight (three sets of 64 registers a thread: 3 to 10 % slower)
constexpr int FIRST_EW = FIRST_DW + NDW, NTHREADS = (FIRST_EW + 4) * 32;
constexpr uint32_t MAX_BN = 256;   // most tokens per tile: two accumulator halves of 128
constexpr int MAX_WST = 12, MAX_BST = 6;
constexpr uint32_t LUT_OFF = 2688;  // of a format's look-up table in shared memory, behind the barriers and scales

struct TcSmem {
  uint32_t w_full, w_empty, b_full, b_empty, a_full, a_empty, d_full, d_empty, drain, tmem_slot, pre, sched, scales, red;
  uint32_t w, b;                   // ring bases
  uint32_t w_stage, b_stage;       // bytes per stage
  uint32_t w_stages, b_stages;
};

// One call, as every role of the kernel sees it.
struct TcArgs {
  QkLayout L;
  TcSmem S;
  const float *xscale;
  float *y;
  float *part;                     // partial tiles: two slots per CTA, [bn][128] f32 each
  unsigned *cnt;                   // arrivals per (split tile, half, CTA of the pair); zeroed by the conversion kernel
  unsigned *status;
  uint64_t ldy;
  uint32_t m;                      // activation rows (of every group, unless counted on the device)
  uint32_t bn, hn;                 // token rows per tile and of its first accumulator half (bn, if that is 128 at most); multiples of 16
  uint32_t tok_blocks;             // token blocks per group (upper bound where the counts are on the device)
  uint32_t row_blocks;             // 128- or 256-row blocks per matrix
  uint32_t min_run;                // fewest super-blocks worth a CTA in the split part
  uint32_t n, n_act;               // weight matrices; distinct activation groups (group e reads e % n_act)
  uint32_t xcap, ycap;             // rows reserved per group in the activation and output arrays
  uint32_t cs;                     // CTAs of a cluster that share a tile along K (CG = 1, one segment each); 1 = see Sched
  uint32_t once;                   // weights are read once: evict-first in L2
  uint32_t ahead;                  // super-blocks of weights asked for before the CTA sets itself up (two at most; not with counts)
  const int *counts;               // device: live rows per activation group, or null (m rows each)
};
// Tensor maps: the matrices, and the fp16 activations as boxes of 64 columns x h tokens x the steps of
// a stage: h = this CTA's share of hn, or one to four times box_unit where the live tokens of a group are
// known on the device only (whole atoms of 8 rows, and never more than the share, so that a stage is no
// larger than the tile: hn rounded up to four boxes of whole atoms had left tiles of 96 tokens two weight stages).
__host__ __device__ constexpr uint32_t box_unit(uint32_t own) { return (own / 4 + 7) / 8 * 8; }
template <int NG>
struct TcMaps {
  CUtensorMap x[NG > 1 ? 4 : 1];
  CUtensorMap w[NG];
  const float *rows[NG];  // the rows' factors, powers of two (SCALED)
};

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// The whole warp waits: one poll where the phase is already over, else the bounded loop.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
}
// Whether the phase is over, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Issued by the lane that has `lead` set; the whole warp walks the producing loops, so that what the
// compiler knows to be uniform stays in uniform registers (a lone thread needs 500 cycles per copy).
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes), "r"(lead)
      : "memory");
}
// `bar`: a barrier of this CTA or, with CG = 2, of either CTA of the pair (cluster address).
template <int CG>
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar, uint32_t lead) {
#define QK_TMA(GROUP)                                                                                                     \
  asm volatile(                                                                                                           \
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"                                                                   \
      "@q cp.async.bulk.tensor.3d" GROUP ".shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}" ::"r"(dst), \
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "r"(lead)                                                               \
      : "memory")
  if (CG == 1) QK_TMA("");
  else QK_TMA(".cta_group::2");
#undef QK_TMA
}
__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar,
                                                 uint64_t policy, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %7, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], "
      "[%5], %6;\n\t}" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy), "r"(lead)
      : "memory");
}
// Shared-memory descriptor of a K-major operand tile, 128-byte swizzle, rows 128 bytes apart, 8-row
// groups 1024 bytes apart: the low word holds the address / 16, the rest is constant.
constexpr uint32_t UMMA_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (1u << 16); }
// D[128 CG x N] (+)= A[128 CG x 16] B[N x 16]^T with A in tensor memory, issued by the lane that has
// `lead` set.  The whole warp walks the issuing loop: in code that the compiler knows to be uniform
// the operands stay in uniform registers.
template <int CG>
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t bdesc_lo, uint32_t idesc,
                                            uint32_t accumulate, uint32_t lead) {
#define QK_UMMA(GROUP)                                                              \
  asm volatile(                                                                     \
      "{\n\t.reg .pred p, q;\n\t.reg .b64 d;\n\t"                                   \
      "mov.b64 d, {%2, %6};\n\t"                                                    \
      "setp.ne.b32 p, %4, 0;\n\t"                                                   \
      "setp.ne.b32 q, %5, 0;\n\t"                                                   \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [%1], d, %3, p;\n\t}"    \
      :                                                                             \
      : "r"(tmem_d), "r"(tmem_a), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(lead), "n"(UMMA_DESC_HI) \
      : "memory")
  if (CG == 1) QK_UMMA("1");
  else QK_UMMA("2");
#undef QK_UMMA
}
// Arrives on the barrier (of both CTAs of a pair) once the MMAs issued so far have retired.
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t lead) {
  if (CG == 1)
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(bar), "r"(lead)
        : "memory");
}
// The same shared-memory address in the first CTA of a pair.
template <int CG>
__device__ __forceinline__ uint32_t in_first(uint32_t addr) {
  if (CG == 1) return addr;
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(0));
  return r;
}
// Arrives on a barrier of either CTA.  What it orders is tensor-memory work, which the tcgen05 fences
// around it order; a release at cluster scope would also wait for every store to global memory that
// this thread still has in flight (measured: 1000 cycles per arrival).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Stores at the same shared-memory address of CTA `rank` of the cluster.
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t rank, float v) {
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.f32 [a], %2;\n\t}" ::"r"(addr), "r"(rank), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
}

// Barrier of the four epilogue warps that also tells whether any thread came with `v` set.
__device__ __forceinline__ bool any_of_128(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }

// ---------------------------------------------------------------- weight formats
// What differs between the formats is how a thread fetches the packed bytes of half a super-block
// (one weight row x 128 columns: half hh) from the staged super-block and expands them, 32 columns
// at a time.  Each format expands in the order its packed words yield values; src(p) names the
// column (inside the super-block) that lands at position p, and the activations are laid out in the
// same order, so the contraction is unchanged.  (Q4_K, whose order spans 64 columns: conv_order.)
//
// Q4_K and Q6_K expand their fields as fp16 subnormals: masked out of its word, q is the half q 2^-24 (2^-20 for a high
// nibble), exact, and one fused multiply-add with scale 2^24 and offset gives the weight, rounded once.  (With an exponent
// or-ed in and subtracted again it is two packed operations per pair, and the expansion is bound by issue.  us, before /
// now: Q4_K 14336 x 4096 by 8 tokens 13.1 / 11.6, by 37 14.4 / 12.6, 4096 x 14336 by 8 15.5 / 14.3, 4096 x 4096 by 128 14.9 /
// 13.1; Q6_K 4096 x 14336 by 8 16.65 / 16.2, 4096 x 4096 by 37 10.8 / 10.5.  Q8_0 and Q4_0, whose scales change with every 32
// columns, gained nothing: 4096 x 4096 by 8 9.06 / 9.12, 8.31 / 8.33.)  scale 2^24 fits a half because the weights of a row
// are expanded over a power of two of the row's own, its factor; the epilogue multiplies the row's results by it again.
// Scale and weights may be up to 2^-8 of the factor this way, which leaves few bits to the weights far below that: under
// 2^-14 of the factor they are subnormals themselves, rounded to 2^-24 of it, and so is the minimum or offset of a block.
// As long as every block's scale is at least 2^-10 of the factor (945 d and 32 d sc: the weights that a block reaches), the
// products of any single block are within 2 % as exact as from weights in full halves (emulated in f64, activations in that
// block alone; at 2^-12, which blocks whose sub-scales leave most of their range unused may come to, a third less exact, at 2^-14
// four times).  A matrix with a row whose blocks differ by more is
// marked when it is uploaded (qk_gemm_tc_factors), and a call with such a matrix takes the former expansion: the fields as
// whole halves, weights over 2^-17 of the factor, normal halves from 2^15 down to 2^-14 (QK_TC_WIDE; us, by a matrix without
// the mark / with it: Q4_K 14336 x 4096 by 8 11.7 / 13.1, 4096 x 14336 by 37 15.3 / 16.7; Q6_K 14.4 / 14.7, 17.8 / 18.3).
//
//   SCALED    whether the format's rows have factors (qk_gemm_tc_factors); UP, BACK: its scales are taken times 2^UP over the
//             factor (rf, an Rf), and sums of products come out over BACK of it
//   BB, BPS   bytes of a block of one row; blocks per super-block.  A staged super-block is
//             [16 chunks][BPS blocks][8 rows x BB bytes], block-major as in HBM
//   Hd        what the four quarters share (scales), head() fetches it (p: the row's chunk, rf: see above)
//   Qt        the packed bytes of quarter k (32 columns); quarter() fetches them
//   expand    quarter k -> sixteen half2
// (The four quarters are unrolled; as a rolled loop of a quarter of the code they take the same time,
// Q4_K 14336 x 4096 by 64 tokens 18.1 against 18.6 us.)
template <int T>
struct WFmt;

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint32_t v;
  asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t word(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// Four nibble pairs of one packed word -> 8 halves: low nibbles q become 1024 + q
// (0x6400 | q), high nibbles 64 + q (0x5400 | q << 4, no shift needed); values come out
// as pairs (byte 0, byte 2), (byte 1, byte 3) of the low nibbles, then of the high ones.
// The exponents come from registers, so that a mask-and-or has one constant of 32 bits, as many as an instruction takes.
struct NibbleMagic { uint32_t lo, hi; };
__device__ __forceinline__ NibbleMagic nibble_magic() {
  NibbleMagic k;
  asm volatile("mov.b32 %0, 0x64006400;" : "=r"(k.lo));
  asm volatile("mov.b32 %0, 0x54005400;" : "=r"(k.hi));
  return k;
}
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t v) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(mask), "r"(v));
  return d;
}
__device__ __forceinline__ void nibbles_to_magic(uint32_t w, const NibbleMagic &k, uint32_t e[4]) {
  const uint32_t wj = w >> 8;
  e[0] = and_or(w, 0x000F000Fu, k.lo), e[1] = and_or(wj, 0x000F000Fu, k.lo);
  e[2] = and_or(w, 0x00F000F0u, k.hi), e[3] = and_or(wj, 0x00F000F0u, k.hi);
}
// The nibbles of one packed word -> 8 halves: low nibbles become q 2^-24, high ones q 2^-20; values come out
// as pairs (byte 0, byte 2), (byte 1, byte 3) of the low nibbles, then of the high ones.
__device__ __forceinline__ void nibbles_to_halves(uint32_t w, __half2 (&e)[4]) {
  const uint32_t wj = w >> 8;
  e[0] = bits_h2(w & 0x000F000Fu), e[1] = bits_h2(wj & 0x000F000Fu);
  e[2] = bits_h2(w & 0x00F000F0u), e[3] = bits_h2(wj & 0x00F000F0u);
}
// rf as the product of two halves, since it may be up to 2^30.  (All that it is multiplied with stays exact on the way, but for
// scales d of a marked Q4_K matrix below 2^-16 of the row's largest where that is above 4.)
struct RowScale {
  uint32_t a, b;
  __device__ __forceinline__ void set(float factor, int up) {  // 2^up / factor
    const int e = up + 127 - (int)(__float_as_uint(factor) >> 23), ea = max(min(e, 15), -14);
    a = (uint32_t)(15 + ea) * 0x04000400u, b = (uint32_t)(15 + e - ea) * 0x04000400u;
  }
  __device__ __forceinline__ __half2 times(__half2 v) const { return __hmul2(__hmul2(v, bits_h2(a)), bits_h2(b)); }
};
// Four unsigned bytes -> halves 1024 + b, in byte order.
__device__ __forceinline__ void bytes_to_magic(uint32_t w, uint32_t &lo, uint32_t &hi) {
  lo = prmt(w, 0x64646464u, 0x4140), hi = prmt(w, 0x64646464u, 0x4342);
}

template <>
struct WFmt<QK_T_Q4_K> {  // d, dmin, 12 bytes of 6-bit scales / mins, 128 bytes of nibbles (reference/q4_k.rs:27-102)
  static constexpr uint32_t BB = 144, BPS = 1, LUT = 0;
  static constexpr bool SCALED = true;
  using Rf = RowScale;
  static constexpr int UP = 24;
  static constexpr float BACK = 1.f;
  __device__ static void fill_lut(unsigned char *, uint32_t, uint32_t) {}
  // position 8 i + j of a 64-group <- column 4 i + {0,2,1,3}[j & 3] + 32 (j >> 2): byte 4 i + b of
  // the group's 32 holds column 4 i + b (low nibble) and 32 + 4 i + b (high nibble)
  struct Hd { uint32_t scw, mnw, d; };  // the half's four 6-bit scales and minima, one per byte; d rf and dmin rf
  struct Qt { uint4 q; };
  // [8 rows x 16 header | 4 groups x 8 rows x 32 nibble bytes]
  __device__ static void head(Hd &c, uint32_t p, uint32_t rr, uint32_t hh, RowScale rf) {
    const uint4 h = lds128(p + rr * 16);
    c.scw = hh ? ((h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u)) : (h.y & 0x3F3F3F3Fu);
    c.mnw = hh ? (((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u)) : (h.z & 0x3F3F3F3Fu);
    c.d = h2_bits(rf.times(bits_h2(h.x)));
  }
  __device__ static void quarter(Qt &t, uint32_t p, uint32_t rr, uint32_t hh, uint32_t k) {
    t.q = lds128(p + 128 + hh * 512 + rr * 32 + (k >> 1) * 256 + (k & 1u) * 16);
  }
  // d * sc and dmin * mn have 17 bits at most, so the fp16 products are the f32 ones rounded once.
  // 6-bit fields as halves: sc exactly (1024 + sc less 1024), sc / 16 for the high nibbles, mn as mn 2^-24.
  __device__ static void expand(const Qt &t, const Hd &c, uint32_t k, uint32_t (&o)[16], uint32_t) {
    const __half2 d = __low2half2(bits_h2(c.d)), m = __hneg2(__high2half2(bits_h2(c.d)));
    const uint32_t lo = 0x4040u + (k >> 1) * 0x0202u, hi = lo + 0x0101u;  // the 64-group's two sub-blocks
    const __half2 s_lo = __hmul2(__hsub2(bits_h2(prmt(c.scw, 0x64646464u, lo)), __float2half2_rn(1024.f)), d);
    const __half2 s_hi = __hmul2(__hsub2(bits_h2(prmt(c.scw, 0x54545454u, hi)), __float2half2_rn(64.f)), d);
    const __half2 m_lo = __hmul2(bits_h2(prmt(c.mnw, 0u, lo)), m), m_hi = __hmul2(bits_h2(prmt(c.mnw, 0u, hi)), m);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      __half2 e[4];
      nibbles_to_halves(word(t.q, i), e);
      o[4 * i + 0] = h2_bits(__hfma2(e[0], s_lo, m_lo));
      o[4 * i + 1] = h2_bits(__hfma2(e[1], s_lo, m_lo));
      o[4 * i + 2] = h2_bits(__hfma2(e[2], s_hi, m_hi));
      o[4 * i + 3] = h2_bits(__hfma2(e[3], s_hi, m_hi));
    }
  }
};

// Rows whose blocks differ widely (see above).  d * sc and dmin * mn have 17 bits at most, so the fp16 products are the f32 ones
// rounded once; q is exact after the subtraction, then one fused q * scale - min.  |d sc| and |dmin| being at most 2^-8 of the
// factor, a weight is at most 78 2^9, and |d| 2^9.
template <>
struct WFmt<QK_T_Q4_K | QK_TC_WIDE> : WFmt<QK_T_Q4_K> {
  static constexpr int UP = 17;
  static constexpr float BACK = 0x1p-17f;
  __device__ static void expand(const Qt &t, const Hd &c, uint32_t k, uint32_t (&o)[16], uint32_t) {
    const __half2 k1024 = __float2half2_rn(1024.f), k_hi = __float2half2_rn(64.f);
    const __half2 d = __low2half2(bits_h2(c.d)), m = __hneg2(__high2half2(bits_h2(c.d)));
    const uint32_t lo = 0x4040u + (k >> 1) * 0x0202u, hi = lo + 0x0101u;  // the 64-group's two sub-blocks
    const __half2 s_lo = __hmul2(__hsub2(bits_h2(prmt(c.scw, 0x64646464u, lo)), k1024), d);
    const __half2 s_hi = __hmul2(__hsub2(bits_h2(prmt(c.scw, 0x64646464u, hi)), k1024), d);
    const __half2 m_lo = __hmul2(__hsub2(bits_h2(prmt(c.mnw, 0x64646464u, lo)), k1024), m);
    const __half2 m_hi = __hmul2(__hsub2(bits_h2(prmt(c.mnw, 0x64646464u, hi)), k1024), m);
    const NibbleMagic km = nibble_magic();
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t e[4];
      nibbles_to_magic(word(t.q, i), km, e);
      o[4 * i + 0] = h2_bits(__hfma2(__hsub2(bits_h2(e[0]), k1024), s_lo, m_lo));
      o[4 * i + 1] = h2_bits(__hfma2(__hsub2(bits_h2(e[1]), k1024), s_lo, m_lo));
      o[4 * i + 2] = h2_bits(__hfma2(__hsub2(bits_h2(e[2]), k_hi), s_hi, m_hi));
      o[4 * i + 3] = h2_bits(__hfma2(__hsub2(bits_h2(e[3]), k_hi), s_hi, m_hi));
    }
  }
};

template <>
struct WFmt<QK_T_Q8_0> {  // block of 32: f16 d, 32 int8 (reference/q8_0.rs)
  static constexpr uint32_t BB = 34, BPS = 8, LUT = 0;
  static constexpr bool SCALED = false;
  using Rf = RowScale;
  static constexpr int UP = 0;
  static constexpr float BACK = 1.f;
  __device__ static void fill_lut(unsigned char *, uint32_t, uint32_t) {}
  __host__ __device__ static uint32_t src(uint32_t p) { return p; }
  struct Hd {};
  struct Qt { uint4 q[2]; uint32_t d; };
  __device__ static void head(Hd &, uint32_t, uint32_t, uint32_t, RowScale) {}
  // A block's 8 rows: [2 granules x 8 rows x 16 int8][8 x d].  Blocks past the end of the row
  // are zero-filled by the copy: d = 0.
  __device__ static void quarter(Qt &t, uint32_t p, uint32_t rr, uint32_t hh, uint32_t k) {
    p += (hh * 4 + k) * 272;
    t.q[0] = lds128(p + rr * 16), t.q[1] = lds128(p + 128 + rr * 16), t.d = lds16(p + 256 + 2 * rr);
  }
  __device__ static void expand(const Qt &t, const Hd &, uint32_t, uint32_t (&o)[16], uint32_t) {
    const __half2 off = __float2half2_rn(1152.f);  // 1024 + 128: (1024 + (q ^ 0x80)) - 1152 = q, exact; q * d rounded once
    const __half2 d = __low2half2(bits_h2(t.d));
#pragma unroll
    for (int i = 0; i < 8; i++) {
      uint32_t a, b2;
      bytes_to_magic(word(t.q[i >> 2], i & 3) ^ 0x80808080u, a, b2);
      o[2 * i] = h2_bits(__hmul2(__hsub2(bits_h2(a), off), d));
      o[2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(b2), off), d));
    }
  }
};

template <>
struct WFmt<QK_T_Q4_0> {  // block of 32: f16 d, 16 bytes; byte j = elements 2 j (low nibble) and 2 j + 1 (high) (reference/q4_0.rs:36-46)
  static constexpr uint32_t BB = 18, BPS = 8, LUT = 0;
  static constexpr bool SCALED = false;
  using Rf = RowScale;
  static constexpr int UP = 0;
  static constexpr float BACK = 1.f;
  __device__ static void fill_lut(unsigned char *, uint32_t, uint32_t) {}
  // a word yields its eight elements as (byte 0, byte 2), (byte 1, byte 3) low nibbles, then the
  // same of the high nibbles
  __host__ __device__ static uint32_t src(uint32_t p) {
    const uint32_t order = 0x73516240u;  // positions 0..7 <- elements 0, 4, 2, 6, 1, 5, 3, 7 of the word
    return (p & ~7u) + ((order >> (4 * (p & 7u))) & 7u);
  }
  struct Hd {};
  struct Qt { uint4 q; uint32_t d; };
  __device__ static void head(Hd &, uint32_t, uint32_t, uint32_t, RowScale) {}
  // A block's 8 rows: [8 rows x 16 nibble bytes][8 x d].
  __device__ static void quarter(Qt &t, uint32_t p, uint32_t rr, uint32_t hh, uint32_t k) {
    p += (hh * 4 + k) * 144;
    t.q = lds128(p + rr * 16), t.d = lds16(p + 128 + 2 * rr);
  }
  __device__ static void expand(const Qt &t, const Hd &, uint32_t, uint32_t (&o)[16], uint32_t) {
    const __half2 off_lo = __float2half2_rn(1032.f), off_hi = __float2half2_rn(72.f);  // (K + q) - (K + 8) = q - 8, exact
    const __half2 d = __low2half2(bits_h2(t.d));
    const NibbleMagic km = nibble_magic();
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t e[4];
      nibbles_to_magic(word(t.q, i), km, e);
      o[4 * i + 0] = h2_bits(__hmul2(__hsub2(bits_h2(e[0]), off_lo), d));
      o[4 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(e[1]), off_lo), d));
      o[4 * i + 2] = h2_bits(__hmul2(__hsub2(bits_h2(e[2]), off_hi), d));
      o[4 * i + 3] = h2_bits(__hmul2(__hsub2(bits_h2(e[3]), off_hi), d));
    }
  }
};

template <>
struct WFmt<QK_T_Q6_K> {  // super-block of 256: ql 128, qh 64, 16 int8 scales, f16 d (reference/q6_k.rs)
  static constexpr uint32_t BB = 210, BPS = 1, LUT = 0;
  static constexpr bool SCALED = true;
  using Rf = RowScale;
  static constexpr int UP = 24;
  static constexpr float BACK = 1.f;
  __device__ static void fill_lut(unsigned char *, uint32_t, uint32_t) {}
  // half hh = ql[64 hh ..], qh[32 hh ..]; its quarter k (columns 32 k ..) = nibble k >> 1 of ql bytes
  // 32 (k & 1) + l and bit pair 2 k of qh byte l
  __host__ __device__ static uint32_t src(uint32_t p) { return p; }
  struct Hd { uint4 qh[2]; uint2 sc; __half2 d; };  // sc: the half's scales + 128; d rf
  struct Qt { uint4 ql[2]; };
  // A block's 8 rows: [12 granules x 8 rows x 16 bytes of ql+qh][8 rows x 16 scales][8 x d].
  __device__ static void head(Hd &c, uint32_t p, uint32_t rr, uint32_t hh, RowScale rf) {
    const uint32_t q = p + rr * 16;
    c.qh[0] = lds128(q + (8 + 2 * hh) * 128), c.qh[1] = lds128(q + (9 + 2 * hh) * 128);
    c.sc = lds64(q + 1536 + 8 * hh);
    c.sc.x ^= 0x80808080u, c.sc.y ^= 0x80808080u;
    c.d = rf.times(__low2half2(bits_h2(lds16(p + 1664 + 2 * rr))));
  }
  __device__ static void quarter(Qt &t, uint32_t p, uint32_t rr, uint32_t hh, uint32_t k) {
    const uint32_t q = p + rr * 16 + (4 * hh + 2 * (k & 1u)) * 128;
    t.ql[0] = lds128(q), t.ql[1] = lds128(q + 128);
  }
  __device__ static void expand(const Qt &t, const Hd &c, uint32_t k, uint32_t (&o)[16], uint32_t) {
    const uint32_t scw = (k >> 1) ? c.sc.y : c.sc.x, pair = (k & 1u) ? 0x4342 : 0x4140, nib = 4 * (k >> 1), rot = (4 - 2 * k) & 31u;
    // 16 columns per scale: 1024 + (sc + 128) less 1152; d * sc has 19 bits at most and is rounded once; q - 32
    const __half2 sp = __hmul2(__hsub2(bits_h2(prmt(scw, 0x64646464u, pair)), __float2half2_rn(1152.f)), c.d);
    const __half2 op = __hmul2(sp, __float2half2_rn(-0x1p-19f));
    const __half2 s[2] = {__low2half2(sp), __high2half2(sp)}, off[2] = {__low2half2(op), __high2half2(op)};
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t lw = word(t.ql[i >> 2], i & 3) >> nib, hw = word(c.qh[i >> 2], i & 3);
      const uint32_t q6 = (lw & 0x0F0F0F0Fu) | (__funnelshift_l(hw, hw, rot) & 0x30303030u);
      o[2 * i] = h2_bits(__hfma2(bits_h2(prmt(q6, 0u, 0x4140)), s[i >> 2], off[i >> 2]));  // bytes as halves b 2^-24
      o[2 * i + 1] = h2_bits(__hfma2(bits_h2(prmt(q6, 0u, 0x4342)), s[i >> 2], off[i >> 2]));
    }
  }
};

// Rows whose blocks differ widely (see above): (1024 + q) - 1056 = q - 32, exact, then one rounding in the product.  |d sc|
// being at most 2^-8 of the factor, a weight is at most 2^14.  (The scales through f32: with pairs of halves, as above,
// 4096 x 14336 by 8 takes 17.4 us instead of 17.0, 14336 x 4096 by 8 15.5 instead of 14.7.)
template <>
struct WFmt<QK_T_Q6_K | QK_TC_WIDE> : WFmt<QK_T_Q6_K> {
  static constexpr int UP = 17;
  static constexpr float BACK = 0x1p-17f;
  struct Rf {
    float f;
    __device__ __forceinline__ void set(float factor, int up) { f = __uint_as_float((uint32_t)(127 + up) << 23) / factor; }
  };
  struct Hd { uint4 qh[2]; uint2 sc; float d; };
  __device__ static void head(Hd &c, uint32_t p, uint32_t rr, uint32_t hh, Rf rf) {
    const uint32_t q = p + rr * 16;
    c.qh[0] = lds128(q + (8 + 2 * hh) * 128), c.qh[1] = lds128(q + (9 + 2 * hh) * 128);
    c.sc = lds64(q + 1536 + 8 * hh);
    c.d = h2f_bits(lds16(p + 1664 + 2 * rr)) * rf.f;
  }
  __device__ static void expand(const Qt &t, const Hd &c, uint32_t k, uint32_t (&o)[16], uint32_t) {
    const __half2 off = __float2half2_rn(1056.f);
    const uint32_t scw = ((k >> 1) ? c.sc.y : c.sc.x) >> (16 * (k & 1u)), nib = 4 * (k >> 1), rot = (4 - 2 * k) & 31u;
    __half2 s[2];  // 16 columns per scale
#pragma unroll
    for (int i = 0; i < 2; i++) s[i] = __float2half2_rn(c.d * (float)(int)(signed char)((scw >> (8 * i)) & 0xFF));
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t lw = word(t.ql[i >> 2], i & 3) >> nib, hw = word(c.qh[i >> 2], i & 3);
      const uint32_t q6 = (lw & 0x0F0F0F0Fu) | (__funnelshift_l(hw, hw, rot) & 0x30303030u);
      uint32_t a, b2;
      bytes_to_magic(q6, a, b2);
      o[2 * i] = h2_bits(__hmul2(__hsub2(bits_h2(a), off), s[i >> 2]));
      o[2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(b2), off), s[i >> 2]));
    }
  }
};

template <>
struct WFmt<QK_T_IQ4_XS> {  // super-block of 256: f16 d, scales_h, scales_l[4], 128 nibble bytes (reference/iq4_xs.rs:47-97)
  // sub-block s = nibble bytes 16 s ..; byte j holds elements 2 j (low) and 2 j + 1 (high); value =
  // d (ls - 32) K[nibble] with the non-linear table K (iq_shared.rs:16-18).  A table in shared memory
  // maps a byte straight to the half2 (K[low], K[high]) of its two adjacent elements; every lane has
  // a copy of its own in its own bank (32 KB), so the look-ups of a warp never conflict.
  static constexpr uint32_t BB = 136, BPS = 1, LUT = 32768;
  static constexpr bool SCALED = false;  // (the table holds whole numbers as they are: one product)
  using Rf = RowScale;
  static constexpr int UP = 0;
  static constexpr float BACK = 1.f;
  __host__ __device__ static uint32_t src(uint32_t p) { return p; }
  __device__ static void fill_lut(unsigned char *lut, uint32_t tid, uint32_t nthreads) {
    constexpr uint32_t K0 = 0xBFAD9881u, K1 = 0xF6EADDCFu, K2 = 0x26190D01u, K3 = 0x71594535u;  // K[0..15] as bytes
    auto val = [&](uint32_t i) {
      const uint32_t w = i < 8 ? (i < 4 ? K0 : K1) : (i < 12 ? K2 : K3);
      return (float)(int)(signed char)((w >> (8 * (i & 3u))) & 0xFFu);
    };
    for (uint32_t i = tid; i < 256 * 32; i += nthreads)
      reinterpret_cast<uint32_t *>(lut)[i] = h2_bits(__floats2half2_rn(val((i >> 5) & 15u), val(i >> 9)));
  }
  struct Hd { float d; uint32_t ls; };  // ls: the half's four 6-bit scales, one per byte
  struct Qt { uint4 q; };
  // A block's 8 rows: [8 granules x 8 rows x 16 nibble bytes][8 rows x 8 header bytes].
  __device__ static void head(Hd &c, uint32_t p, uint32_t rr, uint32_t hh, RowScale) {
    const uint2 h = lds64(p + 1024 + rr * 8);
    c.d = h2f_bits(h.x);
    const uint32_t sl = hh ? h.y >> 16 : h.y, sh = h.x >> (16 + 8 * hh);
    c.ls = (sl & 0x0Fu) | ((sl & 0xF0u) << 4) | ((sl & 0xF00u) << 8) | ((sl & 0xF000u) << 12);
    c.ls |= ((sh & 3u) << 4) | ((sh & 0xCu) << 10) | ((sh & 0x30u) << 16) | ((sh & 0xC0u) << 22);
  }
  __device__ static void quarter(Qt &t, uint32_t p, uint32_t rr, uint32_t hh, uint32_t k) { t.q = lds128(p + (4 * hh + k) * 128 + rr * 16); }
  // lane4: this lane's word of a table row (byte b's is the row at LUT_OFF + 128 b).  The table lies at a constant
  // offset, so an index is a shift and one and-or, and the offset is the load's own (14336 x 4096 by 37: 18.5 -> 17.1 us,
  // eight experts of 14336 x 4096, 256 tokens top 2: 402 -> 380).
  __device__ static void expand(const Qt &t, const Hd &c, uint32_t k, uint32_t (&o)[16], uint32_t lane4) {
    extern __shared__ __align__(1024) unsigned char smem[];
    auto pair = [&](uint32_t b7) { return bits_h2(*reinterpret_cast<const uint32_t *>(smem + LUT_OFF + ((b7 & 0x7F80u) | lane4))); };
    const __half2 dl = __float2half2_rn(c.d * (float)((int)((c.ls >> (8 * k)) & 0x3Fu) - 32));
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t w = word(t.q, i);
      o[4 * i + 0] = h2_bits(__hmul2(pair(w << 7), dl));
      o[4 * i + 1] = h2_bits(__hmul2(pair(w >> 1), dl));
      o[4 * i + 2] = h2_bits(__hmul2(pair(w >> 9), dl));
      o[4 * i + 3] = h2_bits(__hmul2(pair(w >> 17), dl));
    }
  }
};

// ---------------------------------------------------------------- activations -> fp16
// X16[t][256 s + p] = x[t][256 s + (its format's src of p)] / scale[t] in fp16, where scale[t] is the power
// of two that puts the row's largest magnitude in [512, 1024) (2^-126 at least): the division is
// exact, no activation overflows, only those below 2^-24 of the largest fall into fp16's subnormals, and the
// epilogue multiplies the row of results by scale[t] again (also exact).  Columns >= cols are zero.  One CTA per token
// row; a row of up to 16384 columns is read once and stays in registers between the maximum and
// the conversion (a thread's eight positions come from two float4s whatever the format's order).
// GLU: the row is silu(x) * x2, formed here (crates/oxillama-arch/src/common/swiglu.rs:15-21, each
// step rounded), so the hidden activations of a feed-forward block are never written out in f32.
//
// CT threads keep CCH chunks of eight positions each.  512 threads are the faster conversion of few rows, but
// their CTAs and those of the matmul (24 warps of 80 registers) do not fit on an SM together: the matmul's CTA
// there starts, sets itself up and fetches its first weights only when the conversion is over.  From 64 rows
// of up to 4096 columns 256 threads of 40 registers run beside a matmul of 72 registers.  Q4_K 4096 x 4096
// (where the crossing was measured): 37 rows 11.1 (apart) against 11.5 us (beside), 64 rows 13.8 against 12.6, 128
// rows 19.7 against 18.3.  Short rows keep few of 512 threads busy, so the smaller CTAs pay for Q6_K as well, whose
// matmul stays at 80 registers: 4096 x 4096 by 64 rows 15.6 -> 13.7 us, by 2048 66.8 -> 62.2, 300 x 256 by 4096 27.0 -> 16.9.  And for
// the experts of a mixture, whose rows are mostly not live: 16 experts of 1024 x 1024, 900 tokens top 2, 156 -> 129.  Beside gate
// and up together (80 registers) the smaller CTAs pay from two rows an SM on, six of them being on an SM where there are three of
// 512: feed-forward blocks of 4096 x 14336 by 200 94.5 -> 98.8, by 700 243.5 -> 238.8, 2048 x 5632 by 512 59.0 -> 57.3, by 2048
// 176.3 -> 168.0.
struct ConvArgs {
  const float *x, *x2;
  __half *out;
  float *scales;
  unsigned *zero;                 // arrival counters of the matmul that follows, cleared here
  const int *counts, *lists;      // grouped: live rows per group; rows to gather (row t of group e = x[lists[e][t] / list_div])
  uint32_t m, cols, Kp, n_zero, cap, list_stride, list_div, n_act;
};
// Which row conversion CTA (or cluster) i takes, as group * cap + place in the group: without counts i itself, with them the
// i-th live one.  (A CTA per reserved row, most of which left at once, held up the live ones, for which silu(g) * u
// has three places on an SM: 16 experts of 1024 x 2048 by 300 tokens, top 2, 94.6 -> 78.7 us, of it some 4 from
// qk_moe_group_plan_kernel.)
__device__ __forceinline__ bool conv_row(const ConvArgs &A, uint32_t i, uint32_t &t) {
  t = i;
  if (!A.counts) return true;
  const uint32_t lane = threadIdx.x & 31, c = lane < A.n_act ? min((uint32_t)__ldg(A.counts + lane), A.cap) : 0u;
  uint32_t end = c;
#pragma unroll
  for (int o = 1; o < QK_MAX_GROUPS; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= (uint32_t)o) end += v;
  }
  const uint32_t mine = __ballot_sync(0xffffffffu, lane < A.n_act && i < end);
  if (!mine) return false;
  const uint32_t e = __ffs(mine) - 1;
  t = e * A.cap + i - __shfl_sync(0xffffffffu, end - c, e);
  return true;
}

__device__ __forceinline__ float silu_mul(float g, float u) {
  const float sg = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-g)));
  return __fmul_rn(__fmul_rn(g, sg), u);
}
// Columns ka .. + 3 and kb .. + 3 of conv_load in the order in which they land at positions 8 c ..
template <int T>
__device__ __forceinline__ void conv_order(const float (&a)[4], const float (&b)[4], float (&v)[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint32_t e;  // which of the eight values lands at position j
    if constexpr (T == QK_T_Q4_K) e = (j & 4) + ((j & 3) == 1 ? 2 : (j & 3) == 2 ? 1 : (j & 3));
    else e = WFmt<T>::src((uint32_t)j);
    v[j] = e < 4 ? a[e & 3] : b[e & 3];
  }
}
// The eight activations of positions 8 c .. 8 c + 7.
template <int T, bool GLU>
__device__ __forceinline__ void conv_load(const float *__restrict__ x, const float *__restrict__ x2, uint32_t c,
                                          uint32_t cols, bool vec, float (&v)[8]) {
  const uint32_t ka = T == QK_T_Q4_K ? (c >> 3) * 64 + (c & 7u) * 4 : c * 8, kb = T == QK_T_Q4_K ? ka + 32 : ka + 4;
  float a[4], b[4];
  auto quad = [&](uint32_t k, float (&q)[4]) {
    if (vec && k + 4 <= cols) {
      const float4 f = __ldg(reinterpret_cast<const float4 *>(x + k));
      q[0] = f.x, q[1] = f.y, q[2] = f.z, q[3] = f.w;
      if (GLU) {
        const float4 u = __ldg(reinterpret_cast<const float4 *>(x2 + k));
        q[0] = silu_mul(q[0], u.x), q[1] = silu_mul(q[1], u.y), q[2] = silu_mul(q[2], u.z), q[3] = silu_mul(q[3], u.w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        q[i] = k + i < cols ? __ldg(x + k + i) : 0.f;
        if (GLU && k + i < cols) q[i] = silu_mul(q[i], __ldg(x2 + k + i));
      }
    }
  };
  quad(ka, a), quad(kb, b);
  conv_order<T>(a, b, v);
}

__device__ __forceinline__ float conv_scale(float amax) {
  if (!(amax > 0.f && amax <= FLT_MAX)) return 1.f;  // zero, or not finite (a NaN row stays NaN)
  int e;
  frexpf(amax, &e);  // amax = f * 2^e, f in [0.5, 1)
  return ldexpf(1.f, max(e - 10, -126));  // (from -126 on the reciprocal is finite; a row below 2^-116 starts lower in fp16's range)
}
__device__ __forceinline__ void conv_store(__half *orow, uint32_t c, const float (&w)[8], float inv) {
  uint32_t h[4];
#pragma unroll
  for (int j = 0; j < 4; j++) h[j] = h2_bits(__floats2half2_rn(w[2 * j] * inv, w[2 * j + 1] * inv));
  *reinterpret_cast<uint4 *>(orow + 8ull * c) = make_uint4(h[0], h[1], h[2], h[3]);
}

template <int T, bool GLU, int CT, int CCH>
__global__ void __launch_bounds__(CT, CT == 256 ? 6 : 1) qk_x16_kernel(const ConvArgs A) {
  __shared__ float red[CT / 32];
  pdl_launch_dependents();
  pdl_wait();
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < A.n_zero; i += CT) A.zero[i] = 0u;
  uint32_t t;
  if (!conv_row(A, blockIdx.x, t)) return;  // (rows past the live ones: never stored, their values do not matter)
  const float *xr = A.x + (uint64_t)t * A.cols, *ur = A.x2 + (uint64_t)t * A.cols;
  if (A.lists) xr = A.x + (uint64_t)(A.lists[(uint64_t)(t / A.cap) * A.list_stride + t % A.cap] / (int)A.list_div) * A.cols;
  const bool vec = (A.cols & 3u) == 0 && (((uintptr_t)xr | (GLU ? (uintptr_t)ur : 0u)) & 15u) == 0;
  const uint32_t nch = A.Kp / 8;
  float v[CCH][8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < CCH; i++) {
    const uint32_t c = threadIdx.x + i * CT;
    if (c < nch) {
      conv_load<T, GLU>(xr, ur, c, A.cols, vec, v[i]);
#pragma unroll
      for (int j = 0; j < 8; j++) amax = fmaxf(amax, fabsf(v[i][j]));
    }
  }
  for (uint32_t c = threadIdx.x + CCH * CT; c < nch; c += CT) {  // wider rows: read again below
    float w[8];
    conv_load<T, GLU>(xr, ur, c, A.cols, vec, w);
#pragma unroll
    for (int j = 0; j < 8; j++) amax = fmaxf(amax, fabsf(w[j]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < CT / 32; w++) amax = fmaxf(amax, red[w]);
  const float scale = conv_scale(amax);
  const float inv = 1.f / scale;  // a power of two: exact
  if (threadIdx.x == 0) A.scales[t] = scale;
  __half *orow = A.out + (uint64_t)t * A.Kp;
#pragma unroll
  for (int i = 0; i < CCH; i++) {
    const uint32_t c = threadIdx.x + i * CT;
    if (c < nch) conv_store(orow, c, v[i], inv);
  }
  for (uint32_t c = threadIdx.x + CCH * CT; c < nch; c += CT) {
    float w[8];
    conv_load<T, GLU>(xr, ur, c, A.cols, vec, w);
    conv_store(orow, c, w, inv);
  }
}

// silu(x) * x2 rows through shared memory: 512 threads of 40 registers and a row of 14336 columns leave room
// for three CTAs on an SM, where the form above holds one (78 registers) that loads, computes and stores in
// turn (14336 columns by 512 rows alone 27 -> 9 us; behind the matmul that writes them it costs 26 to 30).  CL CTAs, a cluster,
// share a row and meet once for its largest magnitude: exp and the rounded division keep one SM busy for 2 us with a row of 14336.  Eight or four CTAs a row of more than 8192
// columns as long as they are no more than twice the SMs; else one CTA of 1024 threads a row, from a row per SM on of 512 (us, a
// feed-forward block, one CTA a row / clusters: 4096 x 14336 by 8 40.9 / 39.9, by 19 43.0 / 41.6, by 37 44.7 / 43.8, by 48 44.6 /
// 43.7, by 74 52.2 / 52.5; 3584 x 11776 by 5 37.8 / 36.2, by 30 41.4 / 41.5; shorter rows leave most threads of eight CTAs without
// work: 2048 x 8192 by 12 24.8 / 25.3, by 37 26.2 / 27.6; 2304 x 6144 by 12 21.8 / 21.8; 1536 x 4096 by 12 18.0 / 20.2; 1024 x 2816
// by 18 15.1 / 18.1; two CTAs a row for many rows: 4096 x 14336 by 64 45.8 / 47.2, by 512 192 / 196).
template <int T, int CT, int CL>
__global__ void __launch_bounds__(CT, CT == 512 ? 3 : 1) qk_glu16_kernel(const ConvArgs A) {
  extern __shared__ __align__(16) float glu_row[];
  __shared__ float red[CT / 32], parts[CL];
  pdl_launch_dependents();
  if (CL > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (waited for ahead of the stores into other CTAs)
  pdl_wait();
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < A.n_zero; i += CT) A.zero[i] = 0u;
  uint32_t t;
  if (!conv_row(A, blockIdx.x / CL, t)) return;
  const uint32_t rank = blockIdx.x % CL, per = (A.Kp / 256u + CL - 1) / CL * 256u, k0 = min(rank * per, A.Kp), k1 = min(k0 + per, A.Kp);
  const float *xr = A.x + (uint64_t)t * A.cols, *ur = A.x2 + (uint64_t)t * A.cols;
  const bool vec = (A.cols & 3u) == 0 && (((uintptr_t)xr | (uintptr_t)ur) & 15u) == 0;
  float amax = 0.f;
#pragma unroll 2
  for (uint32_t k = k0 + threadIdx.x * 4; k < k1; k += CT * 4) {
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), u = g;
    if (vec && k < A.cols) {
      g = __ldg(reinterpret_cast<const float4 *>(xr + k)), u = __ldg(reinterpret_cast<const float4 *>(ur + k));
    } else {
      if (k < A.cols) g.x = __ldg(xr + k), u.x = __ldg(ur + k);
      if (k + 1 < A.cols) g.y = __ldg(xr + k + 1), u.y = __ldg(ur + k + 1);
      if (k + 2 < A.cols) g.z = __ldg(xr + k + 2), u.z = __ldg(ur + k + 2);
      if (k + 3 < A.cols) g.w = __ldg(xr + k + 3), u.w = __ldg(ur + k + 3);
    }
    const float4 h = make_float4(silu_mul(g.x, u.x), silu_mul(g.y, u.y), silu_mul(g.z, u.z), silu_mul(g.w, u.w));
    amax = fmaxf(fmaxf(fmaxf(amax, fabsf(h.x)), fmaxf(fabsf(h.y), fabsf(h.z))), fabsf(h.w));
    *reinterpret_cast<float4 *>(glu_row + (k - k0)) = h;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[threadIdx.x % (CT / 32)];
#pragma unroll
  for (int o = CT / 64; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (CL > 1) {
    // A CTA whose part of the row is empty comes here at once: the others must have started before it stores into them.
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x < CL) st_cluster(smem_u32(&parts[rank]), threadIdx.x, amax);
    __syncwarp();
    cluster_sync();
#pragma unroll
    for (int c = 0; c < CL; c++) amax = fmaxf(amax, parts[c]);
  }
  const float scale = conv_scale(amax), inv = 1.f / scale;  // a power of two: exact
  if (threadIdx.x == 0 && rank == 0) A.scales[t] = scale;
  for (uint32_t c = k0 / 8 + threadIdx.x; c < k1 / 8; c += CT) {
    const uint32_t ka = T == QK_T_Q4_K ? (c >> 3) * 64 + (c & 7u) * 4 : c * 8, kb = T == QK_T_Q4_K ? ka + 32 : ka + 4;
    const float4 fa = *reinterpret_cast<const float4 *>(glu_row + (ka - k0)), fb = *reinterpret_cast<const float4 *>(glu_row + (kb - k0));
    const float a[4] = {fa.x, fa.y, fa.z, fa.w}, b[4] = {fb.x, fb.y, fb.z, fb.w};
    float v[8];
    conv_order<T>(a, b, v);
    conv_store(A.out + (uint64_t)t * A.Kp, c, v, inv);
  }
}

// ---------------------------------------------------------------- schedule
// The segments of one CTA (pair), the same list for every role: first whole tiles R + pair, + pairs, ..
// (R = the remainder of the tile count over the pairs), then its run of the split tiles 0 .. R - 1, whose
// R * nsb super-blocks are cut into equal runs.  (The split part last, so that all warps of the CTA can add
// the partials up: four warps alone have 16 KB of loads in flight, 25 us for a tile of 256 x 256 from two
// runs, and a whole tile's main loop behind it does not hide that.)
struct Sched {
  uint32_t nsb, R, base, rem, b, e, first_tile, n_split, whole, n_seg, me, pairs;
  // One tile per cluster of cs CTAs, K cut into cs runs.
  __device__ __forceinline__ void init_cluster(uint32_t nsb_, uint32_t cs) {
    const uint32_t k = blockIdx.x % cs;
    nsb = nsb_, first_tile = blockIdx.x / cs, n_split = n_seg = 1, whole = 0, R = pairs = gridDim.x / cs;
    b = first_tile * nsb + k * nsb / cs, e = first_tile * nsb + (k + 1) * nsb / cs;
  }
  template <int CG>
  __device__ __forceinline__ void init(uint32_t tiles, uint32_t nsb_, uint32_t min_run) {
    nsb = nsb_, me = blockIdx.x / CG, pairs = gridDim.x / CG;
    whole = tiles / pairs;
    R = tiles - whole * pairs;
    const uint32_t total = R * nsb, runs = total / min_run;
    const uint32_t n = min(max(max(runs, R), 1u), pairs);           // pairs that share the split part: never fewer than tiles
    base = total / n, rem = total - base * n;                             // the first `rem` runs are one longer
    b = e = first_tile = n_split = 0;
    if (R && me < n) {
      b = start_of(me), e = start_of(me + 1);
      first_tile = b / nsb;
      n_split = (e - 1) / nsb - first_tile + 1;
    }
    n_seg = n_split + whole;
  }
  __device__ __forceinline__ uint32_t start_of(uint32_t pair) const { return pair * base + (pair < rem ? pair : rem); }
  __device__ __forceinline__ uint32_t owner_of(uint32_t sb) const {  // pair whose run holds super-block sb of the split part
    const uint32_t longer = rem * (base + 1);
    return sb < longer ? sb / (base + 1) : rem + (sb - longer) / base;
  }
  __device__ __forceinline__ void get(uint32_t i, uint32_t &tile, uint32_t &s0, uint32_t &s1) const {
    if (i >= whole) {
      tile = first_tile + i - whole;
      s0 = i == whole ? b - tile * nsb : 0u;
      s1 = i + 1 == n_seg ? e - tile * nsb : nsb;
    } else {
      tile = R + me + i * pairs, s0 = 0, s1 = nsb;
    }
  }
};
// Where a tile lies: its matrix, row block, first token inside the group and live tokens of that group.
struct TileAt {
  uint32_t g, rb, t0, live, n;  // n: tokens the MMA covers, a multiple of 16
};

// The order in which a segment's super-blocks are taken, for the producer of the activations and the issuer of the
// MMAs, who meet only at the ring's stages and must agree: one at a time (under half 0, then half 1), but at either
// end of a wide segment two at a time (both under half 0, then both under half 1).
__device__ __forceinline__ uint32_t taken_together(uint32_t sb, uint32_t s0, uint32_t s1) {
  return s1 - sb >= 2 && (sb == s0 || s1 - sb == 2) ? 2u : 1u;
}
// Calls step(sb, half) in that order -> false to stop.
template <class Step>
__device__ __forceinline__ bool walk_segment(uint32_t s0, uint32_t s1, bool wide, Step &&step) {
  for (uint32_t sb = s0; sb < s1;) {
    const uint32_t two = wide ? taken_together(sb, s0, s1) : 1u;
    for (uint32_t h = 0; h < (wide ? 2u : 1u); h++)
      for (uint32_t k = 0; k < two; k++)
        if (!step(sb + k, h)) return false;
    sb += two;
  }
  return true;
}

// ---------------------------------------------------------------- main kernel
// T: weight format, with QK_TC_WIDE for marked matrices.  CG: CTAs per tile (see the top).  NG: 1 = one matrix; otherwise up to NG matrices
// of one shape and format (the projections of a feed-forward block, the experts of a mixture), each
// multiplying its own group of activation rows.
// REGS: registers per thread: 80, or 72 to leave room for CTAs of the conversion beside it, and for the pairs of one
// matrix at every K (72 / 80, neither of them spilling, us: Q8_0 5120 x 5120 by 160 20.0 / 20.7, Q6_K 4096 x 14336 by 80
// 22.6 / 23.4; 0.7 % over 191 calls).
template <int T, int CG, int NG, int REGS>
__global__ void __maxnreg__(REGS)
    qk_gemm_tc_kernel(const __grid_constant__ TcArgs A, const __grid_constant__ TcMaps<NG> M) {
  extern __shared__ __align__(1024) unsigned char smem[];
  using F = WFmt<T>;
  const TcSmem &S = A.S;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = CG == 1 ? 0u : blockIdx.x & 1u;  // in the pair; rank 0 issues the MMAs of both
  // Tensor memory (see the top): accumulators, then na buffers of 128 columns for the expanded weights.
  const bool narrow = A.hn <= 64, both = A.bn > 128;  // (both: a tile owns two accumulator halves)
  const uint32_t na = both ? 2u : 3u, d_step = narrow ? 64u : 128u, a_col = both ? 256u : 128u, alt = narrow ? 1u : 0u;

  pdl_launch_dependents();
  const bool counted = NG > 1 && A.counts;
  // The schedule of a pair of one matrix lies in shared memory, and a role takes its own copy: in registers from the start
  // its twelve words were live in every role, and the pairs spilled (us, so / now: Q8_0 5120 x 5120 by 80 17.0 / 15.9, Q6_K
  // 4096 x 14336 by 80 24.5 / 22.6, Q4_K 5120 x 5120 by 256 25.8 / 24.4).  Single CTAs do not spill and are up to 12 %
  // slower without it in registers; of the pairs of several matrices some are faster, some slower (8 Q4_K experts, 512
  // tokens 461 / 480).
  constexpr bool SHARED_SCHED = CG == 2 && NG == 1;
  Sched own{};
  Sched &sched = SHARED_SCHED ? *reinterpret_cast<Sched *>(smem + S.sched) : own;
  auto make_schedule = [&](uint32_t tiles) {
    Sched t{};
    if (CG == 1 && NG == 1 && A.cs > 1) t.init_cluster((A.L.cols + 255u) / 256u, A.cs);
    else t.template init<CG>(tiles, (A.L.cols + 255u) / 256u, A.min_run);
    sched = t;
  };
  uint32_t *pre = reinterpret_cast<uint32_t *>(smem + S.pre);  // tiles before group g (device-counted groups)
  auto at = [&](uint32_t tile) {
    TileAt q;
    uint32_t tb;
    if (counted) {
      uint32_t g = 0;
      while (tile >= pre[g + 1]) g++;
      q.g = g, q.live = (uint32_t)__ldg(A.counts + g % A.n_act);
      const uint32_t r = tile - pre[g], nt = (q.live + A.bn - 1) / A.bn;
      q.rb = r / nt, tb = r % nt;
    } else {  // a row block's token blocks are neighbours: its weights are read by CTAs that run at the same time
      tb = tile % A.tok_blocks;
      const uint32_t r = tile / A.tok_blocks;
      q.g = NG > 1 ? r / A.row_blocks : 0u, q.rb = NG > 1 ? r % A.row_blocks : r, q.live = A.m;
    }
    q.t0 = tb * A.bn;
    const uint32_t left = q.live - q.t0;
    q.n = left >= A.bn ? A.bn : ((left + 15u) & ~15u);
    return q;
  };
  if (!counted && (!SHARED_SCHED || threadIdx.x == FIRST_DW * 32)) make_schedule(A.n * A.row_blocks * A.tok_blocks);
  // Where A.ahead says so the first weights are asked for before anything else: a CTA that starts when the
  // previous one on its SM has ended gets them 1.9 us later, and the rest of its setting up takes 1.3.
  uint32_t ws = 0, w_ahead = 0;    // (warp 2) ring stage of the next super-block; super-blocks asked for here
  uint32_t w_lead = 0;
  uint64_t policy = 0;
  if (warp == 2) {
    w_lead = elect_one() ? 1u : 0u;
    if (w_lead) {
      for (uint32_t s = 0; s < S.w_stages; s++) mbar_init(sbase + S.w_full + s * 8, 1), mbar_init(sbase + S.w_empty + s * 8, 8);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (A.once) policy = stream_policy();
    else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
    if (CG == 1 && A.ahead && sched.n_seg) {  // of the first segment
      uint32_t tile, s0, s1;
      sched.get(0, tile, s0, s1);
      const TileAt q = at(tile);
      for (uint32_t sb = s0; sb < s1 && ws < A.ahead; sb++, ws++) {
        expect_tx(sbase + S.w_full + ws * 8, S.w_stage, w_lead);
        tma_load_3d_hint(sbase + S.w + ws * S.w_stage, &M.w[NG > 1 ? q.g : 0], 0, (int)(sb * F::BPS), (int)(q.rb * (16 * CG) + rank * 16),
                         sbase + S.w_full + ws * 8, policy, w_lead);
      }
      w_ahead = ws;
    }
  }
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < S.b_stages; s++) mbar_init(sbase + S.b_full + s * 8, 1), mbar_init(sbase + S.b_empty + s * 8, 1);
    for (uint32_t s = 0; s < 3; s++) mbar_init(sbase + S.a_full + s * 8, CG * 8), mbar_init(sbase + S.a_empty + s * 8, 1);
    for (uint32_t s = 0; s < 2; s++) mbar_init(sbase + S.d_full + s * 8, 1), mbar_init(sbase + S.d_empty + s * 8, CG * 4);
    mbar_init(sbase + S.drain, 1);
    *reinterpret_cast<volatile uint32_t *>(smem + S.scales + 2052) = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 32) asm volatile("prefetch.tensormap [%0];" ::"l"(&M.x[0]) : "memory");
  if (F::LUT) F::fill_lut(smem + LUT_OFF, threadIdx.x, NTHREADS);
  if (warp == 3) {
    if (CG == 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + S.tmem_slot), "r"(512u) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + S.tmem_slot), "r"(512u) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
  }
  if (counted) {
    pdl_wait();  // the counts are the work of an earlier kernel
    if (threadIdx.x == 0) {
      uint32_t s = 0;
      for (uint32_t g = 0; g < A.n; g++) {
        pre[g] = s;
        s += A.row_blocks * (((uint32_t)A.counts[g % A.n_act] + A.bn - 1) / A.bn);
      }
      pre[A.n] = s;
    }
  }
  tc_fence_before();
  __syncthreads();
  const bool shared = CG == 1 && NG == 1 && A.cs > 1;  // a tile's K runs in the CTAs of a cluster
  if (CG == 2) cluster_sync();  // the other CTA runs, its barriers are initialised, its tensor memory is there
  if (shared) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (waited for ahead of the stores into other CTAs)
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + S.tmem_slot);

  if (counted) make_schedule(pre[A.n]);
  // Token rows that an activation box brings: each CTA of a pair loads half of the n tokens.
  const uint32_t hq = box_unit(A.hn / CG);
  auto box_of = [&](uint32_t n) { return NG > 1 ? (n / CG + hq - 1) / hq : 1u; };  // the how-manieth box (from 1)
  auto box_rows = [&](uint32_t n) { return NG > 1 ? min(box_of(n) * hq, A.hn / CG) : A.hn / CG; };

  // What the results of four rows are multiplied with (a multiple of 4 the first; the table has whole chunks of 8)
  auto factors4 = [&](uint32_t g, uint32_t row) {
    float4 f = F::SCALED && row < A.L.rows ? __ldg(reinterpret_cast<const float4 *>(M.rows[g] + row)) : make_float4(1.f, 1.f, 1.f, 1.f);
    f.x *= F::BACK, f.y *= F::BACK, f.z *= F::BACK, f.w *= F::BACK;
    return f;
  };
  // The last contributor of a split tile adds the partials up, in the order of their K runs: a warp four
  // tokens at a time, a lane four rows.
  auto add_up = [&](uint32_t tile) {
    __threadfence();
    const Sched sc = sched;
    const TileAt q = at(tile);
    const uint32_t i0 = sc.owner_of(tile * sc.nsb), i1 = sc.owner_of((tile + 1) * sc.nsb - 1), slot = A.bn * BM;
    const uint32_t live = min(q.live - q.t0, q.n), row0 = (q.rb * CG + rank) * BM, rw = row0 + 4 * lane;
    const float *sp = A.xscale + (NG > 1 ? (q.g % A.n_act) * A.xcap : 0u) + q.t0;
    float *yt = A.y + (uint64_t)((NG > 1 ? q.g * A.ycap : 0u) + q.t0) * A.ldy;
    const bool vec = row0 + BM <= A.L.rows && (A.ldy & 3u) == 0 && ((uintptr_t)A.y & 15u) == 0;
    const float4 rk = factors4(NG > 1 ? q.g : 0, rw);
    for (uint32_t c = 4 * warp; c < live; c += NTHREADS / 8) {
      float4 s[4];
#pragma unroll
      for (uint32_t j = 0; j < 4; j++) s[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
      for (uint32_t p = i0; p <= i1; p++) {
        const float *src = A.part + ((p * CG + rank) * 2 + (sc.start_of(p) / sc.nsb == tile ? 0u : 1u)) * slot + c * BM + 4 * lane;
        float4 o[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) o[j] = ldcg4(src + j * BM);  // (token rows past the live ones exist: n is a multiple of 16)
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) s[j].x += o[j].x, s[j].y += o[j].y, s[j].z += o[j].z, s[j].w += o[j].w;
      }
      float *yp = yt + (uint64_t)c * A.ldy + rw;
#pragma unroll
      for (uint32_t j = 0; j < 4; j++, yp += A.ldy) {
        if (c + j >= live) break;
        const float f = __ldg(sp + c + j);
        const float4 v = make_float4(s[j].x * rk.x * f, s[j].y * rk.y * f, s[j].z * rk.z * f, s[j].w * rk.w * f);
        if (vec) {
          *reinterpret_cast<float4 *>(yp) = v;
        } else {
          if (rw < A.L.rows) yp[0] = v.x;
          if (rw + 1 < A.L.rows) yp[1] = v.y;
          if (rw + 2 < A.L.rows) yp[2] = v.z;
          if (rw + 3 < A.L.rows) yp[3] = v.w;
        }
      }
    }
  };
  volatile uint32_t *last = reinterpret_cast<volatile uint32_t *>(smem + S.scales + 2052);  // split segments that this CTA adds up at its end

  bool dead = false;
  if (warp == 0 && rank == 0) {
    // ======================= MMA issuer =======================
    // Narrow tiles are bound by this loop unless it is short: beside its 16 MMAs (14 cycles each) a step has room
    // for some 500 cycles before it takes longer than the expansion.  So what a segment does not change is worked
    // out ahead of its steps, and the next step's barriers are looked at (without waiting) behind the commits.  (As
    // one general step per super-block and half, worked out anew each time: 1250 cycles at 8 to 128 tokens.)
    const Sched sc = sched;
    const uint32_t lead = elect_one() ? 1u : 0u;
    const uint32_t a_full = sbase + S.a_full, a_empty = sbase + S.a_empty, b_full = sbase + S.b_full, b_empty = sbase + S.b_empty;
    const uint32_t nbs = S.b_stages, stage16 = S.b_stage >> 4, bd0 = umma_desc_lo(sbase + S.b), a0 = tmem + a_col;
    uint32_t bs = 0, bph = 0, ab = 0, aph = 0, dph = 0;  // dph bit h: parity of the next wait for half h; bit 2 + h: it was used before
    bool ready = false;                                  // (this lane) the next step's operands were there when last looked at
    auto take_half = [&](uint32_t dh) {                  // a segment's first MMA into an accumulator
      if ((dph >> (2 + dh)) & 1u) {
        if (!warp_wait(sbase + S.d_empty + dh * 8, (dph >> dh) & 1u)) return false;
        tc_fence_after();  // its former contents have been read by other warps
        dph ^= 1u << dh;
      }
      dph |= 4u << dh;
      return true;
    };
    auto issue16 = [&](uint32_t d, uint32_t a, uint32_t bd, uint32_t step16, uint32_t idesc, uint32_t acc) {
#pragma unroll
      for (uint32_t g = 0; g < 4; g++)
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) umma_f16_ta<CG>(d, a + g * 32 + j * 8, bd + g * step16 + j * 2, idesc, g || j ? 1u : acc, lead);
    };
    for (uint32_t i = 0; i < sc.n_seg && !dead; i++) {
      uint32_t tile, s0, s1;
      sc.get(i, tile, s0, s1);
      const TileAt q = at(tile);
      const bool wide = CG == 2 && q.n > A.hn;
      const uint32_t n0 = wide ? A.hn : q.n, idesc0 = (1u << 4) | ((n0 >> 3) << 17) | ((CG * BM >> 4) << 24);
      const uint32_t step0 = box_rows(n0) * 8u;  // a step of the activation stage, in units of 16 bytes
      if (!wide) {
        const uint32_t dh = both ? 0u : i & alt, d = tmem + dh * d_step;
        if (!take_half(dh)) {
          dead = true;
          break;
        }
        uint32_t acc = 0u;
        for (uint32_t sb = s0; sb < s1; sb++) {
          if (!__all_sync(0xffffffffu, ready) && !(warp_wait(a_full + ab * 8, aph) && warp_wait(b_full + bs * 8, bph))) {
            dead = true;
            break;
          }
          tc_fence_after();
          issue16(d, a0 + ab * 128u, bd0 + bs * stage16, step0, idesc0, acc);
          umma_commit<CG>(b_empty + bs * 8, lead);
          umma_commit<CG>(a_empty + ab * 8, lead);
          acc = 1u;
          if (++bs == nbs) bs = 0, bph ^= 1u;
          if (++ab == na) ab = 0, aph ^= 1u;
          ready = mbar_test(a_full + ab * 8, aph) & mbar_test(b_full + bs * 8, bph);
        }
        if (!dead) umma_commit<CG>(sbase + S.d_full + dh * 8, lead);
      } else {
        // Two accumulator halves, in the order of walk_segment; the buffers are walked again under the second half.
        // (Written out: as one step for either half, gate and up of 14336 x 4096 by 512 took 111.6 us under ncu instead of
        // 103.3.)
        const uint32_t n1 = q.n - A.hn, idesc1 = (1u << 4) | ((n1 >> 3) << 17) | ((CG * BM >> 4) << 24), step1 = box_rows(n1) * 8u;
        bool ok = take_half(0);
        ready = false;
        uint32_t acc0 = 0u, acc1 = 0u;
        for (uint32_t sb = s0; sb < s1 && ok;) {
          const uint32_t two = taken_together(sb, s0, s1);
          uint32_t abk = ab, ph = aph;
          for (uint32_t k = 0; k < two && ok; k++) {
            ok = __all_sync(0xffffffffu, ready) || (warp_wait(a_full + abk * 8, ph) && warp_wait(b_full + bs * 8, bph));
            if (!ok) break;
            tc_fence_after();
            issue16(tmem, a0 + abk * 128u, bd0 + bs * stage16, step0, idesc0, acc0);
            umma_commit<CG>(b_empty + bs * 8, lead);
            acc0 = 1u;
            if (++bs == nbs) bs = 0, bph ^= 1u;
            if (++abk == na) abk = 0, ph ^= 1u;
            ready = k + 1 < two && (mbar_test(a_full + abk * 8, ph) & mbar_test(b_full + bs * 8, bph));
          }
          if (sb + two == s1 && ok) umma_commit<CG>(sbase + S.d_full, lead);
          if (!acc1 && ok) ok = take_half(1);
          abk = ab;
          for (uint32_t k = 0; k < two && ok; k++) {
            if (!(ok = warp_wait(b_full + bs * 8, bph))) break;
            issue16(tmem + d_step, a0 + abk * 128u, bd0 + bs * stage16, step1, idesc1, acc1);
            umma_commit<CG>(b_empty + bs * 8, lead);
            umma_commit<CG>(a_empty + abk * 8, lead);
            acc1 = 1u;
            if (++bs == nbs) bs = 0, bph ^= 1u;
            if (++abk == na) abk = 0;
          }
          if (sb + two == s1 && ok) umma_commit<CG>(sbase + S.d_full + 8, lead);
          ab = abk, aph = ph;
          sb += two;
          ready = mbar_test(a_full + ab * 8, aph) & mbar_test(b_full + bs * 8, bph);
        }
        if (!ok) dead = true;
      }
    }
    if (dead) {  // let what was issued retire before the CTA gives its memory back
      if (lead) atomicOr(A.status, QK_DEV_TIMEOUT);
      umma_commit<CG>(sbase + S.drain, lead);
      (void)mbar_wait_bounded(sbase + S.drain, 0);
    }
  } else if (warp == 1) {
    // ======================= activation producer =======================
    const Sched sc = sched;
    const uint32_t lead = elect_one() ? 1u : 0u;
    pdl_wait();  // X16 belongs to the previous kernel until it has finished
    const uint32_t full0 = in_first<CG>(sbase + S.b_full);
    uint32_t bs = 0, bph = 0, rounds = 0, bar = sbase + S.b_full, dst = sbase + S.b, full = full0;
    const uint32_t to_empty = S.b_empty - S.b_full, nst = S.b_stages, stage = S.b_stage;
    for (uint32_t i = 0; i < sc.n_seg && !dead; i++) {
      uint32_t tile, s0, s1;
      sc.get(i, tile, s0, s1);
      const TileAt q = at(tile);
      const bool wide = CG == 2 && q.n > A.hn;
      const uint32_t n0 = wide ? A.hn : q.n, n1 = wide ? q.n - A.hn : 0u, rows0 = box_rows(n0), rows1 = box_rows(n1);
      const uint32_t row0 = (NG > 1 ? (q.g % A.n_act) * A.xcap : 0u) + q.t0;
      const int r0 = (int)(row0 + (rank ? n0 / 2 : 0u)), r1 = (int)(row0 + A.hn + (rank ? n1 / 2 : 0u));
      const CUtensorMap *map0 = &M.x[box_of(n0) - 1], *map1 = &M.x[wide ? box_of(n1) - 1 : 0];
      const bool ok = walk_segment(s0, s1, wide, [&](uint32_t sb, uint32_t h) {
        if (rounds && !warp_wait(bar + to_empty, bph ^ 1u)) return false;
        // the halves of both CTAs land on the barrier of rank 0, which alone announces them
        if (rank == 0) expect_tx(bar, (h ? rows1 : rows0) * 512u * CG, lead);
        tma_load_3d<CG>(dst, h ? map1 : map0, 0, h ? r1 : r0, (int)(sb * 4), full, lead);
        bs++, bar += 8, full += 8, dst += stage;
        if (bs == nst) bs = 0, bph ^= 1u, rounds = 1, bar = sbase + S.b_full, full = full0, dst = sbase + S.b;
        return true;
      });
      if (!ok) dead = true;
    }
    if (dead) {
      if (lead) atomicOr(A.status, QK_DEV_TIMEOUT);
      if (rank == 0)  // copies in flight land before the CTAs end
        for (uint32_t k = 0; k < nst; k++)
          if (rounds || k < bs) (void)mbar_wait_bounded(sbase + S.b_full + k * 8, k < bs ? bph : bph ^ 1u);
    }
  } else if (warp == 2) {
    // ======================= weight producer =======================
    // The weights are immutable: their stream starts before the previous kernel has ended.
    const Sched sc = sched;
    const uint32_t lead = w_lead, to_empty = S.w_empty - S.w_full, nst = S.w_stages, stage = S.w_stage;
    uint32_t wph = 0, rounds = 0;
    if (ws == nst) ws = 0, wph = 1u, rounds = 1;
    uint32_t bar = sbase + S.w_full + ws * 8, dst = sbase + S.w + ws * stage;
    for (uint32_t i = 0; i < sc.n_seg && !dead; i++) {
      uint32_t tile, s0, s1;
      sc.get(i, tile, s0, s1);
      const TileAt q = at(tile);
      const CUtensorMap *map = &M.w[NG > 1 ? q.g : 0];
      for (uint32_t sb = s0 + (i == 0 ? w_ahead : 0u); sb < s1; sb++) {
        if (rounds && !warp_wait(bar + to_empty, wph ^ 1u)) {
          dead = true;
          break;
        }
        expect_tx(bar, stage, lead);
        tma_load_3d_hint(dst, map, 0, (int)(sb * F::BPS), (int)(q.rb * (16 * CG) + rank * 16), bar, policy, lead);
        ws++, bar += 8, dst += stage;
        if (ws == nst) ws = 0, wph ^= 1u, rounds = 1, bar = sbase + S.w_full, dst = sbase + S.w;
      }
    }
    if (dead) {
      if (lead) atomicOr(A.status, QK_DEV_TIMEOUT);
      for (uint32_t k = 0; k < nst; k++)
        if (rounds || k < ws) (void)mbar_wait_bounded(sbase + S.w_full + k * 8, k < ws ? wph : wph ^ 1u);
    }
  } else if (warp >= FIRST_EW) {
    // ======================= epilogue warps =======================
    // Warp `quarter` owns accumulator lanes (weight rows) 32 quarter .. + 32 of every half.
    const Sched sc = sched;
    const uint32_t quarter = warp & 3u, r = 32 * quarter + lane;
    const uint32_t tlane = tmem + ((32 * quarter) << 16);
    const uint32_t d_empty = in_first<CG>(sbase + S.d_empty);
    float *scales = reinterpret_cast<float *>(smem + S.scales) + quarter * 128;  // this warp's copy of a half's token scales
    if (shared) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // the other CTAs run
    volatile uint32_t *told = reinterpret_cast<volatile uint32_t *>(smem + S.scales + 2048);
    uint32_t dph = 0;
    pdl_wait();  // y, the scales and the workspace belong to the previous kernel until it has finished
    const uint64_t ldy = A.ldy;
    uint32_t i = 0;
    for (; i < sc.n_seg && !dead; i++) {
      uint32_t tile, s0, s1;
      sc.get(i, tile, s0, s1);
      const TileAt q = at(tile);
      const bool wide = q.n > A.hn;
      const bool split = s0 != 0 || s1 != sc.nsb;
      const uint32_t row0 = (q.rb * CG + rank) * BM, row = row0 + r;
      const float *sp = A.xscale + (NG > 1 ? (q.g % A.n_act) * A.xcap : 0u) + q.t0;
      float *yt = A.y + (uint64_t)((NG > 1 ? q.g * A.ycap : 0u) + q.t0) * ldy;  // the tile's first token
      const float rk = F::SCALED && !split && row < A.L.rows ? F::BACK * __ldg(M.rows[NG > 1 ? q.g : 0] + row) : 1.f;
      // partial tiles: [slot][token][128 rows]
      const uint32_t slot = A.bn * BM;
      float *mine = A.part + (blockIdx.x * 2 + (i == sc.whole ? 0u : 1u)) * slot + r;
      for (uint32_t h = 0; h < (wide ? 2u : 1u); h++) {
        const uint32_t dh = both ? h : i & alt, hoff = h * A.hn;  // first token of the half inside the tile
        const uint32_t n = h ? q.n - A.hn : wide ? A.hn : q.n;
        const uint32_t live = min(q.live - q.t0 - hoff, n);      // tokens to write
        if (!split) {
          __syncwarp();
#pragma unroll
          for (uint32_t k = 0; k < 4; k++) scales[k * 32 + lane] = k * 32 + lane < live ? __ldg(sp + hoff + k * 32 + lane) : 0.f;
          __syncwarp();
        }
        if (!warp_wait(sbase + S.d_full + dh * 8, (dph >> dh) & 1u)) {
          dead = true;
          break;
        }
        dph ^= 1u << dh;
        tc_fence_after();
        float *yp = yt + (uint64_t)hoff * ldy + row, *pp = mine + hoff * BM;
        for (uint32_t c = 0; c < n; c += 16, pp += 16 * BM) {
          uint32_t v[16];
          tmem_ld16(tlane + dh * d_step + c, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c + 16 == n) {  // read to the end: the half is free for its next tile
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(d_empty + dh * 8);
          }
          if (shared) {
            // to the CTA of the cluster that adds up the token
            const uint32_t own = (live + A.cs - 1) / A.cs, at = sbase + S.red + (blockIdx.x % A.cs * own * BM + r) * 4;
            uint32_t to = c / own, t = c % own;
#pragma unroll
            for (uint32_t j = 0; j < 16; j++) {
              if (c + j < live) st_cluster(at + t * (BM * 4), to, __uint_as_float(v[j]));
              if (++t == own) t = 0, to++;
            }
          } else if (split) {
#pragma unroll
            for (uint32_t j = 0; j < 16; j++) __stcg(pp + j * BM, __uint_as_float(v[j]));
          } else {
            const float4 *f4 = reinterpret_cast<const float4 *>(scales + c);
            if (row0 + 32 * quarter + 32 <= A.L.rows && c + 16 <= live) {  // warp-uniform: all of it is wanted
#pragma unroll
              for (uint32_t j4 = 0; j4 < 4; j4++) {
                const float4 f = f4[j4];
                *yp = __uint_as_float(v[4 * j4]) * rk * f.x, yp += ldy;
                *yp = __uint_as_float(v[4 * j4 + 1]) * rk * f.y, yp += ldy;
                *yp = __uint_as_float(v[4 * j4 + 2]) * rk * f.z, yp += ldy;
                *yp = __uint_as_float(v[4 * j4 + 3]) * rk * f.w, yp += ldy;
              }
            } else {
#pragma unroll
              for (uint32_t j = 0; j < 16; j++, yp += ldy)
                if (row < A.L.rows && c + j < live) *yp = __uint_as_float(v[j]) * rk * scales[c + j];
            }
          }
        }
      }
      if (!split) continue;
      if (shared) break;  // see below
      // Count in, once both halves are in the workspace (the accumulators are free by now); the last
      // contributor adds the partials up, in the order of their K runs.
      const uint32_t i0 = sc.owner_of(tile * sc.nsb), i1 = sc.owner_of((tile + 1) * sc.nsb - 1);
      __threadfence();
      if (any_of_128(dead)) {
        dead = true;
        continue;
      }
      if (warp == FIRST_EW && lane == 0) *told = atomicAdd(A.cnt + tile * 2 + rank, 1u);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (*told != i1 - i0) continue;
      if (warp == FIRST_EW && lane == 0) *last |= 1u << (i - sc.whole);  // all warps add them up, below
    }
    if (dead) {
      // A warp whose wait ran out still comes to the barriers of the split tiles that are left: there the
      // other three, if theirs did not, learn of it.
      if (lane == 0) atomicOr(A.status, QK_DEV_TIMEOUT);
      for (; i < sc.n_seg; i++) {
        uint32_t tile, s0, s1;
        sc.get(i, tile, s0, s1);
        if ((s0 != 0 || s1 != sc.nsb) && !shared) (void)any_of_128(true);
      }
    }
  } else if (warp >= FIRST_DW) {
    // ======================= expanding warps =======================
    // Set `set` takes every second super-block; in it, warp (hh, quarter) the columns [128 hh, + 128)
    // and the tensor-memory lanes 32 quarter .. + 32.
    const uint32_t set = (warp - FIRST_DW) >> 3, hh = ((warp - FIRST_DW) >> 2) & 1u, quarter = warp & 3u;
    const uint32_t r = 32 * quarter + lane, rr = r & 7u;               // weight row inside the tile, inside its chunk
    constexpr uint32_t CHB = 8 * F::BB * F::BPS;                       // a chunk's bytes of one super-block
    uint32_t n_sb = 0;
    for (uint32_t i = 0; i < sched.n_seg; i++) {
      uint32_t tile, s0, s1;
      sched.get(i, tile, s0, s1);
      n_sb += s1 - s0;
    }
    // The factor of this thread's row in the segment that holds super-block j, and in the one behind it
    uint32_t seg = 0, seg_end = 0;
    auto row_of = [&](uint32_t i) {
      if (i >= sched.n_seg) return 1.f;
      uint32_t tile, s0, s1;
      sched.get(i, tile, s0, s1);
      const TileAt q = at(tile);
      const uint32_t row = (q.rb * CG + rank) * BM + r;
      return row < A.L.rows ? __ldg(M.rows[NG > 1 ? q.g : 0] + row) : 1.f;
    };
    auto seg_len = [&](uint32_t i) {
      uint32_t tile, s0, s1;
      sched.get(i, tile, s0, s1);
      return s1 - s0;
    };
    typename F::Rf rf = {};
    float next_factor = 1.f;
    if (F::SCALED && n_sb) rf.set(row_of(0), F::UP), next_factor = row_of(1), seg_end = seg_len(0);
    const uint32_t w_bytes = S.w_stage, nst = S.w_stages, w0 = sbase + S.w + (r >> 3) * CHB;
    const uint32_t ta0 = tmem + ((32 * quarter) << 16) + a_col + hh * 64u, a_full0 = in_first<CG>(sbase + S.a_full);
    uint32_t ws = set, wph = 0;      // ring stage and parity of this set's next super-block
    uint32_t ab = set, auses = 0;                       // its buffer, and how often that has been used (set < na)
    for (uint32_t j = set; j < n_sb; j += 2) {
      if (F::SCALED)
        while (j >= seg_end) rf.set(next_factor, F::UP), next_factor = row_of(++seg + 1), seg_end += seg_len(seg);
      if (!warp_wait(sbase + S.w_full + ws * 8, wph)) {
        dead = true;  // warp-uniform: these warps execute .aligned tcgen05 instructions
        break;
      }
      const uint32_t p = w0 + ws * w_bytes;
      typename F::Hd hd;
      typename F::Qt qt;
      F::quarter(qt, p, rr, hh, 0);
      F::head(hd, p, rr, hh, rf);
      // the MMAs that read this buffer's previous contents must have retired
      if (auses && !warp_wait(sbase + S.a_empty + ab * 8, (auses - 1) & 1u)) {
        dead = true;
        break;
      }
      tc_fence_after();
      const uint32_t ta = ta0 + ab * 128u;
#pragma unroll
      for (uint32_t k = 0; k < 4; k++) {
        typename F::Qt next;
        F::quarter(next, p, rr, hh, k < 3 ? k + 1 : 3);
        uint32_t o[16];
        F::expand(qt, hd, k, o, lane * 4);
        tmem_st16(ta + 16 * k, o);
        qt = next;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(sbase + S.w_empty + ws * 8);  // every lane holds its packed bytes
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(a_full0 + ab * 8);
      ws += 2;
      if (ws >= nst) ws -= nst, wph ^= 1u;
      ab += 2;
      if (ab >= na) ab -= na, auses++;
    }
    if (dead && lane == 0) atomicOr(A.status, QK_DEV_TIMEOUT);
  }

  // common exit: the tensor memory is always returned
  tc_fence_before();
  if (shared && warp < FIRST_EW) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // (the epilogue warps have)
  __syncthreads();
  if (shared) {
    // The partial sums of this CTA's tokens, by the epilogue warps (they alone have waited for the kernels before;
    // for another warp that takes 0.3 us even when it is long over): a lane four rows of one token at a time, the
    // first scale fetched ahead of the meeting.  Added up in the order of the K runs.
    const bool adds = warp >= FIRST_EW;
    const TileAt q = at(sched.first_tile);
    const uint32_t live = min(q.live - q.t0, q.n), own = (live + A.cs - 1) / A.cs, t0 = blockIdx.x % A.cs * own, t1 = min(t0 + own, live);
    const uint32_t first = t0 + warp - FIRST_EW, r = 4 * lane, row = q.rb * BM + r;
    const float *sp = A.xscale + q.t0;
    float f = adds && first < t1 ? __ldg(sp + first) : 0.f;
    const float4 rk = adds ? factors4(0, row) : make_float4(1.f, 1.f, 1.f, 1.f);
    cluster_sync();  // all partial sums are here; nobody leaves while another may still store into its memory
    const bool vec = q.rb * BM + BM <= A.L.rows && (A.ldy & 3u) == 0 && ((uintptr_t)A.y & 15u) == 0;
    for (uint32_t t = first; adds && t < t1; t += 4) {
      const float *red = reinterpret_cast<const float *>(smem + S.red) + (t - t0) * BM + r;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (uint32_t p = 0; p < A.cs; p++) {
        const float4 o = *reinterpret_cast<const float4 *>(red + p * own * BM);
        v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
      }
      if (t != first) f = __ldg(sp + t);
      float *yp = A.y + (uint64_t)(q.t0 + t) * A.ldy + row;
      v.x = v.x * rk.x * f, v.y = v.y * rk.y * f, v.z = v.z * rk.z * f, v.w = v.w * rk.w * f;
      if (vec) {
        *reinterpret_cast<float4 *>(yp) = v;
      } else {
        if (row < A.L.rows) yp[0] = v.x;
        if (row + 1 < A.L.rows) yp[1] = v.y;
        if (row + 2 < A.L.rows) yp[2] = v.z;
        if (row + 3 < A.L.rows) yp[3] = v.w;
      }
    }
  }
  if (CG == 2) cluster_sync();  // neither CTA leaves while the other may still arrive on its barriers or read its operands
  tc_fence_after();
  if (warp == 3) {
    if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
  if (*last)
    for (uint32_t i = 0; i < sched.n_split; i++)
      if (*last >> i & 1u) add_up(sched.first_tile + i);
}

// ---------------------------------------------------------------- host side
constexpr uint32_t GLU_SMEM = 110u * 1024u;    // two CTAs on an SM at least
constexpr uint32_t SMEM_BUDGET = 225u * 1024u;  // leaves room for a CTA of the conversion

struct TcPlan {
  TcSmem S;
  uint32_t cg, cs, smem, bn, hn, tok_blocks, row_blocks, nsb, min_run, grid, xrows;
  size_t o_scale, o_cnt, o_part, bytes;
};
// qk_gemm_tc.cu
bool make_plan(const QkTcCall &c, int sm_count, TcPlan *P);
bool x_map(CUtensorMap *m, __half *x16, uint32_t xrows, uint32_t Kp, uint32_t rows);

inline cudaLaunchAttribute pdl_attr() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

template <int T, int CG, int NG, int REGS = 80>
cudaError_t launch_main(const TcPlan &P, const TcArgs &A, __half *x16, const QkTcCall &c, cudaStream_t s) {
  auto kern = qk_gemm_tc_kernel<T, CG, NG, REGS>;
  static QkPerDevice attr_set;
  if (attr_set.first()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BUDGET);
    if (e != cudaSuccess) return attr_set.reset(), e;
  }
  TcMaps<NG> M;
  for (uint32_t k = 0; k < (NG > 1 ? 4u : 1u); k++)
    if (!x_map(&M.x[k], x16, P.xrows, P.nsb * 256u, NG > 1 ? std::min(box_unit(P.hn / CG) * (k + 1), P.hn / CG) : P.hn / CG)) return cudaErrorInvalidValue;
  for (uint32_t g = 0; g < (NG == 1 ? 1u : c.n); g++) memcpy(&M.w[g], c.maps[g], sizeof(CUtensorMap)), M.rows[g] = c.rows[g];
  cudaLaunchAttribute at[2] = {pdl_attr(), {}};
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CG == 2 ? 2 : P.cs, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.grid), cfg.blockDim = dim3(NTHREADS), cfg.dynamicSmemBytes = P.smem, cfg.stream = s;
  cfg.attrs = at, cfg.numAttrs = CG == 2 || P.cs > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, A, M);
}

template <int T, int CT, int CL>
cudaError_t launch_glu16(const ConvArgs &C, uint32_t rows, cudaStream_t s) {
  static QkPerDevice attr_set;
  if (attr_set.first()) {
    cudaError_t e = cudaFuncSetAttribute(qk_glu16_kernel<T, CT, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GLU_SMEM);
    if (e != cudaSuccess) return attr_set.reset(), e;
  }
  cudaLaunchAttribute at[2] = {pdl_attr(), {}};
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CL, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows * CL), cfg.blockDim = dim3(CT), cfg.dynamicSmemBytes = (C.Kp / 256u + CL - 1) / CL * 1024u, cfg.stream = s;
  cfg.attrs = at, cfg.numAttrs = CL > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, qk_glu16_kernel<T, CT, CL>, C);
}

// The matmul itself.  beside: single CTAs of 72 registers.
template <int T>
cudaError_t launch_matmul(const TcPlan &P, const TcArgs &A, __half *x16, const QkTcCall &c, bool beside, cudaStream_t s) {
  if (c.n == 1 && !c.counts) {
    if (P.cg == 2) return launch_main<T, 2, 1, 72>(P, A, x16, c, s);
    return beside ? launch_main<T, 1, 1, 72>(P, A, x16, c, s) : launch_main<T, 1, 1>(P, A, x16, c, s);
  }
  return P.cg == 1 ? launch_main<T, 1, QK_MAX_GROUPS>(P, A, x16, c, s) : launch_main<T, 2, QK_MAX_GROUPS>(P, A, x16, c, s);
}
// With a marked matrix (qk_tc_q4k_wide.cu, qk_tc_q6k_wide.cu)
cudaError_t launch_wide_q4k(const TcPlan &P, const TcArgs &A, __half *x16, const QkTcCall &c, bool beside, cudaStream_t s);
cudaError_t launch_wide_q6k(const TcPlan &P, const TcArgs &A, __half *x16, const QkTcCall &c, bool beside, cudaStream_t s);

template <int T>
cudaError_t launch_fmt(const QkTcCall &c, unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s) {
  const QkLayout &L = *c.L;
  TcPlan P;
  if (!make_plan(c, sm_count, &P)) return cudaErrorInvalidConfiguration;
  const uint32_t Kp = P.nsb * 256u;
  __half *x16 = reinterpret_cast<__half *>(scratch);
  float *scales = reinterpret_cast<float *>(scratch + P.o_scale);
  unsigned *cnt = reinterpret_cast<unsigned *>(scratch + P.o_cnt);
  ConvArgs C = {};
  C.x = c.x, C.x2 = c.x2, C.out = x16, C.scales = scales, C.zero = cnt, C.n_zero = (uint32_t)sm_count * 2;
  C.counts = c.counts, C.lists = c.lists, C.m = c.m, C.cols = L.cols, C.Kp = Kp, C.cap = c.xcap;
  C.list_stride = c.list_stride, C.list_div = c.list_div ? c.list_div : 1u, C.n_act = c.n_act;
  const bool narrow = (c.counts || c.m >= (c.n == 1 ? 64u : 2 * (uint32_t)sm_count)) && Kp <= 4096;
  // Single CTAs beside the conversion (72 registers).  Q6_K only where the conversion has more rows than a tile: its
  // expansion wants the 80 (us, 80 / 72 registers: 4096 x 4096 by 80 16.5 / 14.4, by 160 17.1 / 15.4; 14336 x 4096 by
  // 64 16.1 / 16.9).
  const bool beside = narrow && c.n == 1 && !c.counts && (T != QK_T_Q6_K || c.m > 64);
  cudaLaunchAttribute at = pdl_attr();
  cudaLaunchConfig_t c0 = {};
  const uint32_t all_rows = c.counts || c.n_act > 1 ? c.n_act * c.xcap : c.m;
  c0.gridDim = dim3(c.counts && c.live < all_rows ? c.live : all_rows), c0.blockDim = dim3(narrow ? 256 : 512), c0.stream = s, c0.attrs = &at, c0.numAttrs = 1;
  cudaError_t e;
  if (c.x2 && !c.lists && Kp * 4 <= GLU_SMEM) {
    const uint32_t rows = c0.gridDim.x, sms = (uint32_t)sm_count, room = !c.counts && Kp > 8192 ? 2 * sms : 0u;
    if (rows * 8 <= room) e = launch_glu16<T, 512, 8>(C, rows, s);
    else if (rows * 4 <= room) e = launch_glu16<T, 512, 4>(C, rows, s);
    else if (!c.counts && rows <= sms) e = launch_glu16<T, 1024, 1>(C, rows, s);
    else e = launch_glu16<T, 512, 1>(C, rows, s);
  } else if (c.x2) {
    c0.blockDim = dim3(512);
    e = cudaLaunchKernelEx(&c0, qk_x16_kernel<T, true, 512, 4>, C);
  } else {
    e = narrow ? cudaLaunchKernelEx(&c0, qk_x16_kernel<T, false, 256, 2>, C) : cudaLaunchKernelEx(&c0, qk_x16_kernel<T, false, 512, 4>, C);
  }
  if (e != cudaSuccess) return e;

  TcArgs A;
  A.L = L, A.S = P.S, A.xscale = scales, A.y = c.y, A.part = reinterpret_cast<float *>(scratch + P.o_part), A.cnt = cnt;
  A.status = status, A.ldy = c.ldy, A.m = c.m, A.bn = P.bn, A.hn = P.hn, A.tok_blocks = P.tok_blocks, A.row_blocks = P.row_blocks;
  A.cs = P.cs, A.min_run = P.min_run, A.n = c.n, A.n_act = c.n_act, A.xcap = c.xcap, A.ycap = c.ycap, A.once = P.tok_blocks == 1, A.counts = c.counts;
  // Early weights get in the way of the conversion's loads where that has many rows (Q8_0 4096 x 4096 by 509 22.7 -> 23.4
  // us), and clusters gain nothing (Q4_K 4096 x 4096 by 8 8.2 -> 8.4); else 14336 x 4096 by 8 13.8 -> 13.1, IQ4_XS by 37
  // 16.7 -> 15.9.
  A.ahead = P.cg == 1 && !c.counts && P.cs == 1 && c.m < 64 ? 2u : 0u;
  if constexpr (T == QK_T_Q4_K)
    if (c.wide) return launch_wide_q4k(P, A, x16, c, beside, s);
  if constexpr (T == QK_T_Q6_K)
    if (c.wide) return launch_wide_q6k(P, A, x16, c, beside, s);
  return launch_matmul<T>(P, A, x16, c, beside, s);
}

}  // namespace qktc

// One translation unit per format.
#define QK_TC_DEFINE(NAME, T)                                                                                          \
  cudaError_t qk_tc_##NAME##_launch(const QkTcCall &c, unsigned *status, unsigned char *scratch, int sm_count, cudaStream_t s) { \
    return qktc::launch_fmt<T>(c, status, scratch, sm_count, s);                                                      \
  }

// Mixture-of-experts projections for a handful of tokens: the decode kernel (qk_gemv_skel.cuh) over
// the experts that were hit, in one launch, sized by the routing on the device.
//
// A *job* is one expert and one or two of the (token, slot) rows routed to it (the plan kernel of
// qk_moe.cu makes the list).  All jobs' 8-row chunks form one sequence; every CTA takes a contiguous
// run of it, cut by cost (a chunk for two rows counts 3, for one row 2: the measured ratio of the
// decode kernel), so that nearly every CTA stays inside one job and the load is even however the
// tokens fell.  Inside a run everything is as in the decode kernel: bulk copies into a ring of stages
// by a producer warp, groups of compute warps that take chunks in turn, partials through a small ring
// to a reducer warp.  At the end of a job's part the compute warps meet, and the next job's split
// activations (prepared once per row by qk_moe_split_kernel) replace the old ones while the ring goes
// on filling.
//
// DUAL: chunks alternate between the gate and the up matrix and the reducer writes silu(gate) * up.
//
// Before, the host read the counts back and ran six launches per expert: 8 experts of 14336 x 4096,
// three tokens, 250 us against 71 us of weight stream.
#pragma once
#include "qk_gemv_skel.cuh"
#include "qk_moe_plan.cuh"

namespace qkdec {

struct MoeArgs {
  QkLayout L;
  const uint8_t *w[2 * QK_MOE_MAX];  // gate (or the only) matrices, then the up matrices from QK_MOE_MAX on
  const QkMoeJobs *jobs;
  const unsigned char *img;          // split rows; row = slot / div
  uint64_t img_stride;
  uint32_t div, rows;               // rows: most rows of a job
  uint32_t early;                    // the job list is older than the previous kernel: weights may be fetched before it ends
  float *y;                          // y[slot][row]
  uint64_t ldy;
  unsigned *status;
  SmemMma S;
  uint32_t Kp, stage_bytes, seg, xch;  // seg: byte offset of the CTA's run, xch: of what the lanes of its warps exchange
  int nstage, nslot;
};
// A CTA's run: per job a range of chunks.
struct MoeSeg {
  uint32_t e, rows, slot0, slot1, chunk, n, ord, pad;  // first chunk, chunks, ordinal of the first (in chunks of either matrix)
};

// Rows of activations -> split images.  With PLAN the first block makes the call's plan meanwhile.
template <class F, bool PLAN>
__global__ void __launch_bounds__(256)
    qk_moe_split_kernel(const float *__restrict__ x, uint32_t rows, uint32_t cols, uint32_t Kp, uint32_t PS,
                        unsigned char *__restrict__ img, uint64_t stride, const qkmoe::PlanArgs P) {
  pdl_launch_dependents();
  pdl_wait();
  if (PLAN && blockIdx.x == 0) {
    qkmoe::plan_block(P);
    return;
  }
  const uint32_t quads = Kp / 4, it = (blockIdx.x - (PLAN ? 1u : 0u)) * 256 + threadIdx.x;
  if (it >= rows * quads) return;  // warp-uniform: quads is a multiple of 64
  const uint32_t r = it / quads, e0 = (it % quads) * 4;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = (e0 + i < cols) ? __ldg(x + (uint64_t)r * cols + e0 + i) : 0.f;
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  float s4 = (v[0] + v[1]) + (v[2] + v[3]);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
  s4 += __shfl_xor_sync(0xffffffffu, s4, 2);
  const float other = __shfl_xor_sync(0xffffffffu, s4, 4);
  const float inv = digit_inv(amax);
  uint32_t w0, w1, w2;
  split_quad(v, inv, w0, w1, w2);
  unsigned char *row = img + (uint64_t)r * stride;
  F::store_digits(row, PS, e0, w0, w1, w2);
  if ((threadIdx.x & 7) == 0) F::store_xs(row + 3 * PS, e0 / 32, digit_scale(amax, s4 + other), s4 + other, s4, other);
}

// F1: the policy of jobs with one row: F, or its variant for them.  BY_TILE: chunks of several k-tiles, whose stages are handed
// back one by one, as in the decode kernel.
template <class F, class F1, bool DUAL, int G, bool BY_TILE>
__global__ void __launch_bounds__((MAX_CW + 2) * 32, 1) qk_gemv_moe_kernel(const __grid_constant__ MoeArgs A) {
  constexpr int CW = MAX_CW, WG = CW / G;
  constexpr uint32_t ND = DUAL ? 2 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  const QkLayout &L = A.L;
  const SmemMma &S = A.S;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nstage = A.nstage, nslot = A.nslot;
  MoeSeg *segs = reinterpret_cast<MoeSeg *>(smem + A.seg);
  volatile uint32_t *meta = reinterpret_cast<volatile uint32_t *>(smem + A.seg + QK_MOE_JOBS * sizeof(MoeSeg));  // segments, chunks

  constexpr bool by_tile = BY_TILE;
  if (A.early) pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < nstage; s++) mbar_init(sbase + S.full + s * 8, 1);
    if (by_tile)
      for (int s = 0; s < nstage; s++) mbar_init(sbase + S.empty + s * 8, WG);
    for (int s = 0; s < nslot; s++) mbar_init(sbase + S.redfull + s * 8, WG);
    mbar_init(sbase + S.xbar, 1);
    *reinterpret_cast<volatile uint32_t *>(smem + S.prog) = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (!A.early) {
    pdl_wait();  // the job list is the previous kernel's work
    pdl_launch_dependents();  // (from here on a later kernel may rely on the list)
  }
  if (warp == 0) {
    // Lane j holds job j; its cost, the prefix sum, this CTA's share of the total.
    const volatile uint32_t *jl = reinterpret_cast<const volatile uint32_t *>(A.jobs);
    const uint32_t n = jl[0];
    uint32_t e = 0, rows = 0, s0 = 0, s1 = 0;
    if (lane < n) e = jl[4 + 4 * lane], rows = jl[5 + 4 * lane], s0 = jl[6 + 4 * lane], s1 = jl[7 + 4 * lane];
    const uint32_t unit = rows == 2 ? 3u : 2u, cost = lane < n ? unit * L.chunks : 0u;
    uint32_t end = cost;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= (uint32_t)o) end += v;
    }
    const uint32_t begin = end - cost, total = __shfl_sync(0xffffffffu, end, 31);
    const uint32_t p0 = (uint32_t)((uint64_t)blockIdx.x * total / gridDim.x), p1 = (uint32_t)((uint64_t)(blockIdx.x + 1) * total / gridDim.x);
    // the chunks whose first cost unit lies in [p0, p1)
    const uint32_t lo = min(max(p0, begin), end) - begin, hi = min(max(p1, begin), end) - begin;
    const uint32_t c0 = (lo + unit - 1) / unit, c1 = (hi + unit - 1) / unit, mine = c1 - c0;
    const uint32_t has = __ballot_sync(0xffffffffu, mine != 0);
    uint32_t ord = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, ord, o);
      if (lane >= (uint32_t)o) ord += v;
    }
    if (mine) segs[__popc(has & ((1u << lane) - 1u))] = {e, rows, s0, s1, c0, mine, (ord - mine) * ND, 0};
    if (lane == 31) meta[0] = __popc(has), meta[1] = ord * ND;
  }
  __syncthreads();
  const uint32_t n_seg = meta[0], n_chunks = meta[1];

  if (warp == CW + 1) {
    // ================= producer warp =================
    const uint32_t lead = elect_lead();
    const uint32_t my_items = __shfl_sync(0xffffffffu, n_chunks, 0) * L.ktiles;
    uint32_t sg = 0, left = 0, which = 0, pkt = 0, pst = 0, item = 0;
    const uint8_t *W0 = nullptr, *W1 = nullptr;  // the next chunk in the gate (or only) and the up matrix
    const uint64_t policy = stream_policy();
    auto issue = [&]() {  // the whole warp
      if (left == 0) {
        const MoeSeg &q = segs[sg++];
        const uint32_t e = __shfl_sync(0xffffffffu, q.e, 0), c0 = __shfl_sync(0xffffffffu, q.chunk, 0);
        left = __shfl_sync(0xffffffffu, q.n, 0);
        W0 = A.w[e] + (uint64_t)c0 * L.chunk_bytes;
        if (DUAL) W1 = A.w[e + QK_MOE_MAX] + (uint64_t)c0 * L.chunk_bytes;
      }
      const uint32_t bytes = QK_TILE_ROWS * qk_tile_nb(L, pkt) * L.bb;
      stream_tile(sbase + S.stage + pst * A.stage_bytes, (which ? W1 : W0) + pkt * L.tile_bytes, bytes, sbase + S.full + pst * 8, policy, lead);
      if (++pkt == L.ktiles) {
        pkt = 0;
        if (++which == ND) which = 0, left--, W0 += L.chunk_bytes, W1 += L.chunk_bytes;
      }
      if (++pst == (uint32_t)nstage) pst = 0;
    };
    auto issue_upto = [&](uint32_t limit) {
      const uint32_t end = limit < my_items ? limit : my_items;
      for (; item < end; item++) issue();
    };
    issue_upto((uint32_t)nstage);
    const volatile uint32_t *prog = reinterpret_cast<const volatile uint32_t *>(smem + S.prog);
    bool alive = true;
    if (!by_tile) {
      uint32_t slot = 0, sph = 0;
      for (uint32_t c = 0; c < n_chunks && item < my_items; c++) {
        alive = mbar_wait_bounded(sbase + S.redfull + slot * 8, sph)  // chunk c handed over
                && wait_read(prog, c);                                // the reducer has read the chunks before c
        if (!alive) break;
        issue_upto(item + L.ktiles);
        if (++slot == (uint32_t)nslot) slot = 0, sph ^= 1;
      }
    } else {  // tile by tile, as in the decode kernel (8 Q4_K experts of 4096 x 14336, three tokens 112.8 -> 107.0 us a layer)
      uint32_t est = 0, eph = 0, c = (uint32_t)nstage / L.ktiles;  // the chunk that the next tile belongs to
      while (alive && item < my_items) {
        alive = mbar_wait_bounded(sbase + S.empty + est * 8, eph) && (pkt || c < (uint32_t)nslot || wait_read(prog, c + 1 - nslot));
        if (!alive) break;
        issue_upto(item + 1);
        if (pkt == 0) c++;
        if (++est == (uint32_t)nstage) est = 0, eph ^= 1;
      }
    }
    if (!alive && lane == 0) atomicOr(A.status, QK_DEV_TIMEOUT);
    return;
  }

  if (warp == CW) {
    // ================= reducer warp =================
    pdl_wait();  // y belongs to the previous kernel until it has finished
    uint32_t slot = 0, sph = 0, sg = 0, c = 0;
    bool dead = false;
    for (; sg < n_seg && !dead; sg++) {
      const MoeSeg q = segs[sg];
      const uint32_t m = lane >> 3, r = lane & 7u;  // lane (m, r) of the first 8 q.rows lanes: row r of activation row m
      float *yr = A.y + (uint64_t)(m ? q.slot1 : q.slot0) * A.ldy;
      float gate_v = 0.f;
      for (uint32_t i = 0; i < q.n * ND; i++, c++) {
        if (!mbar_wait_bounded(sbase + S.redfull + slot * 8, sph)) {
          if (lane == 0) atomicOr(A.status, QK_DEV_TIMEOUT);
          dead = true;
          break;
        }
        const float *red = reinterpret_cast<const float *>(smem + S.red) + slot * (WG * A.rows * 8);
        if (lane < 8 * q.rows) {
          float v = 0.f;
#pragma unroll
          for (int wv = 0; wv < WG; wv++) v += red[(wv * A.rows + m) * 8 + r];
          const uint32_t row = (q.chunk + i / ND) * 8 + r;
          if (DUAL && (i & 1u) == 0) {
            gate_v = v;
          } else if (row < L.rows) {
            if (DUAL) {  // moe.rs:96-112, each step rounded
              const float sg_ = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-gate_v)));
              v = __fmul_rn(v, __fmul_rn(gate_v, sg_));
            }
            yr[row] = v;
          }
        }
        __syncwarp();
        if (lane == 0) *reinterpret_cast<volatile uint32_t *>(smem + S.prog) = c + 1u;  // read: its slot may be written again
        if (++slot == (uint32_t)nslot) slot = 0, sph ^= 1;
      }
    }
    return;
  }

  // ================= compute warps =================
  const uint32_t group = warp / WG, wl = warp % WG;
  const uint32_t g = lane >> 2, tig = lane & 3;
  typename F1::Lane LN;  // (F's with what F1 needs besides)
  LN.init(lane, wl, sbase + S.ximg, S.PS, S.xs_off, A.Kp);
  if constexpr (F1::XCH != 0) LN.set_exchange(sbase + A.xch + warp * F1::XCH, lane);
  pdl_wait();  // the split rows are the previous kernel's work
  uint32_t st = 0, fph = 0, slot = group % nslot;  // next stage and its parity, partial slot of this group's next chunk
  auto skip = [&](uint32_t n) {
    st += n;
    while (st >= (uint32_t)nstage) st -= nstage, fph ^= 1;
  };
  skip(group * L.ktiles);
  bool dead = false;
  uint32_t c = group;  // this group's next chunk
  for (uint32_t sg = 0; sg < n_seg; sg++) {
    const MoeSeg *q = segs + sg;
    const uint32_t rows = q->rows, end = q->ord + q->n * ND;
    if (sg) asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");  // everybody is done with the previous rows
    if (warp == 0 && lane == 0) {
      const uint32_t dig_bytes = 3 * S.PS, xs_bytes = A.Kp / 32 * F::XSB;
      mbar_expect_tx(sbase + S.xbar, rows * (dig_bytes + xs_bytes));
      for (uint32_t m = 0; m < rows; m++) {
        const unsigned char *row = A.img + (uint64_t)((m ? q->slot1 : q->slot0) / A.div) * A.img_stride;
        bulk_g2s(sbase + S.ximg + m * dig_bytes, row, dig_bytes, sbase + S.xbar);
        bulk_g2s(sbase + S.ximg + S.xs_off + m * xs_bytes, row + dig_bytes, xs_bytes, sbase + S.xbar);
      }
    }
    if (!mbar_wait_bounded(sbase + S.xbar, sg & 1u)) dead = true;  // (the wait of the copies in flight, too)
    auto run = [&](auto mtag) {
      constexpr int M = decltype(mtag)::value;
      using P = std::conditional_t<M == 1, F1, F>;
      using Data = typename P::template Data<M>;
      for (; c < end && !dead; c += G) {
        float acc[M][3];
#pragma unroll
        for (int m = 0; m < M; m++) acc[m][0] = acc[m][1] = acc[m][2] = 0.f;
        for (uint32_t kt = 0; kt < L.ktiles; kt++) {
          const uint32_t nbt = qk_tile_nb(L, kt) * L.bs / 256u;  // 256-column spans in this tile
          const uint32_t tile = sbase + S.stage + st * A.stage_bytes;
          if (!mbar_wait_bounded(sbase + S.full + st * 8, fph)) {
            dead = true;
            break;
          }
          const typename P::Base B = P::base(LN, tile, kt);
          auto tile_body = [&](auto full_tag) {
            constexpr bool FULL = decltype(full_tag)::value;
            constexpr int NSB = NBT / WG;
            static_for<0, NSB>([&](auto jt) {
              constexpr int J = decltype(jt)::value;
              if (FULL || wl + J * WG < nbt) {
                Data D;
                P::template load<M, J, WG>(D, B, LN);
                P::template compute<M>(D, LN, acc);
              }
            });
          };
          if (nbt == NBT) tile_body(std::true_type{});
          else tile_body(std::false_type{});
          if (by_tile) {
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + S.empty + st * 8);
          }
          if (++st == (uint32_t)nstage) st = 0, fph ^= 1;
        }
        if (dead) break;
        float *red = reinterpret_cast<float *>(smem + S.red) + slot * (WG * A.rows * 8);
#pragma unroll
        for (int m = 0; m < M; m++) {
          float v = F::finish(acc[m], LN);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (tig == 0) red[(wl * A.rows + m) * 8 + g] = v;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(sbase + S.redfull + slot * 8);
        slot += G;
        while (slot >= (uint32_t)nslot) slot -= nslot;
        skip((G - 1) * L.ktiles);
      }
    };
    if (!dead) {
      if (rows == 1) run(std::integral_constant<int, 1>{});
      else run(std::integral_constant<int, 2>{});
    }
  }
  if (dead) atomicOr(A.status, QK_DEV_TIMEOUT);  // a bounded wait ran out: results are invalid
}

struct PlanMoe {
  PlanMma P;
  uint32_t seg, total;
};
// The decode kernel's plan for `rows` activation rows; the run table goes behind the ring.
inline bool make_plan_moe(const QkLayout &L, uint32_t rows, uint32_t xsb, PlanMoe *p) {
  if (!make_plan_mma(L, rows, &p->P, xsb)) return false;
  const uint32_t table = QK_MOE_JOBS * sizeof(MoeSeg) + 16;
  // (the plan leaves 1 KB of the budget unused; the table takes a stage's place where it does not fit)
  while (p->P.total + table > 227u * 1024u) {
    const int unit = p->P.groups * (int)L.ktiles;
    if (p->P.nstage - unit < (int)L.ktiles + 1 || p->P.nstage - unit < unit) return false;
    p->P.nstage -= unit, p->P.nslot = p->P.nstage + 1, p->P.total -= unit * p->P.stage_bytes;
  }
  p->seg = p->P.total, p->total = p->P.total + table;
  return true;
}

template <class F>
size_t moe_image_stride(const QkLayout &L) {
  const size_t Kp = (size_t)L.nb * L.bs;
  return 3 * (Kp + 64) + Kp / 32 * F::XSB;
}

template <class F>
uint32_t moe_rows(const QkLayout &L) {  // activation rows a job may have: 2, 1 or 0 (not served)
  PlanMoe p;
  if (L.rows == 0 || L.cols == 0) return 0;
  return make_plan_moe(L, 2, F::XSB, &p) ? 2 : make_plan_moe(L, 1, F::XSB, &p) ? 1 : 0;
}

template <class F>
cudaError_t moe_split(const QkLayout &L, const float *x, uint32_t rows, unsigned char *img, const qkmoe::PlanArgs *plan, cudaStream_t s) {
  const uint32_t Kp = L.nb * L.bs;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((rows * (Kp / 4) + 255) / 256 + (plan ? 1 : 0)), c.blockDim = dim3(256), c.stream = s, c.attrs = at, c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, plan ? qk_moe_split_kernel<F, true> : qk_moe_split_kernel<F, false>, x, rows, L.cols, Kp, Kp + 64, img,
                            (uint64_t)moe_image_stride<F>(L), plan ? *plan : qkmoe::PlanArgs{});
}

template <class F, class F1, bool DUAL, int G, bool BY_TILE>
cudaError_t moe_launch_t(const MoeArgs &A, uint32_t smem, int sm_count, cudaStream_t s) {
  auto kern = qk_gemv_moe_kernel<F, F1, DUAL, G, BY_TILE>;
  static QkPerDevice attr_set;
  if (attr_set.first()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return attr_set.reset(), e;
  }
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)sm_count), c.blockDim = dim3((MAX_CW + 2) * 32), c.dynamicSmemBytes = smem, c.stream = s, c.attrs = at, c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, A);
}

// Two kernels.  (As in launch_mma, the hand-overs that rows of a single k-tile never come to move the allocation as a condition
// in the loop.  us a layer of experts, with the condition / a kernel each: 8 Q6_K of 2048 x 4096, top 2, two tokens 35.7 / 34.0, 16
// of 1024 x 1536, top 3, eight 57.6 / 54.3, Q4_K 2048 x 2048, top 1, five 30.2 / 28.7; 0.98 to 1.00 over the formats.)
template <class F, class F1, bool DUAL, int G>
cudaError_t moe_launch_g(const MoeArgs &A, uint32_t smem, int sm_count, cudaStream_t s) {
  return A.L.ktiles > 1 && A.rows <= F::BY_TILE_M ? moe_launch_t<F, F1, DUAL, G, true>(A, smem, sm_count, s)
                                                  : moe_launch_t<F, F1, DUAL, G, false>(A, smem, sm_count, s);
}

template <class P>
struct MoePolicy { using type = P; };
// rows_per_job: what the job list was made for (at most moe_rows(L)).  F1: the policy for jobs with one row, where its
// exchange fits behind the run table (else F itself).
template <class F, class F1>
cudaError_t moe_launch(const QkLayout &L, const uint8_t *const *w, const uint8_t *const *w2, uint32_t n, uint32_t rows_per_job,
                       const QkMoeJobs *jobs, const unsigned char *img, uint32_t div, float *y, uint64_t ldy, unsigned *status,
                       int sm_count, cudaStream_t s) {
  PlanMoe p;
  if (n > QK_MOE_MAX || !make_plan_moe(L, rows_per_job, F::XSB, &p)) return cudaErrorInvalidConfiguration;
  MoeArgs A = {};
  A.L = L, A.jobs = jobs, A.img = img, A.img_stride = moe_image_stride<F>(L), A.div = div, A.rows = rows_per_job, A.early = w2 == nullptr;
  for (uint32_t e = 0; e < n; e++) A.w[e] = w[e], A.w[QK_MOE_MAX + e] = w2 ? w2[e] : nullptr;
  A.y = y, A.ldy = ldy, A.status = status, A.S = p.P.S, A.Kp = p.P.Kp, A.stage_bytes = p.P.stage_bytes, A.seg = p.seg;
  A.nstage = p.P.nstage, A.nslot = p.P.nslot;
  A.xch = (p.total + 127u) & ~127u;
  auto launch = [&](auto policy) {
    using P1 = typename decltype(policy)::type;
    const uint32_t total = P1::XCH ? A.xch + MAX_CW * P1::XCH : p.total;
    switch (p.P.groups) {
      case 4:
        return w2 ? moe_launch_g<F, P1, true, 4>(A, total, sm_count, s) : moe_launch_g<F, P1, false, 4>(A, total, sm_count, s);
      case 2:
        return w2 ? moe_launch_g<F, P1, true, 2>(A, total, sm_count, s) : moe_launch_g<F, P1, false, 2>(A, total, sm_count, s);
      default:
        return w2 ? moe_launch_g<F, P1, true, 1>(A, total, sm_count, s) : moe_launch_g<F, P1, false, 1>(A, total, sm_count, s);
    }
  };
  if constexpr (F1::XCH != 0)
    if (A.xch + MAX_CW * F1::XCH <= 227u * 1024u) return launch(MoePolicy<F1>{});
  return launch(MoePolicy<F>{});
}

}  // namespace qkdec

#define QK_MOE_DEC_DEFINE(NAME, F, F1)                                                                                       \
  uint32_t qk_moe_dec_##NAME##_rows(const QkLayout &L) { return qkdec::moe_rows<F>(L); }                                 \
  size_t qk_moe_dec_##NAME##_image(const QkLayout &L) { return qkdec::moe_image_stride<F>(L); }                          \
  cudaError_t qk_moe_dec_##NAME##_split(const QkLayout &L, const float *x, uint32_t rows, unsigned char *img, \
                                        const qkmoe::PlanArgs *plan, cudaStream_t s) {                                   \
    return qkdec::moe_split<F>(L, x, rows, img, plan, s);                                                                      \
  }                                                                                                                      \
  cudaError_t qk_moe_dec_##NAME##_launch(const QkLayout &L, const uint8_t *const *w, const uint8_t *const *w2, uint32_t n, \
                                         uint32_t rows_per_job, const QkMoeJobs *jobs, const unsigned char *img,         \
                                         uint32_t div, float *y, uint64_t ldy, unsigned *status, int sm_count, cudaStream_t s) { \
    return qkdec::moe_launch<F, F1>(L, w, w2, n, rows_per_job, jobs, img, div, y, ldy, status, sm_count, s);                  \
  }

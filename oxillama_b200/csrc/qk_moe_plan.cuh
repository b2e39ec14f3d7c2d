// Routing of a mixture-of-experts layer on the device (crates/oxillama-arch/src/common/moe.rs:200-248), and the
// plan of a call with a handful of tokens.
#pragma once
#include "qk_kernels.h"

namespace qkmoe {

// One thread per token: softmax over all experts, the top_k largest in descending order
// (equal values keep ascending expert order, as a stable sort would), weights
// renormalised by the selected sum (moe.rs:200-248).
__device__ __forceinline__ void route_token(const float *__restrict__ logits, uint32_t t, uint32_t n_exp, uint32_t top_k,
                                            int *ids, float *wts) {
  const float *l = logits + (uint64_t)t * n_exp;
  const uint32_t ek = top_k < n_exp ? top_k : n_exp;
  float mx = -INFINITY;
  for (uint32_t i = 0; i < n_exp; i++) mx = fmaxf(mx, l[i]);
  float es = 0.f;
  for (uint32_t i = 0; i < n_exp; i++) es = __fadd_rn(es, expf(__fsub_rn(l[i], mx)));
  auto prob = [&](uint32_t i) {
    const float e = expf(__fsub_rn(l[i], mx));
    return es > 0.f ? __fdiv_rn(e, es) : __fdiv_rn(1.f, (float)n_exp);
  };
  float ssum = 0.f;
  for (uint32_t k = 0; k < ek; k++) {  // k-th largest not yet taken; ties to the lower index
    float best = -1.f;
    uint32_t bi = 0;
    for (uint32_t i = 0; i < n_exp; i++) {
      bool taken = false;
      for (uint32_t j = 0; j < k; j++) taken |= ids[(uint64_t)t * top_k + j] == (int)i;
      const float p = prob(i);
      if (!taken && p > best) best = p, bi = i;
    }
    ids[(uint64_t)t * top_k + k] = (int)bi;
    wts[(uint64_t)t * top_k + k] = best;
    ssum = __fadd_rn(ssum, best);
  }
  for (uint32_t k = 0; k < ek; k++) {
    float &w = wts[(uint64_t)t * top_k + k];
    w = ssum > 1e-9f ? __fdiv_rn(w, ssum) : __fdiv_rn(1.f, (float)ek);
  }
  for (uint32_t k = ek; k < top_k; k++) ids[(uint64_t)t * top_k + k] = -1, wts[(uint64_t)t * top_k + k] = 0.f;
}

// The same by one warp, a lane per expert (n_exp <= 32): the same sums in the same order, without the
// chain of loads that one thread would walk (three tokens, eight experts: 7 -> 3 us for the plan).
__device__ __forceinline__ void route_token_warp(const float *__restrict__ logits, uint32_t t, uint32_t n_exp, uint32_t top_k,
                                                 uint32_t lane, int *ids, float *wts) {
  const uint32_t ek = top_k < n_exp ? top_k : n_exp;
  const float l = lane < n_exp ? logits[(uint64_t)t * n_exp + lane] : -INFINITY;
  float mx = l;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float e = lane < n_exp ? expf(__fsub_rn(l, mx)) : 0.f;
  float es = 0.f;
  for (uint32_t i = 0; i < n_exp; i++) es = __fadd_rn(es, __shfl_sync(0xffffffffu, e, i));
  const float p = es > 0.f ? __fdiv_rn(e, es) : __fdiv_rn(1.f, (float)n_exp);
  bool taken = lane >= n_exp;
  float ssum = 0.f, mine = 0.f;
  for (uint32_t k = 0; k < ek; k++) {
    // the largest not yet taken, ties to the lower expert; as in the scan, a value that is not above -1 (a NaN) is never taken
    float best = !taken && p > -1.f ? p : -1.f;
    uint32_t bi = best > -1.f ? lane : 0xFFFFFFFFu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) best = ob, bi = oi;
    }
    if (bi == 0xFFFFFFFFu) bi = 0;
    if (lane == bi) taken = true;
    if (lane == k) mine = best, ids[(uint64_t)t * top_k + k] = (int)bi;
    ssum = __fadd_rn(ssum, best);
  }
  if (lane < ek) wts[(uint64_t)t * top_k + lane] = ssum > 1e-9f ? __fdiv_rn(mine, ssum) : __fdiv_rn(1.f, (float)ek);
  for (uint32_t k = ek + lane; k < top_k; k += 32) ids[(uint64_t)t * top_k + k] = -1, wts[(uint64_t)t * top_k + k] = 0.f;
}

// The same by one thread that holds the logits and probabilities of up to E experts in registers: the same sums in
// the same order, without the loads and the second exponentials of route_token.  Calls store(k, id, weight).
template <int E, class Store>
__device__ __forceinline__ void route_token_regs(const float *__restrict__ logits, uint32_t t, uint32_t n_exp, uint32_t top_k, Store &&store) {
  const float *l = logits + (uint64_t)t * n_exp;
  const uint32_t ek = top_k < n_exp ? top_k : n_exp;
  float p[E], mx = -INFINITY, es = 0.f;
#pragma unroll
  for (int i = 0; i < E; i++) p[i] = i < (int)n_exp ? __ldg(l + i) : -INFINITY;
#pragma unroll
  for (int i = 0; i < E; i++) mx = fmaxf(mx, p[i]);
#pragma unroll
  for (int i = 0; i < E; i++) {
    p[i] = expf(__fsub_rn(p[i], mx));
    if (i < (int)n_exp) es = __fadd_rn(es, p[i]);
  }
#pragma unroll
  for (int i = 0; i < E; i++) p[i] = es > 0.f ? __fdiv_rn(p[i], es) : __fdiv_rn(1.f, (float)n_exp);
  // the largest not yet taken, ties to the lower expert (every p compares: where a logit is NaN or infinite, es is NaN and
  // all are 1 / n_exp)
  uint32_t taken = n_exp < 32 ? ~0u << n_exp : 0u;
  auto next = [&](float &best) {
    uint32_t bi = 0;
    best = -1.f;
#pragma unroll
    for (int i = 0; i < E; i++)
      if (!(taken >> i & 1u) && p[i] > best) best = p[i], bi = (uint32_t)i;
    taken |= 1u << bi;
    return bi;
  };
  const uint32_t all = taken;
  float ssum = 0.f, best;
  for (uint32_t k = 0; k < ek; k++) next(best), ssum = __fadd_rn(ssum, best);
  taken = all;
  for (uint32_t k = 0; k < ek; k++) {
    const uint32_t id = next(best);
    store(k, (int)id, ssum > 1e-9f ? __fdiv_rn(best, ssum) : __fdiv_rn(1.f, (float)ek));
  }
  for (uint32_t k = ek; k < top_k; k++) store(k, -1, 0.f);
}

// Everything the projections of a handful of tokens need to know, by one block of 256 threads: ids and
// weights, the lists of the experts with many rows, the job list of the others.
struct PlanArgs {
  const float *logits;
  uint32_t tokens, n_exp, top_k, expert_begin, n_local, rows_per_job;
  int *ids;
  float *wts;
  int *big, *lists, *pos;
  QkMoeJobs *jobs;
};
__device__ __forceinline__ void plan_block(const PlanArgs &A) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (A.n_exp <= 32 && A.top_k <= 32) {
    for (uint32_t t = warp; t < A.tokens; t += 8) route_token_warp(A.logits, t, A.n_exp, A.top_k, lane, A.ids, A.wts);
  } else if (threadIdx.x < A.tokens) {
    route_token(A.logits, threadIdx.x, A.n_exp, A.top_k, A.ids, A.wts);
  }
  __syncthreads();
  if (warp) return;
  const uint32_t n = A.tokens * A.top_k;
  uint32_t count = 0, first[QK_MOE_DEC_ROWS] = {};
  const int want = lane < A.n_local ? (int)(A.expert_begin + lane) : -2;
  for (uint32_t base = 0; base < n; base += 32) {
    const int id = base + lane < n ? A.ids[base + lane] : -1;
    for (uint32_t j = 0; j < 32 && base + j < n; j++) {
      if (__shfl_sync(0xffffffffu, id, j) != want) continue;
      const uint32_t i = base + j;
#pragma unroll
      for (uint32_t k = 0; k < QK_MOE_DEC_ROWS; k++)
        if (k == count) first[k] = i;
      A.lists[lane * n + count] = (int)i;
      A.pos[i] = (int)count++;
    }
  }
  if (lane < A.n_local) A.big[lane] = count > QK_MOE_DEC_ROWS ? (int)count : 0;
  const uint32_t mine = count > QK_MOE_DEC_ROWS ? 0u : (count + A.rows_per_job - 1) / A.rows_per_job;
  uint32_t end = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= (uint32_t)o) end += v;
  }
  if (lane == 31) A.jobs->n = end;
#pragma unroll
  for (uint32_t k = 0; k < QK_MOE_DEC_ROWS; k++) {
    if (k % A.rows_per_job || k >= count || !mine) continue;
    const bool two = A.rows_per_job == 2 && k + 1 < count;
    auto &j = A.jobs->job[end - mine + k / A.rows_per_job];
    j.expert = lane, j.rows = two ? 2u : 1u, j.slot[0] = first[k], j.slot[1] = two ? first[k + 1 < QK_MOE_DEC_ROWS ? k + 1 : k] : 0u;
  }
}

}  // namespace qkmoe

// Mixture-of-experts FFN around the quantized matmuls (crates/oxillama-arch/src/common/moe.rs:184-258):
// routing, the per-expert token lists, and the element-wise steps between the three
// matmuls of an expert (moe.rs:75-126).  The matmuls themselves are the ordinary dequant-matmul
// kernels: one grouped launch per projection over all local experts, on the decode kernels
// (qk_gemv_moe.cuh) for a handful of tokens, else on the tensor cores.
#include <cfloat>

#include "qk_kernels.h"
#include "qk_moe_plan.cuh"
#include "qk_pipe.cuh"

using namespace qkpipe;

namespace {

cudaLaunchAttribute pdl_attr() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

__global__ void __launch_bounds__(128)
    qk_moe_route_kernel(const float *__restrict__ logits, uint32_t tokens, uint32_t n_exp,
                        uint32_t top_k, int *__restrict__ ids, float *__restrict__ wts) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < tokens) qkmoe::route_token(logits, t, n_exp, top_k, ids, wts);
}

// One warp per local expert: the (token, slot) pairs routed to it, in token order.
__global__ void __launch_bounds__(32)
    qk_moe_lists_kernel(const int *__restrict__ ids, uint32_t tokens, uint32_t top_k,
                        uint32_t expert_begin, int *__restrict__ counts, int *__restrict__ lists,
                        int *__restrict__ pos) {
  const uint32_t e = blockIdx.x, lane = threadIdx.x;
  const int want = (int)(expert_begin + e);
  const uint64_t n = (uint64_t)tokens * top_k;
  uint32_t count = 0;
  for (uint64_t base = 0; base < n; base += 32) {
    const uint64_t i = base + lane;
    const bool hit = i < n && ids[i] == want;
    const uint32_t mask = __ballot_sync(0xffffffffu, hit);
    if (hit) {
      const uint32_t p = count + __popc(mask & ((1u << lane) - 1u));
      lists[(uint64_t)e * n + p] = (int)i;
      if (pos) pos[i] = (int)p;  // where (token, slot) i sits in its expert's list
    }
    count += __popc(mask);
  }
  if (lane == 0) counts[e] = (int)count;
}

// Routing and lists in one block: up to QK_MOE_PLAN_SLOTS (token, slot) pairs, 32 experts, 16 of them local.  A thread
// routes a token; then the block goes through the pairs 1024 at a time: a pair's place in its expert's list is the pairs
// of that expert in the blocks before, in the warps before and in the lanes before.  Bound by its latencies; as two
// launches without programmatic dependency (a thread per token that reads its logits again for every comparison, then a
// warp per expert that walks all pairs) 256 tokens, 8 experts took 6.4 + 7.4 us under ncu; together with the packed
// conversion rows (conv_row) the layer of 8 IQ4_XS experts of 4096 x 14336, 256 tokens top 2, 335.2 -> 323.7.
__global__ void __launch_bounds__(1024)
    qk_moe_group_plan_kernel(const float *__restrict__ logits, uint32_t tokens, uint32_t n_exp, uint32_t top_k,
                             uint32_t expert_begin, uint32_t n_local, int *__restrict__ ids, float *__restrict__ wts,
                             int *__restrict__ counts, int *__restrict__ lists, int *__restrict__ pos) {
  __shared__ signed char local[QK_MOE_PLAN_SLOTS];  // local expert of a pair, -1: none
  __shared__ uint32_t ahead[QK_MOE_MAX][33];        // pairs of an expert in the warps before, of this round
  __shared__ uint32_t total[QK_MOE_MAX];
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t n = tokens * top_k, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < QK_MOE_MAX) total[threadIdx.x] = 0;
  for (uint32_t t = threadIdx.x; t < tokens; t += 1024) {
    auto store = [&](uint32_t k, int id, float w) {
      const uint32_t i = t * top_k + k, e = (uint32_t)(id - (int)expert_begin);
      ids[i] = id, wts[i] = w, local[i] = id >= 0 && e < n_local ? (signed char)e : (signed char)-1;
    };
    if (n_exp <= 8) qkmoe::route_token_regs<8>(logits, t, n_exp, top_k, store);
    else qkmoe::route_token_regs<32>(logits, t, n_exp, top_k, store);
  }
  for (uint32_t base = 0; base < n; base += 1024) {
    if (warp < QK_MOE_MAX) ahead[warp][lane] = 0;
    __syncthreads();
    const uint32_t i = base + threadIdx.x;
    const int e = i < n ? local[i] : -1;
    const uint32_t same = __match_any_sync(0xffffffffu, e), before = __popc(same & ((1u << lane) - 1u));
    if (e >= 0 && before == 0) ahead[e][warp] = __popc(same);
    __syncthreads();
    if (warp < QK_MOE_MAX) {
      const uint32_t v = ahead[warp][lane];
      uint32_t end = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= (uint32_t)o) end += u;
      }
      const uint32_t t0 = total[warp];
      ahead[warp][lane] = t0 + end - v;
      __syncwarp();
      if (lane == 31) total[warp] = t0 + end;
    }
    __syncthreads();
    if (e >= 0) {
      const uint32_t p = ahead[e][warp] + before;
      lists[(uint64_t)e * n + p] = (int)i, pos[i] = (int)p;
    }
    __syncthreads();
  }
  if (threadIdx.x < n_local) counts[threadIdx.x] = (int)total[threadIdx.x];
}

__global__ void __launch_bounds__(256)
    qk_moe_gather_kernel(const float *__restrict__ x, const int *__restrict__ list, uint32_t n,
                         uint32_t top_k, uint32_t hidden, float *__restrict__ xe) {
  const uint32_t i = blockIdx.x;
  if (i >= n) return;
  const float *src = x + (uint64_t)(list[i] / (int)top_k) * hidden;
  for (uint32_t c = threadIdx.x; c < hidden; c += blockDim.x) xe[(uint64_t)i * hidden + c] = src[c];
}

// u <- silu(g) * u  (moe.rs:96-112: g * sigmoid(g), then times up)
__global__ void __launch_bounds__(256)
    qk_moe_silu_mul_kernel(const float *__restrict__ g, float *__restrict__ u, uint64_t n) {
  for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
    const float v = g[i];
    const float sig = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v)));
    u[i] = __fmul_rn(u[i], __fmul_rn(v, sig));
  }
}

// g <- silu(g) * u: swiglu_inplace (crates/oxillama-arch/src/common/swiglu.rs:15-21), each step rounded
__global__ void __launch_bounds__(256)
    qk_swiglu_kernel(float *__restrict__ g, const float *__restrict__ u, uint64_t n) {
  for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
    const float v = g[i];
    const float sig = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v)));
    g[i] = __fmul_rn(__fmul_rn(v, sig), u[i]);
  }
}

// y[token] += w * o[i]; a token occurs at most once in one expert's list.
__global__ void __launch_bounds__(256)
    qk_moe_scatter_kernel(const float *__restrict__ o, const int *__restrict__ list,
                          const float *__restrict__ wts, uint32_t n, uint32_t top_k, uint32_t hidden,
                          float *__restrict__ y) {
  const uint32_t i = blockIdx.x;
  if (i >= n) return;
  const int slot = list[i];
  const float w = wts[slot];
  float *dst = y + (uint64_t)(slot / (int)top_k) * hidden;
  for (uint32_t c = threadIdx.x; c < hidden; c += blockDim.x)
    dst[c] = __fadd_rn(dst[c], __fmul_rn(w, o[(uint64_t)i * hidden + c]));
}

// y[token] = sum over the token's slots, in slot order, of w[slot] * its expert's output row, for the
// slots whose expert is local (moe.rs:232-255 accumulates in that order); a token none of whose experts
// is local gets zeros.
__global__ void __launch_bounds__(256)
    qk_moe_combine_kernel(const float *__restrict__ o, const float *__restrict__ by_slot, const int *__restrict__ big,
                          const int *__restrict__ ids, const int *__restrict__ pos, const float *__restrict__ wts,
                          uint32_t top_k, uint32_t expert_begin, uint32_t n_local, uint32_t cap, uint32_t hidden,
                          float *__restrict__ y) {
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t t = blockIdx.x, c = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (c >= hidden) return;
  // four columns a thread: where a row is whole quads, those of the scratch are 16-byte aligned; y is the caller's
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t k = 0; k < top_k; k++) {
    const uint32_t slot = t * top_k + k;
    const int id = ids[slot];
    if (id < (int)expert_begin || id >= (int)(expert_begin + n_local)) continue;
    const uint32_t e = (uint32_t)(id - (int)expert_begin);
    const float *row = by_slot && !big[e] ? by_slot + (uint64_t)slot * hidden
                                          : o + ((uint64_t)e * cap + (uint32_t)pos[slot]) * hidden;
    const float w = wts[slot];
    if ((hidden & 3u) == 0) {
      const float4 v = *reinterpret_cast<const float4 *>(row + c);
      acc.x = __fadd_rn(acc.x, __fmul_rn(w, v.x)), acc.y = __fadd_rn(acc.y, __fmul_rn(w, v.y));
      acc.z = __fadd_rn(acc.z, __fmul_rn(w, v.z)), acc.w = __fadd_rn(acc.w, __fmul_rn(w, v.w));
    } else {
      acc.x = __fadd_rn(acc.x, __fmul_rn(w, row[c]));
      if (c + 1 < hidden) acc.y = __fadd_rn(acc.y, __fmul_rn(w, row[c + 1]));
      if (c + 2 < hidden) acc.z = __fadd_rn(acc.z, __fmul_rn(w, row[c + 2]));
      if (c + 3 < hidden) acc.w = __fadd_rn(acc.w, __fmul_rn(w, row[c + 3]));
    }
  }
  float *out = y + (uint64_t)t * hidden + c;
  if ((hidden & 3u) == 0 && ((uintptr_t)y & 15u) == 0) {
    *reinterpret_cast<float4 *>(out) = acc;
  } else {
    out[0] = acc.x;
    if (c + 1 < hidden) out[1] = acc.y;
    if (c + 2 < hidden) out[2] = acc.z;
    if (c + 3 < hidden) out[3] = acc.w;
  }
}

// out[i][:] = x[idx[i]][:]: the rows a rank sends to another rank, in send order.
__global__ void __launch_bounds__(256)
    qk_moe_take_rows_kernel(const float *__restrict__ x, const int *__restrict__ idx, uint32_t width,
                            float *__restrict__ out) {
  const uint64_t src = (uint64_t)(uint32_t)idx[blockIdx.x] * width, dst = (uint64_t)blockIdx.x * width;
  for (uint32_t c = threadIdx.x; c < width; c += 256) out[dst + c] = x[src + c];
}

// y[t][:] = +0 + src[idx[t][0]] + src[idx[t][1]] + ... in that order, entries below zero skipped:
// the partial outputs that came back for token t, in the order of the ranks that made them.
__global__ void __launch_bounds__(256)
    qk_moe_sum_rows_kernel(const float *__restrict__ src, const int *__restrict__ idx, uint32_t per_row,
                           uint32_t width, float *__restrict__ y) {
  const uint32_t t = blockIdx.x;
  for (uint32_t c = threadIdx.x; c < width; c += 256) {
    float acc = 0.f;
    for (uint32_t j = 0; j < per_row; j++) {
      const int r = idx[(uint64_t)t * per_row + j];
      if (r >= 0) acc = __fadd_rn(acc, src[(uint64_t)r * width + c]);
    }
    y[(uint64_t)t * width + c] = acc;
  }
}

}  // namespace

cudaError_t qk_launch_moe_route(const float *logits, uint32_t tokens, uint32_t n_exp, uint32_t top_k,
                                int *ids, float *wts, cudaStream_t s) {
  if (tokens == 0) return cudaSuccess;
  qk_moe_route_kernel<<<(tokens + 127) / 128, 128, 0, s>>>(logits, tokens, n_exp, top_k, ids, wts);
  return cudaGetLastError();
}
cudaError_t qk_launch_moe_lists(const int *ids, uint32_t tokens, uint32_t top_k, uint32_t expert_begin,
                                uint32_t n_local, int *counts, int *lists, int *pos, cudaStream_t s) {
  if (n_local == 0) return cudaSuccess;
  qk_moe_lists_kernel<<<n_local, 32, 0, s>>>(ids, tokens, top_k, expert_begin, counts, lists, pos);
  return cudaGetLastError();
}
cudaError_t qk_launch_moe_group_plan(const float *logits, uint32_t tokens, uint32_t n_exp, uint32_t top_k,
                                     uint32_t expert_begin, uint32_t n_local, int *ids, float *wts, int *counts,
                                     int *lists, int *pos, cudaStream_t s) {
  if (tokens == 0 || n_local == 0) return cudaSuccess;
  if ((uint64_t)tokens * top_k <= QK_MOE_PLAN_SLOTS && n_exp <= 32 && n_local <= QK_MOE_MAX) {
    cudaLaunchAttribute at = pdl_attr();
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(1), c.blockDim = dim3(1024), c.stream = s, c.attrs = &at, c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, qk_moe_group_plan_kernel, logits, tokens, n_exp, top_k, expert_begin, n_local, ids, wts, counts, lists, pos);
  }
  cudaError_t e = qk_launch_moe_route(logits, tokens, n_exp, top_k, ids, wts, s);
  return e != cudaSuccess ? e : qk_launch_moe_lists(ids, tokens, top_k, expert_begin, n_local, counts, lists, pos, s);
}
cudaError_t qk_launch_moe_combine(const float *o, const float *by_slot, const int *big, const int *ids, const int *pos,
                                  const float *wts, uint32_t tokens, uint32_t top_k, uint32_t expert_begin,
                                  uint32_t n_local, uint32_t cap, uint32_t hidden, float *y, cudaStream_t s) {
  if (tokens == 0 || hidden == 0) return cudaSuccess;
  cudaLaunchAttribute at = pdl_attr();
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(tokens, (hidden + 1023) / 1024), c.blockDim = dim3(256), c.stream = s, c.attrs = &at, c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, qk_moe_combine_kernel, o, by_slot, big, ids, pos, wts, top_k, expert_begin, n_local, cap, hidden, y);
}
cudaError_t qk_launch_moe_gather(const float *x, const int *list, uint32_t n, uint32_t top_k,
                                 uint32_t hidden, float *xe, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  qk_moe_gather_kernel<<<n, 256, 0, s>>>(x, list, n, top_k, hidden, xe);
  return cudaGetLastError();
}
cudaError_t qk_launch_moe_silu_mul(const float *g, float *u, uint64_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const uint64_t blocks = (n + 255) / 256;
  qk_moe_silu_mul_kernel<<<(unsigned)(blocks > 148 * 16 ? 148 * 16 : blocks), 256, 0, s>>>(g, u, n);
  return cudaGetLastError();
}
cudaError_t qk_launch_swiglu(float *g, const float *u, uint64_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const uint64_t blocks = (n + 255) / 256;
  qk_swiglu_kernel<<<(unsigned)(blocks > 148 * 16 ? 148 * 16 : blocks), 256, 0, s>>>(g, u, n);
  return cudaGetLastError();
}

cudaError_t qk_launch_moe_scatter(const float *o, const int *list, const float *wts, uint32_t n,
                                  uint32_t top_k, uint32_t hidden, float *y, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  qk_moe_scatter_kernel<<<n, 256, 0, s>>>(o, list, wts, n, top_k, hidden, y);
  return cudaGetLastError();
}

cudaError_t qk_launch_moe_take_rows(const float *x, const int *idx, uint32_t n, uint32_t width, float *out,
                                    cudaStream_t s) {
  if (n == 0 || width == 0) return cudaSuccess;
  qk_moe_take_rows_kernel<<<n, 256, 0, s>>>(x, idx, width, out);
  return cudaGetLastError();
}
cudaError_t qk_launch_moe_sum_rows(const float *src, const int *idx, uint32_t tokens, uint32_t per_row,
                                   uint32_t width, float *y, cudaStream_t s) {
  if (tokens == 0 || width == 0) return cudaSuccess;
  qk_moe_sum_rows_kernel<<<tokens, 256, 0, s>>>(src, idx, per_row, width, y);
  return cudaGetLastError();
}

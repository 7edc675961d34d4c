// Router top-k (noaux_tc) and RMSNorm for sm_100a.
//
// router_topk: one warp per token.  score = sigmoid(logit) (or softmax over the experts); the
// selection runs on score + bias, optionally restricted to the `topk_group` best expert groups
// (group score = sum of the two best biased scores when a bias is given, else the best one); ties
// go to the lower expert id; the returned weights are the unbiased scores of the selected experts,
// renormalised by (sum + 1e-20) and multiplied by the routed scaling factor.  Slot order is
// descending biased score.  Semantics follow moeflow/reference.py:21-62 and moeflow/router.py:10-42.
#include "common.cuh"
#include "moeflow_b200.h"
#include "router.cuh"

namespace mf {

constexpr int kRouterWarps = 4;

__global__ void __launch_bounds__(kRouterWarps * 32)
router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias, float* __restrict__ weights,
                   int* __restrict__ ids, int tokens, RouteParams p) {
  extern __shared__ float sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* score = sm + (size_t)warp * 2 * p.E;
  const int t = blockIdx.x * kRouterWarps + warp;
  if (t >= tokens) return;
  float w;
  int id;
  route_token_warp(logits + (size_t)t * p.E, bias, score, score + p.E, p, lane, w, id);
  if (lane < p.K) {
    weights[(size_t)t * p.K + lane] = w;
    ids[(size_t)t * p.K + lane] = id;
  }
}

// out[r, :] = v * rsqrt(mean(v^2) + eps) * gamma with v = x[r, :], or (kAdd) v = sum[r, :] = bf16(x + add); fp32 math.
// One row is 8 KB: a few microseconds of launch, first loads and one block reduction.  Launched with programmatic
// serialization, so the launch and the block's start run under the predecessor; the addition of the attention output is
// one launch (2.5 us in a decode layer) less as part of this kernel.
//
// kLogits (with kAdd): logits[r, e] = out[r, :] . gate[e, :] for the router as well, fp32.  `slices` CTAs per row normalise it each
// for itself and take every slices-th expert, a warp per expert; the first one stores the rows.  As a dense projection of its own
// the router was 9.4 us of a decode layer at 4 sequences and 11.0 at 64 (36 experts), for 0.3 MB of weights.
template <bool kAdd, bool kLogits>
__global__ void __launch_bounds__(256)
rmsnorm_kernel(const __nv_bfloat16* x, const __nv_bfloat16* add, const __nv_bfloat16* gamma, __nv_bfloat16* sum,
               __nv_bfloat16* out, int hidden, float eps, const __nv_bfloat16* gate, int experts, float* logits, int slices) {
  __shared__ float red[8];
  extern __shared__ uint4 s_row[];  // kLogits: the normalised row
  const int token = kLogits ? (int)blockIdx.x / slices : (int)blockIdx.x, slice = kLogits ? (int)blockIdx.x % slices : 0;
  // Resident while its predecessor still runs: no read-only loads, and none ahead of the wait.
  grid_dep_launch();
  if (kLogits) {  // (weights: only towards L2)
    const int lines = (hidden * 2 + 127) / 128;
    for (int e = slice + slices * ((int)threadIdx.x >> 5); e < experts; e += slices * 8)
      for (int i = threadIdx.x & 31; i < lines; i += 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t*>(gate + (size_t)e * hidden) + 128 * i));
  }
  grid_dep_wait_cta();
  const size_t row = (size_t)token * hidden;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row);
  const uint4* ar = reinterpret_cast<const uint4*>(kAdd ? add + row : nullptr);
  const uint4* gr = reinterpret_cast<const uint4*>(gamma);
  uint4* srow = reinterpret_cast<uint4*>(kAdd ? sum + row : nullptr);
  uint4* orow = reinterpret_cast<uint4*>(out + row);
  const int chunks = hidden / 8;
  float ss = 0.f;
  for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
    uint4 v = __ldcg(xr + c);
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
    if (kAdd) {
      const uint4 w = __ldcg(ar + c);
      const __nv_bfloat162* d = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]), e = __bfloat1622float2(d[i]);
        h[i] = __floats2bfloat162_rn(f.x + e.x, f.y + e.y);
      }
      if (!kLogits || slice == 0) srow[c] = v;
      if (kLogits) s_row[c] = v;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)hidden + eps);
  for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
    const uint4 v = kLogits ? s_row[c] : kAdd ? srow[c] : __ldcg(xr + c);  // the sum: this thread's own store
    const uint4 g = __ldcg(gr + c);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      const float2 gf = __bfloat1622float2(gh[i]);
      // everything in fp32, one rounding at the end
      oh[i] = __floats2bfloat162_rn(f.x * inv * gf.x, f.y * inv * gf.y);
    }
    if (!kLogits || slice == 0) orow[c] = o;
    if (kLogits) s_row[c] = o;
  }
  if (!kLogits) return;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int e = slice + slices * ((int)threadIdx.x >> 5); e < experts; e += slices * 8) {
    const uint4* w = reinterpret_cast<const uint4*>(gate + (size_t)e * hidden);
    float acc[2] = {0.f, 0.f};
#pragma unroll 8
    for (int c = lane; c < chunks; c += 32) {
      const uint4 g = __ldcg(w + c), v = s_row[c];
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]), k = __bfloat1622float2(gh[i]);
        acc[0] = fmaf(f.x, k.x, acc[0]);
        acc[1] = fmaf(f.y, k.y, acc[1]);
      }
    }
    float total = acc[0] + acc[1];
    for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
    if (lane == 0) logits[(size_t)token * experts + e] = total;
  }
}

// This step's keys and values into their caches, 16 bytes per thread.  Two generic scatters with an expanded index took
// 4.4-5.9 us each in a decode layer (4 to 64 sequences), nearly all of it launch and indexing.
__global__ void __launch_bounds__(256)
kv_append_kernel(const uint4* k, const uint4* v, long long pitch, uint4* k_cache, uint4* v_cache, const long long* pos, int n,
                 int kv_heads, int S, int chunks) {
  grid_dep_launch();
  grid_dep_wait_cta();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // (sequence, kv head, chunk)
  const long long at = __ldcg(pos);
  if (i >= n || at < 0 || at >= S) return;
  const int c = i % chunks, pair = i / chunks;
  const int b = pair / kv_heads, h = pair - b * kv_heads;
  const long long from = b * pitch + (long long)h * chunks + c, to = ((long long)pair * S + at) * chunks + c;
  k_cache[to] = __ldcg(k + from);
  v_cache[to] = __ldcg(v + from);
}

}  // namespace mf

extern "C" {

int mf_router_topk(const float* logits, const float* bias, float* weights, int* ids, int tokens, int experts,
                   int top_k, int n_group, int topk_group, int sigmoid, int renorm, float scale,
                   mf_stream_t stream) {
  if (tokens == 0) return 0;
  if (top_k > 32 || top_k < 1 || n_group < 1 || n_group > 32 || experts % n_group != 0 || top_k > experts) return -1;
  const size_t smem = (size_t)mf::kRouterWarps * 2 * experts * sizeof(float);
  if (smem > 48 * 1024) return -2;
  const int blocks = (tokens + mf::kRouterWarps - 1) / mf::kRouterWarps;
  const mf::RouteParams p{experts, top_k, n_group, topk_group, sigmoid, renorm, scale};
  mf::router_topk_kernel<<<blocks, mf::kRouterWarps * 32, smem, static_cast<cudaStream_t>(stream)>>>(
      logits, bias, weights, ids, tokens, p);
  return (int)cudaGetLastError();
}

int mf_rmsnorm(const void* x, const void* gamma, void* out, int rows, int hidden, float eps, mf_stream_t stream) {
  if (rows == 0) return 0;
  if (hidden % 8 != 0) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(out)) & 15) return -2;
  return (int)mf::launch_kernel(mf::rmsnorm_kernel<false, false>, dim3(rows), dim3(256), 0, static_cast<cudaStream_t>(stream), true,
                                static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(nullptr),
                                static_cast<const __nv_bfloat16*>(gamma), static_cast<__nv_bfloat16*>(nullptr),
                                static_cast<__nv_bfloat16*>(out), hidden, eps, static_cast<const __nv_bfloat16*>(nullptr), 0,
                                static_cast<float*>(nullptr), 1);
}

int mf_add_rmsnorm(const void* x, const void* add, const void* gamma, void* sum, void* out, int rows, int hidden, float eps,
                   mf_stream_t stream) {
  if (rows == 0) return 0;
  if (hidden % 8 != 0 || !add || !sum) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(gamma) |
       reinterpret_cast<uintptr_t>(sum) | reinterpret_cast<uintptr_t>(out)) & 15)
    return -2;
  return (int)mf::launch_kernel(mf::rmsnorm_kernel<true, false>, dim3(rows), dim3(256), 0, static_cast<cudaStream_t>(stream), true,
                                static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(add),
                                static_cast<const __nv_bfloat16*>(gamma), static_cast<__nv_bfloat16*>(sum),
                                static_cast<__nv_bfloat16*>(out), hidden, eps, static_cast<const __nv_bfloat16*>(nullptr), 0,
                                static_cast<float*>(nullptr), 1);
}

int mf_add_rmsnorm_logits(const void* x, const void* add, const void* gamma, void* sum, void* out, int rows, int hidden, float eps,
                          const void* gate, int experts, float* logits, int n_sms, mf_stream_t stream) {
  if (rows == 0) return 0;
  if (rows < 0 || hidden < 8 || hidden % 8 != 0 || hidden > 16384 || experts < 1 || n_sms < 1 || !add || !sum || !gate || !logits) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(gamma) |
       reinterpret_cast<uintptr_t>(sum) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(gate)) & 15)
    return -2;
  // a warp per expert where that takes at most four CTAs per SM
  const long long room = 4ll * n_sms / rows, want = (experts + 7) / 8;
  const int slices = (int)(room < 1 ? 1 : room < want ? room : want);
  if ((long long)rows * slices > 0x7fffffffLL) return -1;
  return (int)mf::launch_kernel(mf::rmsnorm_kernel<true, true>, dim3(rows * slices), dim3(256), (size_t)hidden * 2,
                                static_cast<cudaStream_t>(stream), true, static_cast<const __nv_bfloat16*>(x),
                                static_cast<const __nv_bfloat16*>(add), static_cast<const __nv_bfloat16*>(gamma),
                                static_cast<__nv_bfloat16*>(sum), static_cast<__nv_bfloat16*>(out), hidden, eps,
                                static_cast<const __nv_bfloat16*>(gate), experts, logits, slices);
}

int mf_kv_append(const void* k, const void* v, long long pitch, void* k_cache, void* v_cache, const long long* pos, int B,
                 int kv_heads, int S, int head_dim, mf_stream_t stream) {
  if (B < 0 || kv_heads < 1 || S < 1 || head_dim < 8 || head_dim % 8 != 0 || pitch % 8 != 0 ||
      (long long)B * kv_heads * (head_dim / 8) > 0x7fffffffLL)
    return -1;
  const uintptr_t all = reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(k_cache) |
                        reinterpret_cast<uintptr_t>(v_cache);
  if ((all & 15) != 0 || !k || !v || !k_cache || !v_cache || !pos) return -2;
  const int chunks = head_dim / 8, n = B * kv_heads * chunks;
  if (n == 0) return 0;
  return (int)mf::launch_kernel(mf::kv_append_kernel, dim3((n + 255) / 256), dim3(256), 0, static_cast<cudaStream_t>(stream), true,
                                static_cast<const uint4*>(k), static_cast<const uint4*>(v), pitch / 8, static_cast<uint4*>(k_cache),
                                static_cast<uint4*>(v_cache), pos, n, kv_heads, S, chunks);
}

}  // extern "C"

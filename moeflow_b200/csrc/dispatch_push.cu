// Dispatch: pack + all-to-all in one kernel, over peer memory.
//
// Token t of source rank s bound for owner rank d always lands in row recv_d[s, t] (fixed position,
// no count exchange).  A row is
//     [ H bf16 hidden lanes | K int32 local expert ids | K fp32 routing weights | int32 valid ]
// with a row pitch padded to a multiple of 16 bytes.  Slots whose expert lives on another rank carry
// id -1 and weight 0; valid = 1 iff at least one slot is on d and t is a live token (t < T and
// t < *num_valid).  Rows t >= T get valid = 0 and all-empty slots; their hidden lanes stay stale.
//
// The kernel writes every row straight into the owner's receive buffer with plain 16-byte stores
// through the peer mapping (NVLink).  Every CTA (one per token position) then fences once at system
// scope and adds one to flag word [s] of every owner: the flags count arrivals, a forward brings exactly
// C of them per source, and the owner's metadata kernel waits for epoch * C.  No CTA has to be the last
// one, so no second fence and no local counter sit between the rows and the flag.  No NCCL call, no
// staging buffer.
//
// Replaces the reference's pack kernel plus its dispatch all_to_all_single
// (moeflow/kernels/dispatch_pack.py:10-95, moeflow/fixed.py:95-125,234).
#include "common.cuh"
#include "expert_meta.cuh"
#include "moeflow_b200.h"
#include "quant.cuh"
#include "router.cuh"

namespace mf {

// A CTA per token: the hidden row is loaded and stored by many lanes at once.
constexpr int kDispatchThreads = 256;
constexpr int kMaxTopK = 32;
constexpr int kMaxRanks = 256;

__global__ void __launch_bounds__(kDispatchThreads) dispatch_push_kernel(const mf_dispatch_args a) {
  __shared__ int s_id[kMaxTopK];
  __shared__ float s_w[kMaxTopK];
  __shared__ unsigned char s_present[kMaxRanks];

  const int t = blockIdx.x;
  const int tid = threadIdx.x;
  unsigned long long* trace = (a.trace != nullptr && blockIdx.x == 0 && tid == 0) ? a.trace : nullptr;
  if (trace) trace[0] = global_timer_ns();
  grid_dep_launch();  // the metadata kernel may get resident now; it waits for this grid to complete
  {
    // First touches in parallel instead of one after the other (see touch() in common.cuh): every page this CTA
    // reads or writes, one lane each; warp 1 also touches this token's row in every destination's receive buffer.
    if (tid < 12) {
      // (a chain of selects: an array of pointers would live in local memory)
      const void* p = tid == 0 ? (const void*)a.epoch : tid == 1 ? (const void*)a.num_valid
                    : tid == 2 ? (a.logits ? (const void*)(a.logits + (size_t)min(t, a.T > 0 ? a.T - 1 : 0) * a.E) : nullptr)
                    : tid == 3 ? (const void*)a.bias : tid == 4 ? (const void*)a.x : tid == 5 ? (const void*)a.peer_recv
                    : tid == 6 ? (const void*)a.peer_flag : tid == 7 ? (const void*)(a.hit + (size_t)t * a.R)
                    : tid == 8 ? (const void*)a.route_w : tid == 9 ? (const void*)a.route_ids
                    : tid == 10 ? (const void*)a.done_counter : (const void*)a.weights;
      touch(p);
    } else if (tid >= 32 && tid < 32 + a.R && tid < 64) {
      const int d = tid - 32;
      touch(reinterpret_cast<const uint8_t*>(a.peer_recv[d]) + ((size_t)a.rank * a.C + t) * a.pitch);
      touch(reinterpret_cast<const unsigned*>(a.peer_flag[d]) + a.rank);
    }
  }
  const unsigned epoch_next = *a.epoch + 1u;
  const bool has_token = t < a.T;
  const bool live = has_token && (a.num_valid == nullptr || t < *a.num_valid);

  if (a.logits != nullptr) {
    // Fused routing: warp 0 routes this CTA's token; the other warps go on to load the hidden row.
    extern __shared__ float s_route[];
    if (tid < 32) {
      float w = 0.f;
      int id = -1;
      if (has_token) {
        const RouteParams p{a.E, a.K, a.n_group, a.topk_group, a.sigmoid, a.renorm, a.scale};
        route_token_warp(a.logits + (size_t)t * a.E, a.bias, s_route, s_route + a.E, p, tid, w, id);
      }
      if (tid < a.K) {
        s_id[tid] = has_token ? id : -1;
        s_w[tid] = has_token ? w : 0.f;
        if (has_token) {
          a.route_w[(size_t)t * a.K + tid] = w;
          a.route_ids[(size_t)t * a.K + tid] = id;
        }
      }
    }
  } else if (tid < a.K) {
    s_id[tid] = has_token ? a.ids[(size_t)t * a.K + tid] : -1;
    s_w[tid] = has_token ? a.weights[(size_t)t * a.K + tid] : 0.f;
  }

  // The hidden row is read once and kept in registers for all destinations.
  const int chunks = a.H / 8;  // 16-byte chunks
  constexpr int kMaxPerThread = 4;  // H <= 8192
  uint4 xv[kMaxPerThread];
  if (has_token) {
    const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.x) + (size_t)t * a.H);
#pragma unroll
    for (int i = 0; i < kMaxPerThread; ++i) {
      const int c = tid + i * kDispatchThreads;
      if (c < chunks) xv[i] = xr[c];
    }
  }
  __syncthreads();
  if (trace) trace[1] = global_timer_ns();  // routed, hidden row loaded

  // Which destinations does this token hit?  One thread per destination, once; the copy loop below then
  // needs no barrier, so the stores to all peers are in flight together.
  for (int d = tid; d < a.R; d += kDispatchThreads) {
    int present = 0;
    if (live)
      for (int k = 0; k < a.K; ++k) present |= (s_id[k] >= 0 && s_id[k] / a.L == d) ? 1 : 0;
    s_present[d] = (unsigned char)present;
    a.hit[(size_t)t * a.R + d] = (unsigned char)present;
  }
  __syncthreads();

  for (int d = 0; d < a.R; ++d) {
    const int present = s_present[d];
    uint8_t* row = reinterpret_cast<uint8_t*>(a.peer_recv[d]) + ((size_t)a.rank * a.C + t) * a.pitch;
    if (has_token && (present || !a.skip_payload)) {
      uint4* dst = reinterpret_cast<uint4*>(row);
#pragma unroll
      for (int i = 0; i < kMaxPerThread; ++i) {
        const int c = tid + i * kDispatchThreads;
        if (c < chunks) dst[c] = xv[i];
      }
    }
    int* meta = reinterpret_cast<int*>(row + (size_t)a.H * 2);
    if (tid < a.K) {
      const bool on = present && s_id[tid] >= 0 && s_id[tid] / a.L == d;
      meta[tid] = on ? s_id[tid] - d * a.L : -1;
      meta[a.K + tid] = on ? __float_as_int(s_w[tid]) : 0;
    } else if (tid == a.K) {
      meta[2 * a.K] = present;
    }
  }

  // Publish: the barrier orders every thread's stores before the system fence of warp 0's lanes (cumulative);
  // then one arrival per destination, issued by different lanes so that they travel together.
  __syncthreads();
  if (trace) trace[2] = global_timer_ns();  // rows stored
  if (tid < 32) {
    fence_before_arrival(a.R);
    if (trace) trace[3] = global_timer_ns();  // fenced
    for (int d = tid; d < a.R; d += 32) red_add_relaxed_sys_u32(reinterpret_cast<unsigned*>(a.peer_flag[d]) + a.rank, 1u);
    if (tid == 0) {
      // the local epoch (read by this rank's later kernels after this grid has completed)
      const unsigned done = atomicAdd(a.done_counter, 1u);
      if (done == gridDim.x - 1) {
        *a.done_counter = 0u;
        *a.epoch = epoch_next;
        if (a.trace) a.trace[5] = global_timer_ns();  // last CTA done
      }
    }
    if (trace) trace[4] = global_timer_ns();  // arrivals sent
  }
}

// The same for prefill sizes (from 512 token positions, up to 32 ranks): a warp per token and four of them per CTA, with
// nothing shared between them but the arrival.  With a CTA per token three of its four warps waited for the one that
// routes, in 3.5 waves of CTAs at 8192 tokens; a quarter of the CTAs also means a quarter of the fences and arrivals.
// Kernel at 8192 tokens 74 / 53 us, at 2000 21 / 14, at 700 18.5 / 10.3, at 512 10.4 / 8.4.  Below, 256 to 511 tokens, it is
// 10.4 / 8.3 as well, but the layer takes the same (185 / 181, 206 / 206, 235 / 238 us with 36 e4m3 experts), and one rank
// uses the local dispatch there (top-8: up to 512 tokens).
// A row's first 4096 values are in flight while its token is routed (with 2048, the others' loads came behind the routing), and one
// rank fences nothing.  At hidden 4096: kernel at 1000 tokens 13.0 / 8.8 us, at 8192 56 / 38; 600 tokens on 36 e4m3 experts 264.6 / 260.5, 520 on
// 72 bf16 ones 246.4 / 242.9, calls at the power cap as before.
constexpr int kManyWarps = 4;

__global__ void __launch_bounds__(32 * kManyWarps) dispatch_push_many_kernel(const mf_dispatch_args a) {
  extern __shared__ float s_many[];  // [kManyWarps][2 E] scores of the tokens being routed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * kManyWarps + warp;
  unsigned long long* trace = (a.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) ? a.trace : nullptr;
  if (trace) trace[0] = global_timer_ns();
  grid_dep_launch();
  const unsigned epoch_next = *a.epoch + 1u;
  if (t < a.C) {
    const bool has_token = t < a.T;
    const bool live = has_token && (a.num_valid == nullptr || t < *a.num_valid);
    // the first kAhead * 256 values of the row are under way while the token is routed, any others are loaded behind it
    const int chunks = a.H / 8;  // 16-byte chunks
    constexpr int kAhead = 16;
    const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.x) + (size_t)t * a.H);
    uint4 xv[kAhead];
    if (has_token) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
        if (lane + 32 * i < chunks) xv[i] = xr[lane + 32 * i];
    }
    float w = 0.f;
    int id = -1;  // lane k (< K): slot k
    if (has_token) {
      if (a.logits != nullptr) {
        float* score = s_many + (size_t)warp * 2 * a.E;
        const RouteParams p{a.E, a.K, a.n_group, a.topk_group, a.sigmoid, a.renorm, a.scale};
        route_token_warp(a.logits + (size_t)t * a.E, a.bias, score, score + a.E, p, lane, w, id);
        if (lane < a.K) {
          a.route_w[(size_t)t * a.K + lane] = w;
          a.route_ids[(size_t)t * a.K + lane] = id;
        }
      } else if (lane < a.K) {
        id = a.ids[(size_t)t * a.K + lane];
        w = a.weights[(size_t)t * a.K + lane];
      }
    }
    if (lane >= a.K) id = -1;
    if (trace) trace[1] = global_timer_ns();  // routed
    const int owner = id >= 0 ? id / a.L : -1;
    for (int d = 0; d < a.R; ++d) {
      const bool on = live && owner == d;
      const int present = __any_sync(0xffffffffu, on) ? 1 : 0;
      uint8_t* row = reinterpret_cast<uint8_t*>(a.peer_recv[d]) + ((size_t)a.rank * a.C + t) * a.pitch;
      if (has_token && (present || !a.skip_payload)) {
        uint4* dst = reinterpret_cast<uint4*>(row);
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
          if (lane + 32 * i < chunks) dst[lane + 32 * i] = xv[i];
#pragma unroll 8
        for (int c = lane + 32 * kAhead; c < chunks; c += 32) dst[c] = xr[c];
      }
      int* meta = reinterpret_cast<int*>(row + (size_t)a.H * 2);
      if (lane < a.K) {
        meta[lane] = on ? id - d * a.L : -1;
        meta[a.K + lane] = on ? __float_as_int(w) : 0;
      }
      if (lane == 0) {
        meta[2 * a.K] = present;
        a.hit[(size_t)t * a.R + d] = (unsigned char)present;
      }
    }
  }
  __syncthreads();
  if (trace) trace[2] = global_timer_ns();  // rows stored
  if (warp == 0) {
    if (a.R > 1) fence_before_arrival(a.R);  // (nobody waits for a single rank's flag: what follows waits for this grid)
    if (trace) trace[3] = global_timer_ns();  // fenced
    // one arrival per token position, as from a CTA per token
    const unsigned rows = (unsigned)min(kManyWarps, a.C - (int)blockIdx.x * kManyWarps);
    if (lane < a.R) red_add_relaxed_sys_u32(reinterpret_cast<unsigned*>(a.peer_flag[lane]) + a.rank, rows);
    if (lane == 0) {
      const unsigned done = atomicAdd(a.done_counter, 1u);
      if (done == gridDim.x - 1) {
        *a.done_counter = 0u;
        *a.epoch = epoch_next;
        if (a.trace) a.trace[5] = global_timer_ns();  // last CTA done
      }
    }
    if (trace) trace[4] = global_timer_ns();  // arrivals sent
  }
}

// The only rank is this GPU, decode sizes: dispatch and metadata in one launch.  There is no peer to wait for, so the CTA
// that stores its row last goes on with the one-pass metadata build (expert_meta.cuh) on the rows it finds in L2: no
// second launch, no flags, no cold start of another kernel behind a weight stream that has swept its code and pages out
// of the caches.  The rows of e4m3 layers are quantised by the CTAs that hold them in registers.  512 threads: one
// 16-byte chunk of a 4096-wide row each, and eight slot words each in the metadata pass.
// The layout is there, from the kernel's start and between passes that stream weights, after 13.1 us at 128 tokens on 288 experts
// (19.6 with the router's scores in shared memory, the payload in front of the fence and the metadata pass unrolled throughout).
//
// Up to kLocalThreads / 32 token positions one more CTA, the bookkeeper, routes all of them for itself, a warp each, and
// builds the layout from shared memory: nothing of it goes through L2 (slot words, fence, arrival and the loads behind it took
// 2.3 us), and the tokens' own CTAs only store their rows.  Layout after 7.0 instead of 9.2 us at 1 token on 288 experts, 4.6
// instead of 6.7 on 32; calls, us: 1 token 69.2 / 67.2 (32 experts of hidden 512, 8 tokens: 26.4 / 23.2), 8 tokens e4m3
// 169.9 / 167.4, decode model of 4 sequences 217 / 211.  Above, a warp would route several tokens one after the other: with
// two, 32 tokens on 36 experts (e4m3) 123.9 / 125.2, 20 on 288 325.7 / 328.4.
constexpr int kLocalThreads = 512;
constexpr int kLocalWarps = kLocalThreads / 32;
constexpr int kKeeperSmem = 112 * 1024;

__device__ __forceinline__ void bookkeeper(const mf_dispatch_args& a, const mf_meta_args& m, int* s_dyn) {
  __shared__ int s_key[kLocalWarps * kMaxTopK], s_bits[kLocalWarps * kMaxTopK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = warp;
  unsigned long long* trace = (m.trace != nullptr && tid == 0) ? m.trace : nullptr;
  grid_dep_launch();
  if (warp == kLocalWarps - 1 && lane < 12) {
    // the pages that the metadata pass stores to
    const void* p = lane == 0 ? (const void*)m.plan : lane == 1 ? (const void*)m.offsets : lane == 2 ? (const void*)m.tile_e
                  : lane == 3 ? (const void*)m.tile_s : lane == 4 ? (const void*)m.tile_n : lane == 5 ? (const void*)m.row_hits
                  : lane == 6 ? (const void*)m.inv : lane == 7 ? (const void*)m.entry_row : lane == 8 ? (const void*)m.entry_slot
                  : lane == 9 ? (const void*)m.entry_w : lane == 10 ? (const void*)(m.counters1 + m.n_counters1) : (const void*)a.epoch;
    touch(p);
  }
  if (t < a.C) {
    const bool has_token = t < a.T;
    float w = 0.f;
    int id = -1;  // lane k (< K): slot k
    if (has_token) {
      if (a.logits != nullptr) {
        float* score = reinterpret_cast<float*>(s_dyn + meta_smem_words(m.L, kLocalThreads)) + (size_t)warp * 2 * a.E;
        const RouteParams p{a.E, a.K, a.n_group, a.topk_group, a.sigmoid, a.renorm, a.scale};
        route_token_warp(a.logits + (size_t)t * a.E, a.bias, score, score + a.E, p, lane, w, id);
      } else if (lane < a.K) {
        id = a.ids[(size_t)t * a.K + lane];
        w = a.weights[(size_t)t * a.K + lane];
      }
    }
    const bool on = has_token && (a.num_valid == nullptr || t < *a.num_valid) && id >= 0 && id < a.L;
    if (lane < a.K) {
      s_key[t * a.K + lane] = on ? id : -1;
      s_bits[t * a.K + lane] = on ? __float_as_int(w) : 0;
    }
  }
  meta_begin<kLocalThreads>(m, s_dyn);
  __syncthreads();
  if (a.trace != nullptr && tid == 0) a.trace[2] = global_timer_ns();  // the slot words stand in shared memory
  if (tid == 0) *a.epoch += 1u;
  meta_one_pass<kLocalThreads>(m, SharedSlots{s_key, s_bits, a.K}, s_dyn, trace);
}

// kPerSm: CTAs an SM should hold.  With at most one token per SM the registers for one CTA are free and nothing spills; above
// that two share an SM (500 tokens: 1 % of the layer).
// kKeeper: the last CTA is the bookkeeper (kernels of their own: with both forms in one the larger sizes lost 0.7 %).
template <int kPerSm, bool kKeeper>
__global__ void __launch_bounds__(kLocalThreads, kPerSm) dispatch_local_kernel(const mf_dispatch_args a, const mf_meta_args m) {
  extern __shared__ int s_dyn[];  // metadata pass, then the router's scores
  __shared__ int s_id[kMaxTopK];
  __shared__ float s_w[kMaxTopK];
  __shared__ int s_last;
  const int t = blockIdx.x, tid = threadIdx.x;
  if (kKeeper && t == a.C) {
    bookkeeper(a, m, s_dyn);
    return;
  }
  unsigned long long* trace = (a.trace != nullptr && blockIdx.x == 0 && tid == 0) ? a.trace : nullptr;
  if (trace) trace[0] = global_timer_ns();
  grid_dep_launch();
  uint8_t* row = const_cast<uint8_t*>(static_cast<const uint8_t*>(m.recv)) + (size_t)t * a.pitch;
  const bool has_token = t < a.T;
  const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.x) + (size_t)t * a.H);
  const int chunks = a.H / 8;
  uint4 xv[2];  // H <= 8192
  if (has_token) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (tid + i * kLocalThreads < chunks) xv[i] = xr[tid + i * kLocalThreads];
  }
  const bool live = has_token && (a.num_valid == nullptr || t < *a.num_valid);
  if (tid < 32) {
    float w = 0.f;
    int id = -1;
    if (a.logits != nullptr) {
      if (has_token) {
        float* score = reinterpret_cast<float*>(s_dyn + meta_smem_words(m.L, kLocalThreads));
        const RouteParams p{a.E, a.K, a.n_group, a.topk_group, a.sigmoid, a.renorm, a.scale};
        route_token_warp(a.logits + (size_t)t * a.E, a.bias, score, score + a.E, p, tid, w, id);
        if (tid < a.K) {
          a.route_w[(size_t)t * a.K + tid] = w;
          a.route_ids[(size_t)t * a.K + tid] = id;
        }
      }
    } else if (has_token && tid < a.K) {
      id = a.ids[(size_t)t * a.K + tid];
      w = a.weights[(size_t)t * a.K + tid];
    }
    if (tid < a.K) {
      s_id[tid] = id;
      s_w[tid] = w;
    }
  } else {
    // in the shadow of the routing warp: the pages that the metadata pass stores to, and its histogram
    if (tid < 48 && (!kKeeper || tid == 43 || tid == 46)) {
      const void* p = tid == 32 ? (const void*)m.plan : tid == 33 ? (const void*)m.offsets : tid == 34 ? (const void*)m.tile_e
                    : tid == 35 ? (const void*)m.tile_s : tid == 36 ? (const void*)m.tile_n : tid == 37 ? (const void*)m.row_hits
                    : tid == 38 ? (const void*)m.inv : tid == 39 ? (const void*)m.entry_row : tid == 40 ? (const void*)m.entry_slot
                    : tid == 41 ? (const void*)m.entry_w : tid == 42 ? (const void*)(m.counters1 + m.n_counters1)
                    : tid == 43 ? (const void*)(row + (size_t)a.H * 2) : tid == 44 ? (const void*)a.epoch
                    : tid == 45 ? (const void*)a.done_counter : tid == 46 ? (const void*)(a.hit + t) : nullptr;
      touch(p);
    }
  }
  if (!kKeeper) meta_begin<kLocalThreads>(m, s_dyn);
  __syncthreads();
  if (trace) trace[1] = global_timer_ns();  // routed, hidden row loaded
  int present = 0;
  if (live)
    for (int k = 0; k < a.K; ++k) present |= (s_id[k] >= 0 && s_id[k] < a.L) ? 1 : 0;
  if (tid < 32) {
    // What the metadata pass reads goes first and is fenced by itself: the fence then waits for one warp's few words, while
    // the other warps store (and quantise) the payload, which only has to be there when the grid is done.
    int* meta = reinterpret_cast<int*>(row + (size_t)a.H * 2);
    if (tid < a.K) {
      const bool on = present && s_id[tid] >= 0 && s_id[tid] < a.L;
      meta[tid] = on ? s_id[tid] : -1;
      meta[a.K + tid] = on ? __float_as_int(s_w[tid]) : 0;
    }
    if (tid == 31) {
      meta[2 * a.K] = present;
      a.hit[t] = (unsigned char)present;
    }
    __syncwarp();
    if (tid == 0 && !kKeeper) {
      __threadfence();  // cumulative: the whole warp's stores, ordered by the barrier
      const unsigned done = atomicAdd(a.done_counter, 1u);
      __threadfence();  // in the last CTA: every other CTA's words come before what follows
      s_last = done == gridDim.x - 1;
      if (s_last) {
        *a.done_counter = 0u;
        *a.epoch += 1u;
      }
    }
    __syncwarp();
  }
  if (has_token && (present || !a.skip_payload)) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = tid + i * kLocalThreads;
      if (c < chunks) {
        reinterpret_cast<uint4*>(row)[c] = xv[i];
        if (m.xq != nullptr && present) quant_chunk(xv[i], c, m.xq + (size_t)t * a.H, m.xs + (size_t)t * (a.H / 128));
      }
    }
  }
  if (kKeeper) return;
  __syncthreads();
  if (trace) trace[2] = global_timer_ns();  // row stored
  if (!s_last) return;
  meta_one_pass<kLocalThreads>(m, RowSlots(m), s_dyn, (m.trace != nullptr && tid == 0) ? m.trace : nullptr);
}

}  // namespace mf

extern "C" int mf_dispatch_local(const mf_dispatch_args* a, const mf_meta_args* m, mf_stream_t stream) {
  using namespace mf;
  if (!a || !m || a->C < 1 || a->T > a->C || a->K < 1 || a->K > kMaxTopK || a->R != 1 || m->R != 1 || a->H % 8 != 0 || a->H > 8192 ||
      (a->pitch & 15) != 0 || a->pitch < (long long)a->H * 2 + (2 * a->K + 1) * 4 || m->pitch != a->pitch || m->rows != a->C ||
      m->K != a->K || m->L != a->L || m->block_m < 1)
    return -1;
  if (m->L < 1 || m->L > kLocalThreads || (long long)a->C * a->K > kLocalThreads * kMetaBatch) return -2;
  if (m->xq != nullptr && (!m->xs || a->H % 128 != 0)) return -3;
  size_t smem = (size_t)meta_smem_words(m->L, kLocalThreads) * sizeof(int);
  const bool keeper = a->C <= kLocalWarps;
  if (a->logits != nullptr) {
    if (a->E < a->K || a->E != a->L || a->n_group < 1 || a->n_group > 32 || a->E % a->n_group != 0 || !a->route_w || !a->route_ids)
      return -4;
    smem += 2 * (size_t)a->E * sizeof(float) * (keeper ? a->C : 1);
  }
  // L = E <= 512: at most 41 KB, with a bookkeeper 102 KB
  if (smem > (keeper ? kKeeperSmem : 48 * 1024)) return -5;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (keeper) {
    static bool configured[64] = {};  // per device: the attribute belongs to (function, device)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
      e = cudaFuncSetAttribute(dispatch_local_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kKeeperSmem);
      if (e != cudaSuccess) return (int)e;
      if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    dispatch_local_kernel<1, true><<<a->C + 1, kLocalThreads, smem, st>>>(*a, *m);
  } else if (a->C <= m->n_sms) {
    dispatch_local_kernel<1, false><<<a->C, kLocalThreads, smem, st>>>(*a, *m);
  } else {
    dispatch_local_kernel<2, false><<<a->C, kLocalThreads, smem, st>>>(*a, *m);
  }
  return (int)cudaGetLastError();
}

extern "C" int mf_dispatch_push(const mf_dispatch_args* a, mf_stream_t stream) {
  constexpr int threads = mf::kDispatchThreads;
  if (!a || a->C < 1 || a->T > a->C || a->K > mf::kMaxTopK || a->R > mf::kMaxRanks || a->H % 8 != 0 ||
      a->H / 8 > threads * 4 || (a->pitch & 15) != 0 || a->pitch < (long long)a->H * 2 + (2 * a->K + 1) * 4)
    return -1;
  size_t smem = 0;
  if (a->logits != nullptr) {
    if (a->E < a->K || a->n_group < 1 || a->n_group > 32 || a->E % a->n_group != 0 || !a->route_w || !a->route_ids) return -2;
    smem = 2 * (size_t)a->E * sizeof(float);
    if (smem > 40 * 1024) return -3;
  }
  if (a->C >= 512 && a->R <= 32 && mf::kManyWarps * smem <= 40 * 1024) {
    const int ctas = (a->C + mf::kManyWarps - 1) / mf::kManyWarps;
    mf::dispatch_push_many_kernel<<<ctas, 32 * mf::kManyWarps, mf::kManyWarps * smem, static_cast<cudaStream_t>(stream)>>>(*a);
  } else {
    mf::dispatch_push_kernel<<<a->C, threads, smem, static_cast<cudaStream_t>(stream)>>>(*a);
  }
  return (int)cudaGetLastError();
}

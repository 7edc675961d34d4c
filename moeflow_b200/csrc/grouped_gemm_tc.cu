// Grouped expert GEMMs on the 5th-generation tensor cores (tcgen05) for sm_100a.
//
// The expert GEMMs of a decode step are weight-streaming bound: a few (1..64) token rows per expert
// against tens of MB of expert weights.  The kernels below are therefore written "swap-AB": the
// 128 weight rows of a block are the UMMA M dimension, the token rows are the UMMA N dimension
// (16..n_max), accumulators live in tensor memory, and the weight stream is a deep TMA pipeline.
//
//   gate/up  : acc_gate[128, n] = W13[e, mb*128 + r, :] . X[n, :]     (and acc_up for rows I + ...)
//              out[entry, mb*128 + r] = bf16( silu(min(gate, lim)) * clamp(up, +-lim) )
//   down     : acc[128, n] = W2[e, mb*128 + r, :] . ACT[n, :]
//              out[entry, mb*128 + r] = bf16( row_scale[entry] * acc )
//              (two_blocks: a unit covers two adjacent weight blocks with two accumulators, like gate/up,
//               so a token tile is fetched from L2 once per 256 output columns: the long-prefill form)
//
// A unit is (token tile, 128-row weight block); it needs k_blocks K steps.  The token tiles and the way
// the units are cut along K come from a device-side plan (see expert_meta.cu), so nothing is read back
// to the host.  Two cuts exist:
//   * K split S in {1, 2, 4, 8} (plan word = S): every unit is cut into S equal segments, segments are
//     handed to the CTAs one by one (work_iter.cuh);
//   * stream-K (plan word = 0): the units' K steps are laid end to end and every CTA takes one contiguous
//     share of that line, so all CTAs stream the same number of weight bytes whatever the unit count
//     (no partly filled last round); a unit that straddles CTA boundaries is cut there.
// A segment that is not a whole unit stores its fp32 partial sums; the last segment to arrive (per
// 32-row quarter) adds the segments in K order, so the result does not depend on arrival order.
//
// Warp roles (256 threads, one CTA per SM, persistent):
//   warp 0      TMA producer for the weight tiles (an elected lane issues); hands the segments out to the other roles
//   warp 1      UMMA issuer (an elected lane issues); owns the tensor-memory allocation
//   warps 2-3   token-operand producers: gather rows by index with cp.async into the swizzled tile, or warp 2 alone fetches
//               contiguous rows by TMA.  256-row tiles of two accumulators gather with warps 12-15; these two then have
//               nothing to do but, where asked for, to expand the down GEMM's e4m3 weights (expand_src)
//   warps 4-7   epilogue: tcgen05.ld -> registers -> activation / scale -> global
//
// CTA pairs (kPair: units of two accumulators on 256-row tiles): the two CTAs of a cluster take adjacent weight blocks of one
// token tile and hold one half of its rows each, as one MMA of M = 256 (cta_group::2, issued by CTA 0).  Per K block of a full
// tile a CTA then pulls 48 KB through L2 and reads 64 KB of operands out of shared memory for 1024 tensor cycles, instead of 64
// and 96, and gathers half of the rows.  Both CTAs run every role but the UMMA issuer's: in CTA 1 that warp reports gathered rows
// (a local barrier, a proxy fence, one arrival at CTA 0; with release.cluster on that arrival a K block took 1.15 us).
// Single CTAs / pairs, kernels alone in a burst, us: gate/up 72 experts 1000 tokens 341 / 323, 2000 tokens 482 / 446, 36 experts
// 8192 tokens 1359 / 1243; down 177 / 174, 247 / 239, 708 / 696.
//
// Replaces the reference's Triton grouped GEMM, unfused SwiGLU and expert-input gather
// (moeflow/kernels/grouped_gemm.py:15-80, moeflow/experts.py:10-17, moeflow/kernels/expert_prepare.py:10-38).
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "expand.cuh"
#include "moeflow_b200.h"
#include "work_iter.cuh"

namespace mf {

constexpr int kBlockM = 128;          // weight rows per block (UMMA M)
constexpr int kTileBytesA = 128 * 128;  // 128 rows x 128 bytes
constexpr int kThreads = 256;
constexpr int kThreadsWithReturn = 384;  // + 4 return warps (fused owner reduce + return push)
// Epilogue warp groups.  Tiles of 256 token columns fill all 512 tensor-memory columns with one accumulator stage
// (two accumulators of 256 columns) when they hold more than 128 rows, so their epilogue is not hidden behind the next unit's main loop: two groups of
// four warps then take half of the token columns each.  The variant with return warps keeps one group.
template <int N_MAX, bool kReturn>
constexpr int kEpiGroups = (N_MAX >= 256 && !kReturn) ? 2 : 1;
constexpr int kRetDepth = 4;            // queued unit descriptors per quarter
// Gather threads: warps 2 and 3, or four warps of their own (12-15) where a 256-row tile has 2048 chunks of 16 bytes per K
// step; the register split then takes from them and from the first four warps what the epilogue needs beyond 128
// (72 x 128 + 168 x 256 + 104 x 128 = 65536, what 512 threads are launched with).
template <bool kGateUp, int N_MAX, bool kReturn>
constexpr bool kWideGather = kGateUp && N_MAX >= 256 && !kReturn;
template <bool kGateUp, int N_MAX, bool kReturn>
constexpr int kLaunchThreads = kReturn ? kThreadsWithReturn : kWideGather<kGateUp, N_MAX, kReturn> ? 512 : 128 + 128 * kEpiGroups<N_MAX, kReturn>;
constexpr int kMaxAccStages = 2;
constexpr int kOutStageBytes = 1024;   // 16 token columns x 32 weight rows of 16-bit outputs, per epilogue warp
constexpr int kMaxDevices = 64;        // devices one process may drive (per-device launch configuration)

template <bool kGateUp, int N_MAX, bool kPair = false>
struct GemmCfg {
  static constexpr int kATiles = kGateUp ? 2 : 1;
  static constexpr int kStageA = kATiles * kTileBytesA;
  static constexpr int kStageB = (kPair ? N_MAX / 2 : N_MAX) * 128;
  static constexpr int kStageBytes = kStageA + kStageB;
  // As many stages as fit in 216 KB of the 227 KB a CTA may use (2 KB more go to alignment slack and
  // barriers): the bytes in flight per SM, not the tensor pipe, bound these weight-streaming kernels.
  static constexpr int kStages = (216 * 1024) / kStageBytes > 10 ? 10 : (216 * 1024) / kStageBytes;
  static constexpr int kAccCols = kATiles * N_MAX;
  // Two accumulator stages: the epilogue of unit i overlaps the main loop of unit i + 1.  With two accumulators of 256
  // columns a wide unit (more than 128 token columns) needs all 512 tensor-memory columns and takes both stages; a narrow
  // one takes one, its accumulators 128 columns apart.  Tiles are narrow more often than not where 256-row tiles begin (36
  // expected rows per expert on CTA pairs, else 80).
  static constexpr int kAccStages = 2;
  static constexpr bool kWide = kAccStages * kAccCols > 512;
  static constexpr int kStageCols = kWide ? 256 : kAccCols;
  static constexpr int kTmemCols = kAccStages * kStageCols;  // power of two for N_MAX in {32, 64, 128, 256}
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 1024 /*barriers, return queue*/ +
                                    (N_MAX >= 256 ? 8 : 4) * kOutStageBytes /*one transposing store buffer per epilogue warp*/;
};

struct PipeState {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance(int n_stages) {
    if (++stage == n_stages) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

// Fused owner reduce + return push, called by one epilogue warp after it has written the final y values
// of `n_rows` entries (first entry `row_start`) for its 32 columns `col0 .. col0+31` of block `mb`.
// For every entry the warp counts one arrival on (received row, block, quarter); the arrival that
// completes a row's hit count sums that row's slots in slot order (fp32, +0.0 start), rounds once to
// bf16 and stores the 32 values into the source rank's combine buffer.  Completed quarters are counted
// on `ret_done`; the warp that brings it to valid_rows * m_blocks * 4 publishes the return flags.
// Returns the number of (row, block, quarter) reductions this call completed; the caller adds them up and
// reports them once with return_finish (one system-scope fence per warp, not per unit).
__device__ __forceinline__ int return_rows(const mf_gemm_args& a, int n_rows, int row_start, int mb, int wq, int lane) {
  const __nv_bfloat16* y = static_cast<const __nv_bfloat16*>(a.out);
  const long long col0 = (long long)mb * kBlockM + wq * 32;  // this quarter's 32 columns (64 bytes, 64-byte aligned)
  int completed = 0;
  for (int n0 = 0; n0 < n_rows; n0 += 32) {
    // One lane per entry: count the arrival; the lane whose arrival completes the row does the whole row
    // (all its slots, 32 columns) by itself, so the rows of a unit are reduced in parallel, not in turn.
    const int n = n0 + lane;
    int r = -1;
    bool last = false;
    if (n < n_rows) {
      r = a.entry_row[row_start + n];
      int* cnt = a.row_cnt + ((long long)r * a.m_blocks + mb) * 4 + wq;
      const int old = atomicAdd(cnt, 1);
      last = (old + 1 == a.row_hits[r]);
      if (last) *cnt = 0;  // self-cleaning: nobody else touches this counter again in this forward
    }
    const unsigned todo = __ballot_sync(0xffffffffu, last);
    if (todo == 0u) continue;
    __threadfence();  // the other slots' y values (written by other CTAs) are visible now
    if (last) {
      float acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0.f;
      for (int k = 0; k < a.ret_K; ++k) {
        const int p = a.inv[(long long)r * a.ret_K + k];
        if (p < 0) continue;
        const uint4* src = reinterpret_cast<const uint4*>(y + (long long)p * a.out_pitch + col0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 v = __ldcg(src + q);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            acc[q * 8 + 2 * i] += f.x;
            acc[q * 8 + 2 * i + 1] += f.y;
          }
        }
      }
      const int src_rank = r / a.ret_C, t = r - src_rank * a.ret_C;
      uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.ret_peer[src_rank]) +
                                            ((long long)a.ret_rank * a.ret_C + t) * a.out_pitch + col0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 o;
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[q * 8 + 2 * i], acc[q * 8 + 2 * i + 1]);
        dst[q] = o;
      }
    }
    completed += __popc(todo);
  }
  return completed;
}

// Report `completed` reductions of this warp; the warp that brings the layer's counter to
// valid_rows * m_blocks * 4 publishes the return flags to every source rank.
__device__ __forceinline__ void return_finish(const mf_gemm_args& a, int completed, int lane) {
  if (completed == 0) return;
  __threadfence_system();  // the peer stores of all lanes precede the count (and so the flags)
  __syncwarp();
  if (lane == 0) {
    const unsigned total = (unsigned)a.plan[MF_PLAN_VALID_ROWS] * (unsigned)a.m_blocks * 4u;
    const unsigned before = atomicAdd(a.ret_done, (unsigned)completed);
    if (before + (unsigned)completed == total) {
      *a.ret_done = 0u;
      const unsigned pushes = *a.ret_epoch + 1u;  // counting flags: C arrivals per return push
      *a.ret_epoch = pushes;
      publish_flags(a.ret_flag, a.ret_R, a.ret_rank, pushes * (unsigned)a.ret_C);
    }
  }
}

// Last step of the epilogue for C values of each of one or two accumulators: the activation (gate/up), or the routing weight
// (down).  v: first accumulator (gate, or the only one); w: second accumulator (up; with two_blocks the second weight block);
// sc: routing weights.  No branch depends on the column, so that the C dependency chains (exp, reciprocal) overlap: the epilogue
// warps are alone on their scheduler and a column-by-column loop ran at one chain's latency (about 300 cycles per column).
template <bool kTwoAcc, int C>
__device__ __forceinline__ void finish(const mf_gemm_args& a, float (&v)[C], float (&w)[C], const float (&sc)[C]) {
  if (kTwoAcc && !a.two_blocks) {
    if (a.round_h) {
#pragma unroll
      for (int j = 0; j < C; ++j) {
        v[j] = bf16_round(v[j]);
        w[j] = bf16_round(w[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < C; ++j) v[j] = swiglu_clamped(v[j], w[j], a.limit);
  } else if (a.row_scale) {
#pragma unroll
    for (int j = 0; j < C; ++j) {
      v[j] *= sc[j];
      if (kTwoAcc) w[j] *= sc[j];
    }
  }
}

// ... of C token columns of one weight row per lane, and their stores, 2 bytes each.
template <bool kTwoAcc, int C>
__device__ __forceinline__ void finish_store(const mf_gemm_args& a, float (&v)[C], float (&w)[C], const float (&sc)[C],
                                             int n0, int n_rows, int row_start, long long out_col) {
  finish<kTwoAcc, C>(a, v, w, sc);
  const bool second = kTwoAcc && a.two_blocks;  // the other weight block's outputs, 128 columns further
  const bool all = n0 + C <= n_rows;
  __nv_bfloat16* p = static_cast<__nv_bfloat16*>(a.out) + (long long)(row_start + n0) * a.out_pitch + out_col;
#pragma unroll
  for (int j = 0; j < C; ++j) {
    if (all || n0 + j < n_rows) {
      p[(long long)j * a.out_pitch] = __float2bfloat16_rn(v[j]);
      if (second) p[(long long)j * a.out_pitch + kBlockM] = __float2bfloat16_rn(w[j]);
    }
  }
}

// Outputs of 16 token columns x 32 weight rows, in the layout of tmem_ld_16x16 (x[8 h ..]: weight rows 16 h ..), to global memory
// through 1 KB of shared memory owned by the warp: pairs of tokens are rounded together and stored transposed, a token's 32 values
// in four chunks of 16 bytes (chunk c of token t at place c ^ (t / 2 & 3): no bank conflicts either way), and every lane then
// stores 16 bytes of one token.  `p`: the first token's first value of this warp.
__device__ __forceinline__ void store_16x32(const float (&x)[16], uint8_t* stage, int lane, __nv_bfloat16* p, int pitch, int rows) {
  const int m = lane >> 3, j = lane & 7;
  const uint32_t to = smem_u32(stage) + j * 64 + ((m ^ (j >> 1)) << 4);
  __syncwarp();  // the previous block's reads are done
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t r[4] = {pack_bf16x2(x[4 * k], x[4 * k + 1]), pack_bf16x2(x[4 * k + 2], x[4 * k + 3]),
                           pack_bf16x2(x[8 + 4 * k], x[8 + 4 * k + 1]), pack_bf16x2(x[8 + 4 * k + 2], x[8 + 4 * k + 3])};
    stmatrix_x4_trans(to + k * 512, r);
  }
  __syncwarp();
  const int t = lane >> 2, c = lane & 3;
  const uint8_t* from = stage + t * 64 + ((c ^ (t >> 1)) << 4);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 y = *reinterpret_cast<const uint4*>(from + h * 512);
    if (t + 8 * h < rows) *reinterpret_cast<uint4*>(p + (long long)(t + 8 * h) * pitch + c * 8) = y;
  }
}

template <bool kGateUp, int N_MAX, bool kReturn = false, bool kPair = false>
__global__ void __launch_bounds__(kLaunchThreads<kGateUp, N_MAX, kReturn>, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_b,
                    const mf_gemm_args a) {
  static_assert(!kPair || (kGateUp && !kReturn), "pairs: two accumulators, no return warps");
  using Cfg = GemmCfg<kGateUp, N_MAX, kPair>;
  constexpr int STAGES = Cfg::kStages;
  constexpr int kGroups = kEpiGroups<N_MAX, kReturn>;
  constexpr int kRowsB = kPair ? N_MAX / 2 : N_MAX;  // token rows of a tile that this CTA holds
  constexpr bool kFourGather = kWideGather<kGateUp, N_MAX, kReturn>;
  constexpr int kGatherThreads = kFourGather ? 128 : 64, kGatherStep = kGatherThreads / 8;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;                                 // STAGES x kStageA
  uint8_t* sB = smem + STAGES * Cfg::kStageA;         // STAGES x kStageB
  SegRing* ring = reinterpret_cast<SegRing*>(smem + STAGES * Cfg::kStageBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + 1);
  uint64_t* full_bar = bars;                          // [STAGES]
  uint64_t* empty_bar = bars + STAGES;                // [STAGES]
  uint64_t* acc_full = bars + 2 * STAGES;             // [kMaxAccStages]
  uint64_t* acc_empty = acc_full + kMaxAccStages;     // [kMaxAccStages]
  uint64_t* ret_full = acc_empty + kMaxAccStages;        // [4][kRetDepth] epilogue warp -> return warp
  uint64_t* ret_empty = ret_full + 4 * kRetDepth;     // [4][kRetDepth]
  int* ret_desc = reinterpret_cast<int*>(ret_empty + 4 * kRetDepth);  // [4][kRetDepth][4]: n_rows, row_start, mb
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ret_desc + 4 * kRetDepth * 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // Pairs have no return queue: CTA 1's mail from CTA 0 lies there, and the barriers of the gathered rows.
  PairMail* mail = reinterpret_cast<PairMail*>(ret_full);
  uint64_t* rows_bar = reinterpret_cast<uint64_t*>(mail + 1);  // [STAGES] CTA 1: the rows it gathers are there
  static_assert(sizeof(SegRing) + (2 * STAGES + 2 * kMaxAccStages + 8 * kRetDepth) * 8 + 4 * kRetDepth * 16 + 8 <= 1024,
                "barriers, segment ring and return queue");
  static_assert(!kPair || (sizeof(PairMail) + STAGES * 8 <= 8 * kRetDepth * 8 && STAGES + 2 <= kPairMail), "mail");
  uint8_t* out_stage = smem + STAGES * Cfg::kStageBytes + 1024;  // [4 epilogue warps][kOutStageBytes]
  // The fused return path runs on four extra warps (the kernel is then launched with 384 threads).
  constexpr bool with_return = kReturn;  // the down GEMM with four extra warps for the fused return path

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  // Token operand by TMA (contiguous rows) instead of the cp.async gather: warp 2 issues one bulk copy per
  // stage, warp 3 has nothing to do.
  const bool b_tma = a.b_tmap != nullptr;
  // Pairs: CTA 0 issues the MMAs.  Both fill their operands for them; all of it is counted by CTA 0's full barriers.
  const int rank = kPair ? (int)cluster_rank() : 0;
  const int cta = kPair ? (int)blockIdx.x / 2 : (int)blockIdx.x, ctas = kPair ? (int)gridDim.x / 2 : (int)gridDim.x;
  // Optional per-CTA time stamps: 0 entry, 1 dependencies met, 2 first weight tile requested, 3 first
  // operand stage complete, 4 first accumulator complete, 5 last epilogue done, 6 exit.
  unsigned long long* trace = a.trace ? a.trace + (size_t)blockIdx.x * 16 : nullptr;
  // Once-only stamps of the epilogue keep their "already written" bit in a per-thread word (reading the trace word
  // back would be a global load per 16-column group).  The two stamps inside the per-K-block loops of the producer
  // and the MMA issuer test the trace word itself instead: with the per-thread word live in those loops the
  // streaming kernels measured 0.7 us slower per unit (15 us per layer at 72 local experts), tracing off.
  uint32_t stamped = 0;
#define MF_STAMP_ONCE(i)                                   \
  do {                                                     \
    if (trace != nullptr && !(stamped & (1u << (i)))) {    \
      stamped |= 1u << (i);                                \
      trace[(i)] = global_timer_ns();                      \
    }                                                      \
  } while (0)
  if (trace && tid == 0) trace[0] = global_timer_ns();

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      // weight TMA expect_tx arrive + (one per gather thread | the token TMA expect_tx arrive)
      // (pairs: both CTAs' bytes in one arrival each; CTA 1 adds one arrival for the rows that it has gathered)
      mbar_init(&full_bar[s], b_tma ? 2 : (kPair ? 2 : 1) + kGatherThreads);
      mbar_init(&empty_bar[s], 1);                  // tcgen05.commit
      if (kPair) mbar_init(&rows_bar[s], kGatherThreads);
    }
    for (int s = 0; s < Cfg::kAccStages; ++s) {
      mbar_init(&acc_full[s], 1);   // tcgen05.commit
      mbar_init(&acc_empty[s], 4 * kGroups * (kPair ? 2 : 1));  // one per epilogue warp (of both CTAs: CTA 0's barrier)
    }
    if (kPair) mail->init();
    for (int s = 0; !kPair && s < 4 * kRetDepth; ++s) {
      mbar_init(&ret_full[s], 1);
      mbar_init(&ret_empty[s], 1);
    }
    ring->init(1 + (b_tma ? 1 : kGatherThreads / 32) + 4 * kGroups);  // UMMA, token producers, epilogue
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    if (b_tma) tma_prefetch_desc(&tmap_b);
  }
  if (kPair) __syncwarp();
  if (warp == 1) {
    if (kPair) {
      tmem_alloc_pair(tmem_slot, Cfg::kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, Cfg::kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  if (kPair) {
    __syncwarp();
    cluster_sync_all();  // the other CTA's barriers exist, both have their tensor memory
  } else {
    __syncthreads();
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // Everything above overlaps the tail of the previous kernel.  The gate/up GEMM needs the plan
  // of the metadata kernel right away, so it waits first and only then lets the next kernel start:
  // when the down GEMM starts, the plan is therefore complete and it may stream weight tiles while
  // the gate/up GEMM is still finishing; only its token-operand producers wait for the activations.
  if (tid < 8) {
    // While the predecessor runs: touch the pages read right after the wait (see touch() in common.cuh).
    const void* p = tid == 0 ? (const void*)a.plan : tid == 1 ? (const void*)a.tile_e : tid == 2 ? (const void*)a.tile_s
                  : tid == 3 ? (const void*)a.tile_n : tid == 4 ? (const void*)a.b_index : tid == 5 ? (const void*)a.row_scale
                  : tid == 6 ? (const void*)a.counters : (const void*)a.tile_wait;
    touch(p);
  }
  if (kGateUp && !a.two_blocks) {
    grid_dep_wait_cta();
    grid_dep_launch();
  } else {
    grid_dep_launch();
    // token-operand producers (act rows) and epilogue: after the whole gate/up grid, unless the activations
    // are handed over tile by tile (tile_wait), in which case nothing here depends on that grid's completion
    if (warp >= 2 && a.tile_wait == nullptr) {
      if (lane == 0) grid_dep_wait();  // one waiting thread per warp (see grid_dep_wait_cta)
      __syncwarp();
    }
  }

  if (trace && tid == 0) trace[1] = global_timer_ns();
  if (kReturn && blockIdx.x == 0 && tid == 64) {
    // Fused return path with nothing to return: the flags must still be published (thread 64 belongs to
    // the warps that waited for the previous kernel).
    if (a.plan[MF_PLAN_VALID_ROWS] == 0) {
      const unsigned pushes = *a.ret_epoch + 1u;
      *a.ret_epoch = pushes;
      publish_flags(a.ret_flag, a.ret_R, a.ret_rank, pushes * (unsigned)a.ret_C);
    }
  }
  // ---- the plan: tile count and the K cut, checked against what the caller's buffers can hold -----------
  int n_tiles = __ldcg(a.plan + MF_PLAN_N_TILES);
  const int cut = __ldcg(a.plan + a.split_word);  // 0 = stream-K, else the K split
  int slot_cols = __ldcg(a.plan + MF_PLAN_SLOT_COLS);
  if (slot_cols <= 0 || slot_cols > N_MAX) slot_cols = N_MAX;
  const long long slot_floats = (long long)Cfg::kATiles * slot_cols * kBlockM;
  const unsigned long long wait_ns = a.wait_ns;
  WorkIter work;
  work.init(a, N_MAX, n_tiles, cut, cta, ctas);
  constexpr int kCtas = kPair ? 2 : 1;  // a pair's unit is two units of the plan, next to each other
  {
    // A plan that does not fit the buffers it indexes (a tile count or a cut larger than what the caller
    // sized the scratch for) is refused here, on the device, before anything is stored: every thread of
    // every CTA sees the same words and takes the same branch.
    bool bad = n_tiles < 0 || !(cut == 0 || cut == 1 || cut == 2 || cut == 4 || cut == 8) ||
               (cut > 1 && a.k_blocks % cut != 0);
    bad = bad || (a.max_tiles > 0 && n_tiles > a.max_tiles);
    bad = bad || (a.n_counters > 0 && (long long)n_tiles * a.m_blocks * kCtas * 4 * kGroups > (long long)a.n_counters);
    bad = bad || (a.partial_floats > 0 && work.slots_needed() * kCtas * slot_floats > a.partial_floats);
    if (bad) {
      if (tid == 0) report_status(a.status, kBadArgument, 6, blockIdx.x, 0);
      n_tiles = 0;
      work.init(a, N_MAX, 0, 1, cta, ctas);
    }
  }
  // MMA columns of a tile: its rows in steps of 16; of 32 for a pair, whose CTAs hold one half of the rows each.
  auto tile_cols = [&](int n_rows) {
    const int n = kPair ? (n_rows + 31) & ~31 : (n_rows + 15) & ~15;
    return n < 16 * kCtas ? 16 * kCtas : n;
  };
  // Block (or two adjacent blocks) of a unit that is this CTA's.
  auto block_of = [&](const Seg& s) { return kPair ? 2 * s.mb + rank : s.mb; };
  auto slot_ix = [&](const Seg& s, int seg) { return (long long)slot_of(s, seg) * kCtas + rank; };

  SegReader reader(ring, abort_flag, wait_ns);
  // Token-operand producers that gather rows by index (gt: 0 .. kGatherThreads - 1).
  auto gather_rows = [&](const int gt) {
    const int r_in = gt >> 3;      // first row (its low three bits are the swizzle phase)
    const int chunk = gt & 7;      // 16-byte chunk inside the 128-byte row
    const uint32_t sw_off = (uint32_t)((chunk ^ (r_in & 7)) << 4);
    PipeState st;
    bool ok = true;
    Seg sg, nx;
    int ready_tile = -1;
    int idx[kRowsB / kGatherStep];  // source rows of the segment at hand, fetched during the previous one
    // a pair's CTA 1 gathers the rows behind the first half of the tile's columns
    auto first_row = [&](const Seg& s_) { return r_in + (kPair ? rank * (tile_cols(s_.n_rows) / 2) : 0); };
    auto row_indices = [&](const Seg& s_) {
      const int first = first_row(s_);
#pragma unroll
      for (int i = 0; i < kRowsB / kGatherStep; ++i) {
        const int n = first + kGatherStep * i;
        if (n < s_.n_rows) idx[i] = a.b_index ? __ldcg(a.b_index + s_.row_start + n) : s_.row_start + n;
      }
    };
    bool have = reader.next(sg, ok), more = false;
    if (have) row_indices(sg);
    while (ok && have) {
      if (a.tile_wait != nullptr && sg.tt != ready_tile) {
        bool got = wait_count_ge_gpu(a.tile_wait + sg.tt, a.tile_wait_target, wait_ns);
        ok = __all_sync(0xffffffffu, got);
        if (!ok) {
          if (lane == 0) {
            *abort_flag = 1;
            report_status(a.status, kGemmFullTimeout, 6, blockIdx.x, 0);
          }
          break;
        }
        ready_tile = sg.tt;
      }
      const int n_rows = sg.n_rows;
      const int n_tile = tile_cols(n_rows) / kCtas;
      const int first = first_row(sg);
      const uint8_t* rp[kRowsB / kGatherStep];
#pragma unroll
      for (int i = 0; i < kRowsB / kGatherStep; ++i) {
        const int n = first + kGatherStep * i;
        rp[i] = n < n_rows ? static_cast<const uint8_t*>(a.b_base) + (long long)idx[i] * a.b_pitch + chunk * 16 : nullptr;
      }
      for (int j = 0; j < sg.nkb; ++j) {
        const int kb = sg.kb0 + j;
        ok = mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
          break;
        }
        const uint32_t b_stage = smem_u32(sB + st.stage * Cfg::kStageB);
#pragma unroll
        for (int i = 0; i < kRowsB / kGatherStep; ++i) {
          const int n = r_in + kGatherStep * i;
          if (n < n_tile) {
            const bool live = rp[i] != nullptr;
            cp_async_16(b_stage + n * 128 + sw_off, live ? (const void*)(rp[i] + (long long)kb * 128) : a.b_base,
                        live ? 16u : 0u);
          }
        }
        cp_async_mbar_arrive_noinc(kPair && rank == 1 ? &rows_bar[st.stage] : &full_bar[st.stage]);
        st.advance(STAGES);
        // the producer warp publishes the next segment during the third K block of this one
        if (j == (sg.nkb < 4 ? sg.nkb - 1 : 3)) {
          more = reader.next(nx, ok);
          if (more) row_indices(nx);
          if (!ok) break;
        }
      }
      sg = nx;
      have = more;
    }
    // Drain this thread's cp.async operations before the CTA may exit.
    asm volatile("cp.async.wait_all;" ::: "memory");
  };
  // (The register split stands at the head of each warpgroup's branch: in front of a common join the compiler keeps everything
  // behind it within the smallest share.)
  if (warp < 4) {
    if (kFourGather) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------------------------------------------ weight TMA producer
      PipeState st;
      bool ok = true;
      SegFeedOf<kPair> feed(work, ring, abort_flag, wait_ns);
      if (kPair) {
        feed.mail = mail;
        feed.rank = rank;
      }
      // Tiles of up to 64 rows are decode: an expert usually has one tile, and its weights are then read once per forward.
      // Skewed routing gives a hot expert several that read the same blocks, but they run close together and most blocks are
      // still read once: evict-first / normal, us per layer, 1 token 81 / 96, 128 tokens 1325 / 1347 (bf16, 288 experts), 8
      // tokens e4m3 220 / 241; zipf popularity: 100 tokens on 36 experts bf16 149 / 160, e4m3 113 / 126, 128 on 288 e4m3
      // 116 / 129, 250 on 72 e4m3 (inter 2048) 223 / 230.
      const uint64_t policy = N_MAX <= 64 ? l2_evict_first() : l2_evict_normal();
      Seg sg;
      bool have = feed.first(sg);
      if (N_MAX >= 256 && !have && a.w_wait != nullptr && blockIdx.x == 0) {
        // A grid without segments (a rank that received no rows, a refused plan) waits for no token tile and no counter, but the
        // GEMM before it expands all the same: what follows may set the counter back and write to the weights' scratch, and has
        // an edge from this grid's end only.
        if (lane == 0) grid_dep_wait();
        __syncwarp();
      }
      if (N_MAX >= 256 && have && a.w_wait != nullptr) {
        // the weights are expanded by the GEMM before this one
        const bool got = lane != 0 || wait_count_ge_gpu(a.w_wait, a.w_wait_target, wait_ns);
        ok = __all_sync(0xffffffffu, got);
        __syncwarp();             // lane 0's acquire comes before what the other lanes do (the vote orders no memory)
        fence_proxy_async_all();  // the copies below, by whichever lane, come after the acquire
        if (!ok && lane == 0) {
          *abort_flag = 1;
          report_status(a.status, kGemmFullTimeout, 9, blockIdx.x, 0);
        }
      }
      while (ok && have) {
        const int row0 = sg.e * a.rows_per_expert + block_of(sg) * (a.two_blocks ? 2 * kBlockM : kBlockM);
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 0, blockIdx.x, 0);
            break;
          }
          if (elect_one()) {
            if (!kPair || rank == 0) mbar_arrive_expect_tx(&full_bar[st.stage], Cfg::kStageA * kCtas);
            uint8_t* dst = sA + st.stage * Cfg::kStageA;
            if (trace && trace[2] == 0) trace[2] = global_timer_ns();  // see the note at MF_STAMP_ONCE
            if (kPair) {
              const uint32_t bar = cluster_map(smem_u32(&full_bar[st.stage]), 0);
              tma_load_2d_pair(dst, &tmap_w, bar, kb * 64, row0, policy);
              tma_load_2d_pair(dst + kTileBytesA, &tmap_w, bar, kb * 64, row0 + a.up_row_offset, policy);
            } else {
              tma_load_2d(dst, &tmap_w, &full_bar[st.stage], kb * 64, row0, policy);
              if (kGateUp) tma_load_2d(dst + kTileBytesA, &tmap_w, &full_bar[st.stage], kb * 64, row0 + a.up_row_offset, policy);
            }
          }
          __syncwarp();
          st.advance(STAGES);
          feed.advance();
        }
        if (ok) have = feed.next(sg);
      }
      if (feed.bad_tile && lane == 0) report_status(a.status, kBadArgument, 7, blockIdx.x, 0);
      // Pairs: the last MMAs' commits arrive in both CTAs; neither leaves before.
      for (int s = 0; kPair && ok && s < STAGES; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
        st.advance(STAGES);
      }
      if (!ok) {
        // Give copies that are still in flight a moment to land before the CTA goes away.
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) __nanosleep(1000);
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ UMMA issuer
      PipeState st, acc;
      bool ok = true;
      Seg sg;
      while (ok && reader.next(sg, ok)) {
        if (kPair && rank == 1) {
          // CTA 1 tells CTA 0 that its gathered rows are there
          for (int j = 0; !b_tma && j < sg.nkb; ++j) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&rows_bar[st.stage], st.phase, abort_flag, wait_ns));
            if (!ok) {
              if (lane == 0) report_status(a.status, kGemmFullTimeout, 1, blockIdx.x, 0);
              break;
            }
            fence_proxy_async_smem();
            if (lane == 0) mbar_arrive_cluster(cluster_map(smem_u32(&full_bar[st.stage]), 0));
            __syncwarp();
            st.advance(STAGES);
          }
          continue;
        }
        const uint32_t n_tile = (uint32_t)tile_cols(sg.n_rows);
        const uint32_t idesc = umma_idesc(1, 1, kBlockM * kCtas, n_tile);
        const bool wide = Cfg::kWide && n_tile > 128;
        PipeState acc2 = acc;  // a wide unit's second stage
        acc2.advance(Cfg::kAccStages);
        ok = mbar_wait_bounded(&acc_empty[acc.stage], acc.phase ^ 1u, abort_flag, wait_ns);
        if (wide && ok) ok = mbar_wait_bounded(&acc_empty[acc2.stage], acc2.phase ^ 1u, abort_flag, wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmAccTimeout, 1, blockIdx.x, 0);
          break;
        }
        tc_fence_after_sync();
        const uint32_t d0 = tmem_base + (wide ? 0 : acc.stage * Cfg::kStageCols);
        const uint32_t d1 = d0 + (Cfg::kWide && !wide ? 128 : N_MAX);
        for (int j = 0; j < sg.nkb; ++j) {
          ok = mbar_wait_bounded(&full_bar[st.stage], st.phase, abort_flag, wait_ns);
          ok = __all_sync(0xffffffffu, ok);
          if (trace && lane == 0 && trace[3] == 0) trace[3] = global_timer_ns();
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmFullTimeout, 1, blockIdx.x, 0);
            break;
          }
          tc_fence_after_sync();
          if (!b_tma) fence_proxy_async_smem();  // the gathered rows
          const uint64_t a_desc = umma_desc_sw128(smem_u32(sA + st.stage * Cfg::kStageA));
          const uint64_t b_desc = umma_desc_sw128(smem_u32(sB + st.stage * Cfg::kStageB));
          if (kGateUp) umma_block<false, kPair>(d0, d1, a_desc, a_desc + (kTileBytesA >> 4), b_desc, idesc, j > 0 ? 1u : 0u);
          else umma_block<false>(d0, a_desc, b_desc, idesc, j > 0 ? 1u : 0u);
          if (kPair) umma_commit_pair(&empty_bar[st.stage]);
          else umma_commit(&empty_bar[st.stage]);
          st.advance(STAGES);
        }
        if (!ok) break;
        if (kPair) {
          umma_commit_pair(&acc_full[acc.stage]);
          if (wide) umma_commit_pair(&acc_full[acc2.stage]);
        } else {
          umma_commit(&acc_full[acc.stage]);
          if (wide) umma_commit(&acc_full[acc2.stage]);
        }
        acc.advance(Cfg::kAccStages);
        if (wide) acc.advance(Cfg::kAccStages);
      }
    } else if (b_tma) {
      // ------------------------------------------------------------------ token-operand producer (TMA)
      if (warp == 2) {
        PipeState st;
        bool ok = true;
        Seg sg;
        int ready_tile = -1;
        const int box_rows = a.b_box_rows > 0 ? a.b_box_rows : N_MAX;
        while (ok && reader.next(sg, ok)) {
          if (a.tile_wait != nullptr && sg.tt != ready_tile) {
            // the tile's activations are final once every gate/up unit of the tile has reported its four quarters
            bool got = true;
            if (lane == 0) got = wait_count_ge_gpu(a.tile_wait + sg.tt, a.tile_wait_target, wait_ns);
            ok = __all_sync(0xffffffffu, got);
            __syncwarp();
            fence_proxy_async_all();  // the TMA reads below, by whichever lane, come after the acquire
            if (!ok) {
              if (lane == 0) {
                *abort_flag = 1;
                report_status(a.status, kGemmFullTimeout, 6, blockIdx.x, 0);
              }
              break;
            }
            ready_tile = sg.tt;
          }
          const int cols = tile_cols(sg.n_rows) / kCtas;  // (pairs: this CTA's half of the tile's columns)
          const int n_box = kPair ? (cols + box_rows - 1) / box_rows : max(1, (sg.n_rows + box_rows - 1) / box_rows);
          const int first = sg.row_start + rank * cols;
          for (int j = 0; j < sg.nkb; ++j) {
            const int kb = sg.kb0 + j;
            ok = mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
              if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
              break;
            }
            if (elect_one()) {
              // as many boxes as hold the tile's rows: rows past the tile (the next expert's entries, or zero fill
              // past the end of the buffer) land in smem rows the MMA does not read or in accumulator columns the
              // epilogue skips
              if (!kPair || rank == 0) mbar_arrive_expect_tx(&full_bar[st.stage], n_box * box_rows * 128 * kCtas);
              for (int i = 0; i < n_box; ++i) {
                uint8_t* dst = sB + st.stage * Cfg::kStageB + i * box_rows * 128;
                if (kPair)
                  tma_load_2d_pair(dst, &tmap_b, cluster_map(smem_u32(&full_bar[st.stage]), 0), kb * 64, first + i * box_rows, l2_evict_normal());
                else
                  tma_load_2d(dst, &tmap_b, &full_bar[st.stage], kb * 64, sg.row_start + i * box_rows);
              }
            }
            __syncwarp();
            st.advance(STAGES);
          }
        }
        if (!ok) {
          const unsigned long long t0 = global_timer_ns();
          while (global_timer_ns() - t0 < 100000ull) __nanosleep(1000);
        }
      }
    } else if (!kFourGather) {
      gather_rows(tid - 64);
    } else if (a.expand_src != nullptr) {
      // ------------------------------------------------------------------ the down GEMM's weights, by two warps that have nothing to do
      const int n = expand_pieces(a, 2 * blockIdx.x + (warp - 2), 2 * gridDim.x, lane);
      __threadfence();  // every lane's stores are visible device-wide before the count
      __syncwarp();
      if (lane == 0 && n > 0) atomicAdd(a.expand_done, n);
    }
  } else if (kFourGather && warp >= 12) {
    if (kFourGather) asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    if (!b_tma) gather_rows(tid - 384);
  } else if (warp < 4 + 4 * kGroups) {
    if (kFourGather) asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    // ------------------------------------------------------------------ epilogue
    const int wq = warp & 3;                 // TMEM lane quarter this warp may read
    const int grp = (warp - 4) >> 2;         // column group (0 unless kGroups == 2)
    const int row = wq * 32 + lane;          // weight row inside the block
    PipeState acc;
    PipeState rq;                            // position in this quarter's return queue
    bool ok = true;
    // Hand a finished unit (final y values stored) to this quarter's return warp.  n_rows < 0 ends it.
    auto enqueue_return = [&](int n_rows_, int row_start_, int mb_) -> bool {
      __threadfence();  // the y stores of all lanes are visible device-wide before the hand-over
      __syncwarp();
      const int slot = wq * kRetDepth + rq.stage;
      bool k = mbar_wait_bounded(&ret_empty[slot], rq.phase ^ 1u, abort_flag, wait_ns);
      k = __all_sync(0xffffffffu, k);
      if (!k) return false;
      if (lane == 0) {
        int* d = ret_desc + slot * 4;
        d[0] = n_rows_;
        d[1] = row_start_;
        d[2] = mb_;
        mbar_arrive(&ret_full[slot]);
      }
      __syncwarp();
      rq.advance(kRetDepth);
      return true;
    };
    auto acc_free = [&](int stage) {
      if (kPair) mbar_arrive_cluster(cluster_map(smem_u32(&acc_empty[stage]), 0));
      else mbar_arrive(&acc_empty[stage]);
    };
    Seg sg;
    while (ok && reader.next(sg, ok)) {
      const int mb = block_of(sg);
      const int n_rows = sg.n_rows;
      const int row_start = sg.row_start;
      const int n_tile = tile_cols(n_rows);
      const bool wide = Cfg::kWide && n_tile > 128;
      PipeState acc2 = acc;
      acc2.advance(Cfg::kAccStages);
      ok = mbar_wait_bounded(&acc_full[acc.stage], acc.phase, abort_flag, wait_ns);
      if (wide && ok) ok = mbar_wait_bounded(&acc_full[acc2.stage], acc2.phase, abort_flag, wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (warp == 4 && lane == 0) MF_STAMP_ONCE(4);
      if (!ok) {
        if (lane == 0) report_status(a.status, kGemmAccTimeout, 3, blockIdx.x, 0);
        break;
      }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(wq * 32) << 16) + (wide ? 0 : acc.stage * Cfg::kStageCols);
      const uint32_t tup = taddr + (Cfg::kWide && !wide ? 128 : N_MAX);
      const long long out_col = (long long)mb * (a.two_blocks ? 2 * kBlockM : kBlockM) + row;

      const bool scaled = a.row_scale != nullptr && (!kGateUp || a.two_blocks);
      // this warp group's share of the token columns (whole 16-column groups)
      const int c_half = kGroups == 2 ? ((n_tile / 16 + 1) / 2) * 16 : n_tile;
      const int c_begin = grp * c_half;
      const int c_end = (kGroups == 2 && grp == 0) ? c_half : n_tile;
      const int counter_ix = ((sg.unit * kCtas + rank) * 4 + wq) * kGroups + grp;
      if (sg.nseg == 1) {
        // A real loop over 16-column groups (one copy of the code: unrolled over the whole tile it no longer fits
        // the instruction cache, and every group is executed once per unit).  Lane l fetches the routing weight of
        // column c0 + (l & 15) one group ahead.
        auto scale_of = [&](int c0) {
          const int n = c0 + (lane & 15);
          return (scaled && n < n_rows) ? __ldcg(a.row_scale + row_start + n) : 1.f;
        };
        float s_next = scale_of(c_begin);
        // 16-byte stores need rows that start on 16 bytes
        const bool wide_stores = (a.out_pitch & 7) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
        uint8_t* stage = out_stage + (warp - 4) * kOutStageBytes;
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + (long long)row_start * a.out_pitch + (out_col - lane);
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_end && wide_stores; c0 += 16) {
          uint32_t g[16], up[16];
          tmem_ld_16x16(taddr + c0, g);
          tmem_ld_16x16(taddr + (16u << 16) + c0, g + 8);
          if (kGateUp) {
            tmem_ld_16x16(tup + c0, up);
            tmem_ld_16x16(tup + (16u << 16) + c0, up + 8);
          }
          const float s_cur = s_next;
          s_next = scale_of(c0 + 16);
          tmem_ld_wait();
          if (warp == 4 && lane == 0) MF_STAMP_ONCE(8);
          float v[16], w[16], sc[16], s4[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) s4[j] = scaled ? __shfl_sync(0xffffffffu, s_cur, 8 * (j >> 1) + 2 * (lane & 3) + (j & 1)) : 1.f;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            v[j] = __uint_as_float(g[j]);
            w[j] = kGateUp ? __uint_as_float(up[j]) : 0.f;
            sc[j] = s4[(j >> 2 & 1) * 2 + (j & 1)];
          }
          finish<kGateUp, 16>(a, v, w, sc);
          __nv_bfloat16* p = out + (long long)c0 * a.out_pitch;
          store_16x32(v, stage, lane, p, a.out_pitch, n_rows - c0);
          if (kGateUp && a.two_blocks) store_16x32(w, stage, lane, p + kBlockM, a.out_pitch, n_rows - c0);
          if (warp == 4 && lane == 0) MF_STAMP_ONCE(9);
        }
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_end && !wide_stores; c0 += 16) {
          uint32_t g[16], up[16];
          tmem_ld_16(taddr + c0, g);
          if (kGateUp) tmem_ld_16(tup + c0, up);
          const float s_cur = s_next;
          s_next = scale_of(c0 + 16);
          tmem_ld_wait();
          float v[16], w[16], sc[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            v[j] = __uint_as_float(g[j]);
            w[j] = kGateUp ? __uint_as_float(up[j]) : 0.f;
            sc[j] = scaled ? __shfl_sync(0xffffffffu, s_cur, j) : 1.f;
          }
          finish_store<kGateUp, 16>(a, v, w, sc, c0, n_rows, row_start, out_col);
        }
        if (warp == 4 && lane == 0) MF_STAMP_ONCE(10);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          acc_free(acc.stage);
          if (wide) acc_free(acc2.stage);
        }
        if (a.tile_done != nullptr) {
          __threadfence();  // every lane's stores are visible device-wide before the count
          __syncwarp();
          if (lane == 0) atomicAdd(a.tile_done + sg.tt, 1);
        }
        if (with_return) ok = enqueue_return(n_rows, row_start, mb);
      } else {
        // The unit is cut along K: park the fp32 partial sums, then the last quarter-warp to arrive adds
        // the segments in K order.
        float* mine = a.partial + slot_ix(sg, sg.seg) * slot_floats;
        for (int c0 = c_begin; c0 < c_end; c0 += 16) {
          uint32_t g[16], up[16];
          tmem_ld_16(taddr + c0, g);
          if (kGateUp) tmem_ld_16(tup + c0, up);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int n = c0 + j;
            if (n < n_rows) {
              __stcg(&mine[(long long)n * kBlockM + row], __uint_as_float(g[j]));
              if (kGateUp) __stcg(&mine[(long long)(slot_cols + n) * kBlockM + row], __uint_as_float(up[j]));
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          acc_free(acc.stage);
          if (wide) acc_free(acc2.stage);
        }
        __threadfence();
        __syncwarp();
        int old = 0;
        if (lane == 0) old = atomicAdd(&a.counters[counter_ix], 1);
        old = __shfl_sync(0xffffffffu, old, 0);
        if (old == sg.nseg - 1) {
          __threadfence();
          // Eight token columns at a time: their loads are independent and issued together (a loop that
          // took one column per L2 round trip cost tens of microseconds on 64-column tiles); the sums
          // still run over the segments in K order for every column.
          constexpr int kFix = 8;
          const int n_stop = n_rows < c_end ? n_rows : c_end;  // this group's columns that hold rows
          for (int n0 = c_begin; n0 < n_stop; n0 += kFix) {
            float v[kFix], w[kFix];
#pragma unroll
            for (int j = 0; j < kFix; ++j) v[j] = w[j] = 0.f;
            for (int s = 0; s < sg.nseg; ++s) {
              const float* p = a.partial + slot_ix(sg, s) * slot_floats;
              float pv[kFix], pw[kFix];
#pragma unroll
              for (int j = 0; j < kFix; ++j) {
                const int n = n0 + j;
                pv[j] = n < n_rows ? __ldcg(&p[(long long)n * kBlockM + row]) : 0.f;
                pw[j] = (kGateUp && n < n_rows) ? __ldcg(&p[(long long)(slot_cols + n) * kBlockM + row]) : 0.f;
              }
#pragma unroll
              for (int j = 0; j < kFix; ++j) {
                v[j] += pv[j];
                w[j] += pw[j];
              }
            }
            float sc[kFix];
#pragma unroll
            for (int j = 0; j < kFix; ++j) sc[j] = (scaled && n0 + j < n_rows) ? __ldcg(a.row_scale + row_start + n0 + j) : 1.f;
            finish_store<kGateUp, kFix>(a, v, w, sc, n0, n_rows, row_start, out_col);
          }
          if (lane == 0) a.counters[counter_ix] = 0;
          if (a.tile_done != nullptr) {
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicAdd(a.tile_done + sg.tt, 1);
          }
          if (with_return) ok = enqueue_return(n_rows, row_start, mb);
        }
      }
      acc.advance(Cfg::kAccStages);
      if (wide) acc.advance(Cfg::kAccStages);
      if (trace && warp == 4 && lane == 0) {
        const unsigned long long now = global_timer_ns();
        trace[5] = now;
        if (!(stamped & (1u << 7))) {
          stamped |= 1u << 7;
          trace[7] = now;
        }
      }
    }
    if (with_return) enqueue_return(-1, 0, 0);  // tell the return warp that nothing more will come
  } else {
    // ------------------------------------------------------------------ return warps (fused owner reduce + push)
    const int wq = warp & 3;
    PipeState rq;
    int completed = 0;
    while (true) {
      const int slot = wq * kRetDepth + rq.stage;
      bool k = mbar_wait_bounded(&ret_full[slot], rq.phase, abort_flag, wait_ns);
      k = __all_sync(0xffffffffu, k);
      if (!k) {
        if (lane == 0) report_status(a.status, kGemmAccTimeout, 5, blockIdx.x, 0);
        break;
      }
      const int* d = ret_desc + slot * 4;
      const int n_rows = d[0], row_start = d[1], mb = d[2];
      __syncwarp();
      if (lane == 0) mbar_arrive(&ret_empty[slot]);
      rq.advance(kRetDepth);
      if (n_rows < 0) break;
      completed += return_rows(a, n_rows, row_start, mb, wq, lane);
    }
    return_finish(a, completed, lane);
  }

  __syncwarp();
  tc_fence_before_sync();
  if (kPair) cluster_sync_all();  // neither CTA leaves while the other may still use its memories
  else __syncthreads();
  if (trace && tid == 0) trace[6] = global_timer_ns();
  if (warp == 1) {
    tc_fence_after_sync();
    if (kPair) tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    else tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// -------------------------------------------------------------------------------------------------
// host side
// -------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(p);
  return fn;
}

#undef MF_STAMP_ONCE

template <bool kGateUp, int N_MAX, bool kReturn = false, bool kPair = false>
static int launch(const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  using Cfg = GemmCfg<kGateUp, N_MAX, kPair>;
  // The shared-memory attribute belongs to (function, device): set it once per device this process drives.
  static bool configured[kMaxDevices] = {};
  auto kern = grouped_gemm_kernel<kGateUp, N_MAX, kReturn, kPair>;
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess) return (int)de;
  if (dev < 0 || dev >= kMaxDevices || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < kMaxDevices) configured[dev] = true;
  }
  CUtensorMap tm, tb;
  memcpy(&tm, tmap, sizeof(tm));
  memcpy(&tb, args->b_tmap ? args->b_tmap : tmap, sizeof(tb));
  const int threads = kLaunchThreads<kGateUp, N_MAX, kReturn>;
  mf_gemm_args b = *args;
  if (kPair) {
    b.m_blocks /= 2;
    grid &= ~1;
  }
  return (int)launch_cluster(kern, dim3(grid), dim3(threads), Cfg::kSmemBytes, stream, true, kPair ? 2 : 1, tm, tb, b);
}

// Two accumulators (gate and up, or two weight blocks) on tiles of up to 256 rows: CTA pairs wherever they can be formed, that
// is, for an even number of units per token tile, two CTAs or more, and token boxes that fit one half of a tile.  They are the
// faster form for all tiles of this height (whole layer, single / pairs: 72 experts, 85 rows expected 548 / 520, 111 rows 610 / 577
// us, 265 rows 831 / 781; 36 experts, 882 rows 1350 / 1276, 1820 rows 2901 / 2739).
static int launch_two_256(const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  if (args->expand_src != nullptr) {
    const uintptr_t all = reinterpret_cast<uintptr_t>(args->expand_src) | reinterpret_cast<uintptr_t>(args->expand_out);
    if (args->b_tmap != nullptr || !args->expand_scale || !args->expand_out || !args->expand_done || (all & 15) != 0 || args->expand_rows < 1 ||
        args->expand_cols < 1 || args->expand_rows % 128 != 0 || args->expand_cols % 128 != 0 ||
        (long long)args->expand_rows * args->expand_cols / 16 > 0x7fffffffLL - 256)
      return -12;
  }
  const bool boxes = args->b_tmap == nullptr || (args->b_box_rows > 0 && args->b_box_rows <= 128);  // a half of the rows per CTA
  if (args->m_blocks % 2 == 0 && grid >= 2 && boxes) return launch<true, 256, false, true>(tmap, args, grid, stream);
  return launch<true, 256>(tmap, args, grid, stream);
}

static int check_args(const mf_gemm_args* a, int n_max, int grid) {
  if (!a || grid < 1) return -1;
  if (n_max != 32 && n_max != 64 && n_max != 128 && n_max != 256) return -2;
  if (a->m_blocks < 1 || a->k_blocks < 1) return -3;
  if ((a->b_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(a->b_base) & 15) != 0) return -4;
  if (a->b_box_rows < 0 || (a->b_box_rows > 0 && (a->b_box_rows % 16 != 0 || n_max % a->b_box_rows != 0))) return -8;
  if (a->b_tmap != nullptr && a->b_index != nullptr) return -5;  // TMA token tiles need contiguous rows
  if (n_max != 256 && (a->expand_src != nullptr || a->w_wait != nullptr)) return -12;
  return 0;
}

}  // namespace mf

extern "C" {

int mf_make_pitched_tmap(void* out_tmap, const void* base, long long rows, long long k_elems, int elem_bytes,
                         long long pitch_bytes, int box_rows) {
  auto fn = mf::get_encode_fn();
  if (!fn) return -10;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (pitch_bytes & 15) != 0 || pitch_bytes < k_elems * elem_bytes) return -11;
  if (box_rows < 1 || box_rows > 256 || rows < 1) return -13;
  CUtensorMap tm;
  cuuint64_t dims[2] = {(cuuint64_t)k_elems, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch_bytes};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUresult r = fn(&tm, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return -12 - (int)r * 100;
  memcpy(out_tmap, &tm, sizeof(tm));
  return 0;
}

int mf_make_tile_tmap(void* out_tmap, const void* base, long long rows, long long k_elems, int elem_bytes,
                      int box_rows) {
  return mf_make_pitched_tmap(out_tmap, base, rows, k_elems, elem_bytes, k_elems * elem_bytes, box_rows);
}

int mf_make_weight_tmap(void* out_tmap, const void* w, long long rows, long long k_elems, int elem_bytes) {
  return mf_make_tile_tmap(out_tmap, w, rows, k_elems, elem_bytes, 128);
}

int mf_gemm_smem_bytes(int gate_up, int n_max) {
  if (gate_up) {
    if (n_max == 32) return mf::GemmCfg<true, 32>::kSmemBytes;
    if (n_max == 64) return mf::GemmCfg<true, 64>::kSmemBytes;
    if (n_max == 128) return mf::GemmCfg<true, 128>::kSmemBytes;
    if (n_max == 256) return mf::GemmCfg<true, 256>::kSmemBytes;
  } else {
    if (n_max == 32) return mf::GemmCfg<false, 32>::kSmemBytes;
    if (n_max == 64) return mf::GemmCfg<false, 64>::kSmemBytes;
    if (n_max == 128) return mf::GemmCfg<false, 128>::kSmemBytes;
    if (n_max == 256) return mf::GemmCfg<false, 256>::kSmemBytes;
  }
  return -1;
}

int mf_gemm_gate_up(const void* tmap, const mf_gemm_args* args, int n_max, int grid, mf_stream_t stream) {
  int c = mf::check_args(args, n_max, grid);
  if (c) return c;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n_max == 32) return mf::launch<true, 32>(tmap, args, grid, s);
  if (n_max == 64) return mf::launch<true, 64>(tmap, args, grid, s);
  if (n_max == 128) return mf::launch<true, 128>(tmap, args, grid, s);
  return mf::launch_two_256(tmap, args, grid, s);
}

int mf_gemm_down(const void* tmap, const mf_gemm_args* args, int n_max, int grid, mf_stream_t stream) {
  int c = mf::check_args(args, n_max, grid);
  if (c) return c;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (args->two_blocks) {
    // two adjacent weight blocks per unit: the kernel form with two operand tiles and two accumulators
    if (args->ret_peer != nullptr || args->up_row_offset != mf::kBlockM) return -7;
    if (n_max == 32) return mf::launch<true, 32>(tmap, args, grid, s);
    if (n_max == 64) return mf::launch<true, 64>(tmap, args, grid, s);
    if (n_max == 128) return mf::launch<true, 128>(tmap, args, grid, s);
    return mf::launch_two_256(tmap, args, grid, s);
  }
  if (args->ret_peer != nullptr) {  // owner reduce + return push fused into the epilogue (four extra warps)
    if (n_max == 32) return mf::launch<false, 32, true>(tmap, args, grid, s);
    if (n_max == 64) return mf::launch<false, 64, true>(tmap, args, grid, s);
    if (n_max == 128) return mf::launch<false, 128, true>(tmap, args, grid, s);
    return mf::launch<false, 256, true>(tmap, args, grid, s);
  }
  if (n_max == 32) return mf::launch<false, 32>(tmap, args, grid, s);
  if (n_max == 64) return mf::launch<false, 64>(tmap, args, grid, s);
  if (n_max == 128) return mf::launch<false, 128>(tmap, args, grid, s);
  return mf::launch<false, 256>(tmap, args, grid, s);
}

}  // extern "C"

// -------------------------------------------------------------------------------------------------
// Down projection without any allocation (declared in moeflow_b200.h, MF_STATIC_SCRATCH_* limits).
//
// The split-K scratch (fp32 partial sums, then the arrival counters) lives in the file-scope device
// array below instead of a caller-provided buffer.  Every GPU that loads this library holds the array
// until the process exits.  In host code the array's name is only a stand-in for the symbol; the
// device address comes from cudaGetSymbolAddress, taken once per device with that device current.
// -------------------------------------------------------------------------------------------------
namespace mf {

constexpr int kStaticNMax = 64;                                             // token rows per tile
constexpr size_t kStaticSlotFloats = (size_t)kStaticNMax * kBlockM;         // one accumulator tile
constexpr size_t kStaticPartialBytes = (size_t)MF_STATIC_SCRATCH_MAX_SLOTS * kStaticSlotFloats * sizeof(float);
constexpr size_t kStaticCounterBytes = (size_t)MF_STATIC_SCRATCH_MAX_COUNTERS * sizeof(int);

static __device__ __align__(256) unsigned char g_static_scratch[kStaticPartialBytes + kStaticCounterBytes];

// One host thread at a time per device is assumed for the first call (the table is written without a lock;
// two threads racing here would both store the same address).
static void* g_static_scratch_addr[kMaxDevices] = {nullptr};

}  // namespace mf

extern "C" int mf_gemm_down_static_scratch(const void* tmap, const mf_gemm_args* args, int max_tiles, int split,
                                           int grid, mf_stream_t stream) {
  using namespace mf;
  if (!tmap || !args || grid < 1 || max_tiles < 1) return -1;
  if (split != 1 && split != 2 && split != 4 && split != 8) return -2;
  if (args->m_blocks < 1 || args->k_blocks < 1 || args->k_blocks % split != 0) return -3;
  if ((args->b_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(args->b_base) & 15) != 0) return -4;
  // Sizes beyond the static array are refused, never truncated.
  const long long slots = (long long)max_tiles * args->m_blocks * split;
  const long long counters = (long long)max_tiles * args->m_blocks * 4;
  if (slots > MF_STATIC_SCRATCH_MAX_SLOTS) return -20;     // too many (tile, block, split) partial tiles
  if (counters > MF_STATIC_SCRATCH_MAX_COUNTERS) return -21;

  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return -22;
  if (g_static_scratch_addr[dev] == nullptr) {
    // First call on this device: resolve the symbol and size the kernel's shared memory.
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(grouped_gemm_kernel<false, kStaticNMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             GemmCfg<false, kStaticNMax>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    g_static_scratch_addr[dev] = p;
  }
  unsigned char* base = static_cast<unsigned char*>(g_static_scratch_addr[dev]);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // The array keeps whatever the previous call left: the arrival counters must start at zero.
  e = cudaMemsetAsync(base + kStaticPartialBytes, 0, (size_t)counters * sizeof(int), s);
  if (e != cudaSuccess) return (int)e;

  mf_gemm_args a = *args;
  a.partial = reinterpret_cast<float*>(base);
  a.counters = reinterpret_cast<int*>(base + kStaticPartialBytes);
  a.max_split_slots = MF_STATIC_SCRATCH_MAX_SLOTS;
  a.b_tmap = nullptr;  // this entry always gathers the token rows
  // What the kernel may index, for its own check of the plan words (they live in device memory and can
  // disagree with max_tiles / split): the whole partial area, the counters cleared above, the declared tiles.
  a.partial_floats = (long long)(kStaticPartialBytes / sizeof(float));
  a.n_counters = (int)counters;
  a.max_tiles = max_tiles;
  CUtensorMap tm;
  memcpy(&tm, tmap, sizeof(tm));
  grouped_gemm_kernel<false, kStaticNMax>
      <<<grid, kThreads, GemmCfg<false, kStaticNMax>::kSmemBytes, s>>>(tm, tm, a);
  return (int)cudaGetLastError();
}

// The one-pass metadata build (decode sizes) and what all metadata kernels share.  Included by the stand-alone metadata
// kernels and by the dispatch kernel, whose last CTA runs the pass when the only rank is this GPU.
#pragma once

#include "common.cuh"
#include "moeflow_b200.h"

namespace mf {

constexpr int kMetaBatch = 8;  // warp-wide steps whose loads are issued together

// Exclusive scan of one int per thread over the whole block; `total` gets the sum.
template <int kThreads>
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += o;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kThreads / 32 ? warp_sums[lane] : 0;
    int wi = w;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, wi, off);
      if (lane >= off) wi += o;
    }
    warp_sums[lane] = wi - w;            // exclusive prefix of the warp sums
    if (lane == 31) warp_sums[32] = wi;  // grand total
  }
  __syncthreads();
  const int res = warp_sums[warp] + incl - v;
  total = warp_sums[32];
  __syncthreads();
  return res;
}

// Row pitch of the per-warp histograms, in words: odd, so that one expert's counts in the rows of different warps lie on
// different banks.
__host__ __device__ __forceinline__ int hist_pitch(int L) { return L | 1; }

// Clears what the two GEMMs of this forward will count on: the finished quarters of the token tiles in use, and,
// for a GEMM whose units are cut along K, the arrival counters of those units.  (The counters are zero again after
// every complete forward; a forward that gave up part-way leaves some set, which is why they are cleared at all.)
// Only the words in use: clearing the arrays whole was 100 KB to 400 KB of stores by one CTA at 288 experts.
template <int kThreads>
__device__ __forceinline__ void clear_counters(const mf_meta_args& a, int n_tiles, int cut1, int cut2) {
#pragma unroll 1
  for (int i = threadIdx.x; i < min(n_tiles, a.n_tile_done); i += kThreads) a.counters1[a.n_counters1 + i] = 0;
  if (cut1 != 1)
#pragma unroll 1
    for (int i = threadIdx.x; i < min(n_tiles * a.m_blocks1 * 8, a.n_counters1); i += kThreads) a.counters1[i] = 0;
  if (cut2 != 1)
#pragma unroll 1
    for (int i = threadIdx.x; i < min(n_tiles * a.m_blocks2 * 8, a.n_counters2); i += kThreads) a.counters2[i] = 0;
}

// Cost of the K split S = 2^log_s, or kNoSplit.  In units of one K block of 64 values of streaming: a unit costs its
// K blocks plus a fixed overhead (pipeline fill, epilogue, and for S > 1 the partial-sum round trip);
// the kernel takes ceil(units * S / SMs) rounds of such units.  K is cut between steps of k_step blocks: the e4m3 kernels
// work on K blocks of 128 values (k_step 2) and refuse a split that does not divide those.  units * 8 fits 32 bits (16
// million token tiles of 32 weight blocks).
// What a cut unit costs more (split_kb blocks of streaming) depends on the kernels: 1 for bf16, 8 for e4m3, whose K blocks are
// half as long and whose fix-up is exposed.  us per layer, graph replay, split_kb 1 / 8:
//   e4m3, 64-row tiles: 288 experts, 1 token 62.0 / 57.6, 4 tokens 113 / 104, 8 tokens 174 / 166; 72 experts, 16 tokens 181 / 172;
//   e4m3, 128-row tiles: 8 experts, 10 rows 147 / 79; 4 experts, 50 rows 73.5 / 58.9; 72 experts, 40 and 400 tokens, 36 experts,
//   8 to 1000 tokens, and 144 experts, 800 tokens: not cut with either, the same within 1 %;
//   bf16: 288 experts, 1 token 67.3 / 69.9, 4 tokens 169 / 172; 72 experts, 16 tokens 306 / 309; 36 experts, 4 tokens the same.
// Units of fewer than kMinCutBlocks blocks are not cut where there are kMinCutUnits of them: the round trip takes longer than what
// it saves of the stream.  bf16, us per layer, cut / whole: 4 blocks (8 experts) 1 token 22.6 / 20.2, 8 tokens 24.3 / 20.4;
// 8 blocks (32 experts) 24.5 / 22.4, 24.6 / 22.8; 12 blocks (16 experts) 26.8 / 24.7, 27.9 / 25.8; 14 blocks, 4 tokens 28.2 / 26.9.
// With one to three units nearly the whole chip is idle, and a cut pays from 12 blocks on: 12 blocks 22.2 / 22.7, 14 blocks
// 23.4 / 23.6; 8 blocks 22.6 / 21.2, 22.6 / 21.5 and 21.8 / 20.9, 4 blocks 22.1 / 20.2.  (For so few units no line is drawn all
// the same: before the GEMMs' instruction issue got cheaper a cut paid from 8 blocks on.  At 4 to 8 blocks it costs 1 to 2 us now.)
constexpr long long kNoSplit = 0x7fffffffffffffffll;
constexpr int kMinCutBlocks = 16, kMinCutUnits = 4;
__host__ __device__ __forceinline__ long long split_cost(int log_s, int units, int k_blocks, int k_step, int n_sms, int max_slots,
                                                         int overhead_kb, int cols, int split_kb) {
  const int s = 1 << log_s;
  const int rounds = (int)(((unsigned)units * (unsigned)s + (unsigned)n_sms - 1u) / (unsigned)n_sms);
  if (s == 1) return (long long)rounds * (k_blocks + overhead_kb);
  if (k_blocks < kMinCutBlocks && units >= kMinCutUnits) return kNoSplit;
  if ((k_blocks & (s * k_step - 1)) != 0 || (k_blocks >> log_s) < 2 || (long long)units * s > max_slots) return kNoSplit;
  // the partial-sum round trip of a split unit grows with the tile's token columns (measured: splitting
  // 64-column tiles in two cost more than the idle SMs of an uneven last round)
  const int wide = cols > 16 ? (cols - 16) / 8 : 0;
  return (long long)rounds * ((k_blocks >> log_s) + overhead_kb + split_kb + wide);
}

// The cheapest of the splits 1, 2, 4, 8; ties go to the smaller one.
__host__ __device__ __forceinline__ int choose_split(int units, int k_blocks, int k_step, int n_sms, int max_slots,
                                                     int overhead_kb, int cols, int split_kb) {
  if (units <= 0) return 1;
  int best = 0;
  long long best_cost = split_cost(0, units, k_blocks, k_step, n_sms, max_slots, overhead_kb, cols, split_kb);
  for (int log_s = 1; log_s < 4; ++log_s) {
    const long long cost = split_cost(log_s, units, k_blocks, k_step, n_sms, max_slots, overhead_kb, cols, split_kb);
    if (cost < best_cost) {
      best_cost = cost;
      best = log_s;
    }
  }
  return 1 << best;
}

// K steps of the bound experts' kernels, in blocks of 64 values (1 unless the caller says 2).
__device__ __forceinline__ int k_step_of(const mf_meta_args& a) { return a.k_step == 2 ? 2 : 1; }
__device__ __forceinline__ int split_kb_of(const mf_meta_args& a) { return a.split_kb > 0 ? a.split_kb : 1; }

// The K cut of one GEMM: stream-K (0) when asked for, the units do not fill many rounds of the persistent CTAs
// (below 8 units per CTA an uneven last round costs more than the partial tiles of the cut units) and the
// scratch holds the two partial tiles a CTA may need; else the K split of choose_split.
__device__ __forceinline__ int choose_cut(const mf_meta_args& a, int units, int k_blocks, int slots, int overhead_kb,
                                          int cols) {
  if (a.stream_k && units > 0 && units < 8 * a.n_sms && units % a.n_sms != 0 && slots >= 2 * a.n_sms) return 0;
  return choose_split(units, k_blocks, k_step_of(a), a.n_sms, slots, overhead_kb, cols, split_kb_of(a));
}

// The same choice by the four lanes of a group (lane & 3 = log2 of the split it weighs; the whole warp calls): the splits
// are weighed side by side, where one thread went through them one after the other, in the tail of the pass that the GEMMs
// wait for.
__device__ __forceinline__ int choose_cut_lanes(const mf_meta_args& a, int units, int k_blocks, int slots, int overhead_kb,
                                                int cols, int log_s) {
  const long long cost = split_cost(log_s, units, k_blocks, k_step_of(a), a.n_sms, slots, overhead_kb, cols, split_kb_of(a));
  long long key = cost != kNoSplit ? cost * 4 + log_s : kNoSplit;  // ties go to the smaller split
#pragma unroll
  for (int off = 1; off < 4; off <<= 1) {
    const long long o = __shfl_xor_sync(0xffffffffu, key, off);
    key = o < key ? o : key;
  }
  if (units <= 0) return 1;
  if (a.stream_k && units < 8 * a.n_sms && units % a.n_sms != 0 && slots >= 2 * a.n_sms) return 0;
  return 1 << (int)(key & 3);
}

// ---------------------------------------------------------------------------------------------------
// Decode sizes (rows * K <= kMetaThreads * kMetaBatch = 8192 slot words): the same layout in one pass.
// Every thread keeps its (at most kMetaBatch) keys and weight bits in registers: the received rows are
// read once, with all loads of a thread in flight together; the position of an entry inside its warp's
// range is recorded while the warp histogram is built, so that after the scans the placement is pure
// arithmetic and stores (no second sweep over the rows, no second round of matching).
// Identical output to expert_meta_kernel; about a quarter of its latency.
// ---------------------------------------------------------------------------------------------------
// Shared memory: meta_smem_words(L, kThreads) ints at `sm`.  meta_begin clears the histogram (any time before the pass, with a
// barrier in between).
__host__ __device__ __forceinline__ int meta_smem_words(int L, int threads) { return threads / 32 * hist_pitch(L) + 2 * L + 40; }

struct MetaSpan {  // slot words of a warp
  int N, per, n_warps;
  __device__ __forceinline__ MetaSpan(const mf_meta_args& a, int warps) {
    N = a.rows * a.K;
    per = ((N + warps - 1) / warps + 31) & ~31;  // <= 32 * kMetaBatch by the launcher's choice of this pass
    n_warps = (N + per - 1) / per;               // warps that hold slot words (one at a single token)
  }
};

template <int kThreads>
__device__ __forceinline__ void meta_begin(const mf_meta_args& a, int* sm) {
  const int P = hist_pitch(a.L);
  const MetaSpan span(a, kThreads / 32);
#pragma unroll 1
  for (int i = threadIdx.x; i < span.n_warps * P; i += kThreads) sm[i] = 0;
  if (threadIdx.x == 0) sm[kThreads / 32 * P + 2 * a.L + 34] = sm[kThreads / 32 * P + 2 * a.L + 35] = 0;
}

// Slot words of the received rows.  `valid`: the row's flag, 0 for a row without an entry here.
struct RowSlots {
  const uint8_t* recv;
  long long pitch;
  size_t meta_off;
  int K;
  __device__ __forceinline__ explicit RowSlots(const mf_meta_args& a)
      : recv(static_cast<const uint8_t*>(a.recv)), pitch(a.pitch), meta_off((size_t)a.H * 2), K(a.K) {}
  __device__ __forceinline__ void get(int row, int slot, int& id, int& valid, int& wbits) const {
    const int* meta = reinterpret_cast<const int*>(recv + (size_t)row * pitch + meta_off);
    id = __ldcg(meta + slot);
    valid = __ldcg(meta + 2 * K);
    wbits = __ldcg(meta + K + slot);
  }
};
// The same words, [row][K] each, in shared memory.
struct SharedSlots {
  const int *id, *wbits;
  int K;
  __device__ __forceinline__ void get(int row, int slot, int& id_, int& valid, int& wbits_) const {
    id_ = id[row * K + slot];
    valid = 1;
    wbits_ = wbits[row * K + slot];
  }
};

template <int kThreads, typename Slots>
__device__ __forceinline__ void meta_one_pass(const mf_meta_args& a, const Slots& slots, int* sm, unsigned long long* trace) {
  constexpr int kWarps = kThreads / 32;
  const int L = a.L, K = a.K, P = hist_pitch(a.L);
  int* hist = sm;                       // [kWarps][P]
  int* cnt = hist + kWarps * P;         // [L]
  int* offs = cnt + L;                  // [L]
  int* warp_sums = offs + L;            // [40]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const MetaSpan span(a, kWarps);
  const int N = span.N, n_warps = span.n_warps;
  const int begin = min(N, warp * span.per), end = min(N, (warp + 1) * span.per);
  int* my_hist = hist + warp * P;

  // The only reads of the slot words: id, valid flag and weight bits of every slot word of this thread, none of them
  // used before all are requested.
  // Every instruction of this pass runs once, so it costs what its fetch costs (about 4 cycles each): the loops over batches
  // leave at the first empty one, and no loop is unrolled further than its usual count.  With all eight batches walked
  // through and 64 registers (reloads from local memory on the way) the part behind the loads took 4.2 us for one token of
  // 288 experts and 8.2 us for 128; it takes 1.8 and 4.0.
  int key[kMetaBatch], wbits[kMetaBatch], pre[kMetaBatch], flag[kMetaBatch];
#pragma unroll
  for (int b = 0; b < kMetaBatch; ++b) {
    if (begin + b * 32 >= end) break;  // warp-uniform
    const int i = begin + b * 32 + lane;
    key[b] = -1;
    wbits[b] = flag[b] = 0;
    if (i < end) {
      const int row = i / K;
      slots.get(row, i - row * K, key[b], flag[b], wbits[b]);
    }
  }
  if (trace) trace[6] = global_timer_ns();  // loads issued

  // warp histogram; pre[b] = entries of the same expert earlier in this warp's range
  const unsigned lt_mask = (1u << lane) - 1u;
  int rows_hit = 0;
  const bool k_pow2 = (K & (K - 1)) == 0 && K <= 32;
#pragma unroll
  for (int b = 0; b < kMetaBatch; ++b) {
    if (begin + b * 32 >= end) break;
    {
      if (flag[b] == 0 || key[b] < 0 || key[b] >= L) key[b] = -1;
      const unsigned same = __match_any_sync(0xffffffffu, key[b]);
      int before = 0;
      if (key[b] >= 0) before = my_hist[key[b]];
      pre[b] = before + __popc(same & lt_mask);
      __syncwarp();
      if (key[b] >= 0 && lane == __ffs(same) - 1) my_hist[key[b]] = before + __popc(same);
      __syncwarp();
      if (k_pow2) {
        // a received row is K consecutive slot words of one warp step: its hit count is a ballot away
        const unsigned live = __ballot_sync(0xffffffffu, key[b] >= 0);
        const int g0 = lane & ~(K - 1);
        const unsigned gmask = (K == 32 ? 0xffffffffu : ((1u << K) - 1u)) << g0;
        const int hits = __popc(live & gmask);
        const int i = begin + b * 32 + lane;
        if (lane == g0 && i < end) {
          if (a.row_hits != nullptr) a.row_hits[i / K] = hits;
          rows_hit += hits > 0 ? 1 : 0;
        }
      }
    }
  }
  if (k_pow2) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) rows_hit += __shfl_xor_sync(0xffffffffu, rows_hit, off);
    if (lane == 0 && rows_hit) atomicAdd(&warp_sums[35], rows_hit);
  }
  if (trace) trace[7] = global_timer_ns();  // this warp's histogram done (its loads have landed)
  __syncthreads();
  if (trace) trace[3] = global_timer_ns();  // histogram done

  // Per expert (one thread each): exclusive prefix over the warps and total count.  The counts of four warps are loaded
  // together; a warp scan per expert instead was 18 dependent rounds per warp at 288 experts.
#pragma unroll 1
  for (int e = tid; e < L; e += kThreads) {
    int run = 0;
    int* h = hist + e;
#pragma unroll 1
    for (int left = n_warps; left > 0; left -= 4, h += 4 * P) {
      const int c0 = h[0], c1 = left > 1 ? h[P] : 0, c2 = left > 2 ? h[2 * P] : 0, c3 = left > 3 ? h[3 * P] : 0;
      h[0] = run;
      if (left > 1) h[P] = run + c0;
      if (left > 2) h[2 * P] = run + c0 + c1;
      if (left > 3) h[3 * P] = run + c0 + c1 + c2;
      run += c0 + c1 + c2 + c3;
    }
    cnt[e] = run;
  }
  if (!k_pow2) {
    // general K: rows do not line up with warp steps; count their hits from the rows (cache hits by now)
    int mine = 0;
    for (int r = tid; r < a.rows; r += kThreads) {
      int hits = 0;
      for (int k = 0; k < K; ++k) {
        int id, valid, wb;
        slots.get(r, k, id, valid, wb);
        hits += (valid != 0 && id >= 0 && id < L) ? 1 : 0;
      }
      if (a.row_hits != nullptr) a.row_hits[r] = hits;
      mine += hits > 0 ? 1 : 0;
    }
    if (mine) atomicAdd(&warp_sums[35], mine);
  }
  __syncthreads();

  // scan over experts (L <= kThreads: one expert per thread): entry offsets and tile bases.  Both sums stay below 8193
  // (kThreads * kMetaBatch slot words), so one scan carries them in the halves of a word.
  const int my_cnt = tid < L ? cnt[tid] : 0;
  const int my_nt = (my_cnt + a.block_m - 1) / a.block_m;
  int total;
  const int base = block_exclusive_scan<kThreads>(my_cnt | (my_nt << 16), warp_sums, total);
  const int n_entries = total & 0xffff, n_tiles = total >> 16;
  const int my_off = base & 0xffff, my_tb = base >> 16;
  if (tid < L) {
    offs[tid] = my_off;
    a.offsets[tid] = my_off;
#pragma unroll 1
    for (int j = 0; j < my_nt; ++j) {
      const int idx = my_tb + j;
      if (idx < a.max_tiles) {
        a.tile_e[idx] = tid;
        a.tile_s[idx] = my_off + j * a.block_m;
        a.tile_n[idx] = min(a.block_m, my_cnt - j * a.block_m);
      }
    }
    if (my_cnt > 0) atomicMax(&warp_sums[34], min(my_cnt, a.block_m));
  }
  __syncthreads();
  if (warp == kWarps - 1) {
    // the plan words, by the last warp (its range of slot words is the shortest, often empty): lanes 0-3 weigh the
    // splits 1, 2, 4, 8 of the gate/up GEMM, lanes 4-7 those of the down GEMM
    const int nt = min(n_tiles, a.max_tiles);
    int cols = (warp_sums[34] + 15) & ~15;
    if (cols < 16) cols = 16;
    const bool second = (lane & 4) != 0;
    int room = a.max_split_slots;
    if (a.partial_floats > 0)  // partial tiles of 256 * cols floats (two accumulators) or 128 * cols
      room = (int)((unsigned)min((long long)0x7fffffff, a.partial_floats >> (second && !a.pair2 ? 7 : 8)) / (unsigned)cols);
    const int cut = choose_cut_lanes(a, nt * (second ? a.m_blocks2 : a.m_blocks1), second ? a.k_blocks2 : a.k_blocks1, room,
                                     second ? 8 : 4, cols, lane & 3);
    if (lane == 0) {
      warp_sums[36] = a.plan[MF_PLAN_SPLIT1] = cut;
      a.offsets[L] = n_entries;
      a.plan[MF_PLAN_N_TILES] = nt;
      a.plan[MF_PLAN_N_ENTRIES] = n_entries;
      a.plan[MF_PLAN_NEXT1] = a.plan[MF_PLAN_NEXT2] = 0;
      a.plan[MF_PLAN_SLOT_COLS] = a.partial_floats > 0 ? cols : 0;
      a.plan[MF_PLAN_VALID_ROWS] = warp_sums[35];
    } else if (lane == 4) {
      warp_sums[37] = a.plan[MF_PLAN_SPLIT2] = cut;
    }
  }
  if (trace) trace[4] = global_timer_ns();  // offsets and tiles written

  // placement: arithmetic and stores only
#pragma unroll
  for (int b = 0; b < kMetaBatch; ++b) {
    if (begin + b * 32 >= end) break;
    const int i = begin + b * 32 + lane;
    if (i < end) {
      int pos = -1;
      if (key[b] >= 0) {
        pos = offs[key[b]] + my_hist[key[b]] + pre[b];
        // pos < N always holds for a consistent buffer; the guard keeps a racing writer (a peer that runs ahead
        // in a truncated stage-timing run) from causing a stray store
        if (pos < N) {
          const int row = i / K;
          a.entry_row[pos] = row;
          a.entry_slot[pos] = i - row * K;
          a.entry_w[pos] = __int_as_float(wbits[b]);
        } else {
          pos = -1;
        }
      }
      a.inv[i] = pos;
    }
  }
  __syncthreads();  // the cuts are in warp_sums
  clear_counters<kThreads>(a, min(n_tiles, a.max_tiles), warp_sums[36], warp_sums[37]);
  if (trace) trace[5] = global_timer_ns();  // entries placed
}

}  // namespace mf

// Expert metadata: from the received rows build, on the device and in one launch,
//   * offsets[L+1]: entries of local expert e are [offsets[e], offsets[e+1]) in expert-major order,
//     stable in (row, slot);
//   * entry_row / entry_slot / entry_w for every expert-major position, and the inverse map
//     inv[row*K + slot] = position (or -1 when the slot is empty or the row is not valid);
//   * the token tiles (expert, first entry, entry count <= block_m) the grouped GEMMs iterate over;
//   * the plan words: tile count, K-split factors for both GEMMs, entry count.
// It first waits (bounded) for every source rank's dispatch flag of this forward, so the receive
// buffer is complete when it is read, and clears the counters that the GEMMs of this forward use.
//
// The stable expert-major order is a counting sort: every warp owns a contiguous range of the flat
// (row, slot) index space, counts its keys per expert, a scan over (expert, warp) turns the counts
// into start positions, and a second sweep places the entries.  No atomics, so the layout is the
// same on every run.
//
// Replaces moeflow/kernels/metadata.py:24-137 (single-CTA Triton sort), the torch
// sort/scatter_add/cumsum chain in moeflow/fixed.py:179-186 and build_tile_schedule
// (moeflow/kernels/grouped_gemm.py:83-98).
#include "common.cuh"
#include "expert_meta.cuh"
#include "moeflow_b200.h"
#include "quant.cuh"

namespace mf {

constexpr int kMetaThreads = 1024;
constexpr int kMetaWarps = kMetaThreads / 32;

__global__ void __launch_bounds__(kMetaThreads) expert_meta_kernel(const mf_meta_args a) {
  extern __shared__ int sm[];
  const int L = a.L, K = a.K, P = hist_pitch(a.L);
  int* hist = sm;                       // [kMetaWarps][P]
  int* cnt = hist + kMetaWarps * P;     // [L]
  int* offs = cnt + L;                  // [L]
  int* warp_sums = offs + L;            // [33]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long* trace = (a.trace != nullptr && tid == 0) ? a.trace : nullptr;
  if (trace) trace[0] = global_timer_ns();
  grid_dep_launch();
  for (int i = tid; i < kMetaWarps * P; i += kMetaThreads) hist[i] = 0;
  grid_dep_wait_cta();  // the dispatch kernel of this forward has completed (epoch, local rows)
  if (trace) trace[1] = global_timer_ns();
  const unsigned epoch = a.epoch ? *a.epoch : 0u;

  // counting flags: every source adds one per token position (rows / R of them) in every forward
  if (a.flags != nullptr && tid < a.R) {
    if (!wait_flag_ge(a.flags + tid, epoch * (unsigned)(a.rows / a.R), a.wait_ns))
      report_status(a.status, kDispatchFlagTimeout, tid, 0, epoch);
  }
  __syncthreads();
  if (trace) trace[2] = global_timer_ns();  // flags seen

  const int N = a.rows * K;
  int per = (N + kMetaWarps - 1) / kMetaWarps;
  per = (per + 31) & ~31;
  const int begin = min(N, warp * per), end = min(N, (warp + 1) * per);
  const uint8_t* recv = static_cast<const uint8_t*>(a.recv);
  const size_t meta_off = (size_t)a.H * 2;
  int* my_hist = hist + warp * P;

  // Keys of a batch of kMetaBatch warp-wide steps are loaded together (independent loads in flight at
  // once) before the dependent match/count steps: the received rows are cold in cache when this kernel
  // starts, and one load latency per step would dominate it.
  auto load_keys = [&](int i0, int (&key)[kMetaBatch], int (&wbits)[kMetaBatch], bool want_w) {
#pragma unroll
    for (int b = 0; b < kMetaBatch; ++b) {
      const int i = i0 + b * 32 + lane;
      key[b] = -1;
      wbits[b] = 0;
      if (i < end) {
        const int row = i / K, slot = i - row * K;
        const int* meta = reinterpret_cast<const int*>(recv + (size_t)row * a.pitch + meta_off);
        const int id = meta[slot];
        const int valid = meta[2 * K];
        const int wb = want_w ? meta[K + slot] : 0;
        if (valid != 0 && id >= 0 && id < L) {
          key[b] = id;
          wbits[b] = wb;
        }
      }
    }
  };

  // sweep 1: per-warp histogram
  for (int i0 = begin; i0 < end; i0 += 32 * kMetaBatch) {
    int key[kMetaBatch], wbits[kMetaBatch];
    load_keys(i0, key, wbits, false);
#pragma unroll
    for (int b = 0; b < kMetaBatch; ++b) {
      const unsigned same = __match_any_sync(0xffffffffu, key[b]);
      if (key[b] >= 0 && lane == __ffs(same) - 1) my_hist[key[b]] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  if (trace) trace[3] = global_timer_ns();  // histogram sweep done

  // per expert: prefix over warps, total count
  for (int e = tid; e < L; e += kMetaThreads) {
    int run = 0;
    for (int w = 0; w < kMetaWarps; ++w) {
      const int c = hist[w * P + e];
      hist[w * P + e] = run;
      run += c;
    }
    cnt[e] = run;
  }
  __syncthreads();

  // scans over experts (L <= 1024: one expert per thread): entry offsets and tile bases
  const int my_cnt = tid < L ? cnt[tid] : 0;
  int n_entries, n_tiles;
  const int my_off = block_exclusive_scan<kMetaThreads>(my_cnt, warp_sums, n_entries);
  const int my_nt = (my_cnt + a.block_m - 1) / a.block_m;
  const int my_tb = block_exclusive_scan<kMetaThreads>(my_nt, warp_sums, n_tiles);
  if (tid < L) {
    offs[tid] = my_off;
    a.offsets[tid] = my_off;
    for (int j = 0; j < my_nt; ++j) {
      const int idx = my_tb + j;
      if (idx < a.max_tiles) {
        a.tile_e[idx] = tid;
        a.tile_s[idx] = my_off + j * a.block_m;
        a.tile_n[idx] = min(a.block_m, my_cnt - j * a.block_m);
      }
    }
  }
  // per received row: number of slots that live here (the fused return path of the down GEMM needs it),
  // and the number of rows with at least one
  if (tid == 0) warp_sums[35] = 0;
  __syncthreads();
  if (a.row_hits != nullptr) {
    int mine = 0;
    for (int r = tid; r < a.rows; r += kMetaThreads) {
      const int* meta = reinterpret_cast<const int*>(recv + (size_t)r * a.pitch + meta_off);
      int hits = 0;
      if (meta[2 * K] != 0)
        for (int k = 0; k < K; ++k) hits += (meta[k] >= 0 && meta[k] < L) ? 1 : 0;
      a.row_hits[r] = hits;
      mine += hits > 0 ? 1 : 0;
    }
    if (mine) atomicAdd(&warp_sums[35], mine);
  }
  // widest token tile: the split-K partial slots are sized for it, so a decode step (few rows per
  // expert) can afford many more, smaller K splits than the worst case would allow
  if (tid == 0) warp_sums[34] = 0;
  __syncthreads();
  if (tid < L && my_cnt > 0) atomicMax(&warp_sums[34], min(my_cnt, a.block_m));
  __syncthreads();
  if (tid == 0) {
    a.offsets[L] = n_entries;
    const int nt = min(n_tiles, a.max_tiles);
    int cols = (warp_sums[34] + 15) & ~15;
    if (cols < 16) cols = 16;
    const int wide_cols = cols;
    int slots1 = a.max_split_slots, slots2 = a.max_split_slots;
    if (a.partial_floats > 0) {
      slots1 = (int)min((long long)0x7fffffff, a.partial_floats / (2ll * cols * 128));
      slots2 = (int)min((long long)0x7fffffff, a.partial_floats / ((a.pair2 ? 2ll : 1ll) * cols * 128));
    } else {
      cols = 0;  // fixed slots of the kernel's n_max columns
    }
    a.plan[MF_PLAN_N_TILES] = nt;
    warp_sums[36] = a.plan[MF_PLAN_SPLIT1] = choose_cut(a, nt * a.m_blocks1, a.k_blocks1, slots1, 4, wide_cols);
    warp_sums[37] = a.plan[MF_PLAN_SPLIT2] = choose_cut(a, nt * a.m_blocks2, a.k_blocks2, slots2, 8, wide_cols);
    a.plan[MF_PLAN_N_ENTRIES] = n_entries;
    a.plan[MF_PLAN_NEXT1] = a.plan[MF_PLAN_NEXT2] = 0;
    a.plan[MF_PLAN_SLOT_COLS] = cols;
    a.plan[MF_PLAN_VALID_ROWS] = warp_sums[35];
  }
  __syncthreads();
  clear_counters<kMetaThreads>(a, min(n_tiles, a.max_tiles), warp_sums[36], warp_sums[37]);
  if (trace) trace[4] = global_timer_ns();  // offsets, tiles and plan written

  // sweep 2: place the entries
  for (int i0 = begin; i0 < end; i0 += 32 * kMetaBatch) {
    int key[kMetaBatch], wbits[kMetaBatch];
    load_keys(i0, key, wbits, true);
#pragma unroll
    for (int b = 0; b < kMetaBatch; ++b) {
      const int i = i0 + b * 32 + lane;
      const unsigned same = __match_any_sync(0xffffffffu, key[b]);
      if (key[b] >= 0) {
        // pos < N always holds when the rows did not change between the two sweeps; the guard keeps a
        // racing writer (a peer that runs ahead in a truncated stage-timing run) from causing a stray store.
        const int pos = offs[key[b]] + my_hist[key[b]] + __popc(same & ((1u << lane) - 1u));
        if (pos < N) {
          const int row = i / K;
          a.entry_row[pos] = row;
          a.entry_slot[pos] = i - row * K;
          a.entry_w[pos] = __int_as_float(wbits[b]);
        }
        a.inv[i] = pos < N ? pos : -1;
      } else if (i < end) {
        a.inv[i] = -1;
      }
      __syncwarp();
      if (key[b] >= 0 && lane == __ffs(same) - 1) my_hist[key[b]] += __popc(same);
      __syncwarp();
    }
  }
  if (trace) trace[5] = global_timer_ns();  // entries placed
}


// Received rows -> e4m3 (layers with block-scaled experts), by the CTAs behind the first one: the two jobs read the same
// rows and neither needs the other, so the quantiser costs no launch and no time of its own.
__device__ __forceinline__ void quantise_received_rows(const mf_meta_args& a) {
  grid_dep_wait_cta();
  if (a.flags != nullptr && threadIdx.x < a.R) {
    const unsigned epoch = a.epoch ? __ldcg(a.epoch) : 0u;
    if (!wait_flag_ge(a.flags + threadIdx.x, epoch * (unsigned)(a.rows / a.R), a.wait_ns))
      report_status(a.status, kDispatchFlagTimeout, threadIdx.x, blockIdx.x, epoch);
  }
  __syncthreads();
  const int chunks = a.H / 8, groups = a.H / 128;  // chunks: a multiple of 16, so a group's threads work on one row
  const long long total = (long long)a.rows * chunks;
  const uint8_t* recv = static_cast<const uint8_t*>(a.recv);
  const size_t valid_off = (size_t)a.H * 2 + (size_t)8 * a.K;
  for (long long i = (long long)(blockIdx.x - 1) * kMetaThreads + threadIdx.x; i < total; i += (long long)(gridDim.x - 1) * kMetaThreads) {
    const int row = (int)(i / chunks), c = (int)(i - (long long)row * chunks);
    const uint8_t* src = recv + (size_t)row * a.pitch;
    if (__ldcg(reinterpret_cast<const int*>(src + valid_off)) == 0) continue;
    quant_chunk(src, c, a.xq + (size_t)row * a.H, a.xs + (size_t)row * groups);
  }
}

__global__ void __launch_bounds__(kMetaThreads) expert_meta_small_kernel(const mf_meta_args a) {
  extern __shared__ int sm[];
  if (blockIdx.x > 0) {
    if (!a.late_launch) grid_dep_launch();
    quantise_received_rows(a);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long* trace = (a.trace != nullptr && tid == 0) ? a.trace : nullptr;
  if (trace) trace[0] = global_timer_ns();
  if (!a.late_launch) grid_dep_launch();
  meta_begin<kMetaThreads>(a, sm);
  {
    const MetaSpan span(a, kMetaWarps);
    const int K = a.K, begin = min(span.N, warp * span.per), end = min(span.N, (warp + 1) * span.per);
    const uint8_t* recv = static_cast<const uint8_t*>(a.recv);
    const size_t meta_off = (size_t)a.H * 2;
    // While the dispatch kernel runs: touch every page this kernel reads or writes after the wait.
    if (tid == 0) {
      touch(a.epoch);
      touch(a.flags);
      touch(a.plan);
      touch(a.offsets);
      touch(a.tile_e);
      touch(a.tile_s);
      touch(a.tile_n);
      touch(a.row_hits);
    }
    const int i = begin + lane;
    if (i < end) {
      touch(recv + (size_t)(i / K) * a.pitch + meta_off);
      touch(a.inv + i);
      touch(a.entry_row + i);
      touch(a.entry_slot + i);
      touch(a.entry_w + i);
    }
    if (tid == 0) touch(a.counters1 + a.n_counters1);
  }
  grid_dep_wait_cta();  // the dispatch kernel of this forward has completed (epoch, local rows)
  if (trace) trace[1] = global_timer_ns();
  const unsigned epoch = a.epoch ? __ldcg(a.epoch) : 0u;
  if (a.flags != nullptr && tid < a.R) {
    if (!wait_flag_ge(a.flags + tid, epoch * (unsigned)(a.rows / a.R), a.wait_ns))
      report_status(a.status, kDispatchFlagTimeout, tid, 0, epoch);
  }
  __syncthreads();
  if (trace) trace[2] = global_timer_ns();  // flags seen

  meta_one_pass<kMetaThreads>(a, RowSlots(a), sm, trace);
}


// ---------------------------------------------------------------------------------------------------
// Multi-CTA variant for prefill sizes: the flat (row, slot) index space is cut into one contiguous
// chunk per CTA (and inside a CTA into one contiguous range per warp, as above).  Launch 1 counts:
// per-CTA expert histograms go to cta_hist.  Launch 2 recomputes its own per-warp histograms, adds the
// counts of the CTAs before it (a plain loop over cta_hist: no atomics, no waiting between CTAs, so the
// layout is again the same on every run and equal to the single-CTA kernel's) and places its entries.
// ---------------------------------------------------------------------------------------------------
struct MetaRange {
  int begin, end;
};
__device__ __forceinline__ MetaRange meta_range(int N, int n_ctas, int cta, int warp) {
  int chunk = (N + n_ctas - 1) / n_ctas;
  chunk = (chunk + 31) & ~31;
  const int cb = min(N, cta * chunk), ce = min(N, (cta + 1) * chunk);
  int per = (ce - cb + kMetaWarps - 1) / kMetaWarps;
  per = (per + 31) & ~31;
  MetaRange r;
  r.begin = min(ce, cb + warp * per);
  r.end = min(ce, cb + (warp + 1) * per);
  return r;
}

// keys (local expert id or -1) and weight bits of kMetaBatch warp-wide steps starting at i0
__device__ __forceinline__ void meta_load_keys(const mf_meta_args& a, int i0, int end, int lane, bool want_w,
                                               int (&key)[kMetaBatch], int (&wbits)[kMetaBatch]) {
  const uint8_t* recv = static_cast<const uint8_t*>(a.recv);
  const size_t meta_off = (size_t)a.H * 2;
#pragma unroll
  for (int b = 0; b < kMetaBatch; ++b) {
    const int i = i0 + b * 32 + lane;
    key[b] = -1;
    wbits[b] = 0;
    if (i < end) {
      const int row = i / a.K, slot = i - row * a.K;
      const int* meta = reinterpret_cast<const int*>(recv + (size_t)row * a.pitch + meta_off);
      const int id = meta[slot];
      const int valid = meta[2 * a.K];
      const int wb = want_w ? meta[a.K + slot] : 0;
      if (valid != 0 && id >= 0 && id < a.L) {
        key[b] = id;
        wbits[b] = wb;
      }
    }
  }
}

__device__ __forceinline__ void meta_histogram(const mf_meta_args& a, MetaRange r, int lane, int* my_hist) {
  for (int i0 = r.begin; i0 < r.end; i0 += 32 * kMetaBatch) {
    int key[kMetaBatch], wbits[kMetaBatch];
    meta_load_keys(a, i0, r.end, lane, false, key, wbits);
#pragma unroll
    for (int b = 0; b < kMetaBatch; ++b) {
      const unsigned same = __match_any_sync(0xffffffffu, key[b]);
      if (key[b] >= 0 && lane == __ffs(same) - 1) my_hist[key[b]] += __popc(same);
      __syncwarp();
    }
  }
}

__global__ void __launch_bounds__(kMetaThreads) expert_meta_count_kernel(const mf_meta_args a) {
  extern __shared__ int sm[];
  const int L = a.L, K = a.K, P = hist_pitch(a.L);
  int* hist = sm;                    // [kMetaWarps][P]
  int* warp_sums = hist + kMetaWarps * P;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cta = blockIdx.x, n_ctas = gridDim.x;
  grid_dep_launch();
  for (int i = tid; i < kMetaWarps * P; i += kMetaThreads) hist[i] = 0;
  if (tid == 0) warp_sums[0] = 0;
  grid_dep_wait_cta();  // the dispatch kernel of this forward has completed (epoch, local rows)
  const unsigned epoch = a.epoch ? *a.epoch : 0u;
  if (a.flags != nullptr && tid < a.R) {
    if (!wait_flag_ge(a.flags + tid, epoch * (unsigned)(a.rows / a.R), a.wait_ns))
      report_status(a.status, kDispatchFlagTimeout, tid, cta, epoch);
  }
  __syncthreads();

  const int N = a.rows * K;
  meta_histogram(a, meta_range(N, n_ctas, cta, warp), lane, hist + warp * P);
  __syncthreads();
  for (int e = tid; e < L; e += kMetaThreads) {
    int total = 0;
    for (int w = 0; w < kMetaWarps; ++w) total += hist[w * P + e];
    a.cta_hist[(size_t)cta * L + e] = total;
  }
  // slots per received row, and the number of rows with at least one
  const uint8_t* recv = static_cast<const uint8_t*>(a.recv);
  const size_t meta_off = (size_t)a.H * 2;
  int mine = 0;
  for (int r = cta * kMetaThreads + tid; r < a.rows; r += n_ctas * kMetaThreads) {
    const int* meta = reinterpret_cast<const int*>(recv + (size_t)r * a.pitch + meta_off);
    int hits = 0;
    if (meta[2 * K] != 0)
      for (int k = 0; k < K; ++k) hits += (meta[k] >= 0 && meta[k] < L) ? 1 : 0;
    if (a.row_hits != nullptr) a.row_hits[r] = hits;
    mine += hits > 0 ? 1 : 0;
  }
  if (mine) atomicAdd(&warp_sums[0], mine);
  __syncthreads();
  if (tid == 0 && warp_sums[0] != 0) atomicAdd(&a.acc[0], warp_sums[0]);  // a count: the order does not matter
}

__global__ void __launch_bounds__(kMetaThreads) expert_meta_place_kernel(const mf_meta_args a) {
  extern __shared__ int sm[];
  const int L = a.L, K = a.K, P = hist_pitch(a.L);
  int* hist = sm;                       // [kMetaWarps][P]
  int* cnt = hist + kMetaWarps * P;     // [L] entries of the expert over all CTAs
  int* offs = cnt + L;                  // [L] first position of this CTA's entries of the expert
  int* warp_sums = offs + L;            // [40]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cta = blockIdx.x, n_ctas = gridDim.x;
  grid_dep_launch();
  for (int i = tid; i < kMetaWarps * P + 2 * L; i += kMetaThreads) hist[i] = 0;  // and cnt, offs behind it
  if (tid == 0) warp_sums[34] = 0;
  grid_dep_wait_cta();  // the count launch has completed (and with it the dispatch kernel)
  __syncthreads();

  const int N = a.rows * K;
  const MetaRange range = meta_range(N, n_ctas, cta, warp);
  int* my_hist = hist + warp * P;
  meta_histogram(a, range, lane, my_hist);
  __syncthreads();

  // Entries of every expert in all CTAs and in those before this one.  The threads share the CTAs between them (whole warps
  // to an expert range, so that the loads are coalesced): one thread per expert went through up to 148 counts, four in
  // flight: 17 us of the kernel at 16384 slot words, 13 now.
  {
    const int span = (L + 31) & ~31, parts = kMetaThreads / span;  // L <= kMetaThreads
    const int part = tid / span, e = tid - part * span;
    if (part < parts && e < L) {
      int before = 0, total = 0;
#pragma unroll 8
      for (int c = part; c < n_ctas; c += parts) {
        const int v = a.cta_hist[(size_t)c * L + e];
        before += c < cta ? v : 0;
        total += v;
      }
      atomicAdd(&cnt[e], total);
      atomicAdd(&offs[e], before);
    }
  }
  for (int e = tid; e < L; e += kMetaThreads) {
    int run = 0;
    for (int w = 0; w < kMetaWarps; ++w) {
      const int c = hist[w * P + e];
      hist[w * P + e] = run;
      run += c;
    }
  }
  __syncthreads();

  const int my_cnt = tid < L ? cnt[tid] : 0;
  int n_entries, n_tiles;
  const int my_off = block_exclusive_scan<kMetaThreads>(my_cnt, warp_sums, n_entries);
  const int my_nt = (my_cnt + a.block_m - 1) / a.block_m;
  const int my_tb = block_exclusive_scan<kMetaThreads>(my_nt, warp_sums, n_tiles);
  if (tid < L) {
    offs[tid] += my_off;
    if (cta == 0) {
      a.offsets[tid] = my_off;
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
  }
  __syncthreads();
  if (cta == 0 && tid == 0) {
    a.offsets[L] = n_entries;
    const int nt = min(n_tiles, a.max_tiles);
    int cols = (warp_sums[34] + 15) & ~15;
    if (cols < 16) cols = 16;
    const int wide_cols = cols;
    int slots1 = a.max_split_slots, slots2 = a.max_split_slots;
    if (a.partial_floats > 0) {
      slots1 = (int)min((long long)0x7fffffff, a.partial_floats / (2ll * cols * 128));
      slots2 = (int)min((long long)0x7fffffff, a.partial_floats / ((a.pair2 ? 2ll : 1ll) * cols * 128));
    } else {
      cols = 0;
    }
    a.plan[MF_PLAN_N_TILES] = nt;
    warp_sums[36] = a.plan[MF_PLAN_SPLIT1] = choose_cut(a, nt * a.m_blocks1, a.k_blocks1, slots1, 4, wide_cols);
    warp_sums[37] = a.plan[MF_PLAN_SPLIT2] = choose_cut(a, nt * a.m_blocks2, a.k_blocks2, slots2, 8, wide_cols);
    a.plan[MF_PLAN_N_ENTRIES] = n_entries;
    a.plan[MF_PLAN_NEXT1] = a.plan[MF_PLAN_NEXT2] = 0;
    a.plan[MF_PLAN_SLOT_COLS] = cols;
    a.plan[MF_PLAN_VALID_ROWS] = a.acc[0];
    a.acc[0] = 0;  // ready for the next forward (its count launch runs after this one)
  }
  if (cta == 0) {
    __syncthreads();
    clear_counters<kMetaThreads>(a, min(n_tiles, a.max_tiles), warp_sums[36], warp_sums[37]);
  }

  for (int i0 = range.begin; i0 < range.end; i0 += 32 * kMetaBatch) {
    int key[kMetaBatch], wbits[kMetaBatch];
    meta_load_keys(a, i0, range.end, lane, true, key, wbits);
#pragma unroll
    for (int b = 0; b < kMetaBatch; ++b) {
      const int i = i0 + b * 32 + lane;
      const unsigned same = __match_any_sync(0xffffffffu, key[b]);
      if (key[b] >= 0) {
        const int pos = offs[key[b]] + my_hist[key[b]] + __popc(same & ((1u << lane) - 1u));
        if (pos < N) {
          const int row = i / K;
          a.entry_row[pos] = row;
          a.entry_slot[pos] = i - row * K;
          a.entry_w[pos] = __int_as_float(wbits[b]);
        }
        a.inv[i] = pos < N ? pos : -1;
      } else if (i < range.end) {
        a.inv[i] = -1;
      }
      __syncwarp();
      if (key[b] >= 0 && lane == __ffs(same) - 1) my_hist[key[b]] += __popc(same);
      __syncwarp();
    }
  }
}

}  // namespace mf

extern "C" int mf_plan_split(int units, int k_blocks, int n_sms, int max_slots, int overhead_kb, int cols) {
  return mf_plan_split_steps(units, k_blocks, 1, n_sms, max_slots, overhead_kb, cols);
}

extern "C" int mf_plan_split_steps(int units, int k_blocks, int k_step, int n_sms, int max_slots, int overhead_kb, int cols) {
  return mf_plan_split_costs(units, k_blocks, k_step, n_sms, max_slots, overhead_kb, cols, 1);
}

extern "C" int mf_plan_split_costs(int units, int k_blocks, int k_step, int n_sms, int max_slots, int overhead_kb, int cols, int split_kb) {
  return mf::choose_split(units, k_blocks, k_step, n_sms, max_slots, overhead_kb, cols, split_kb);
}

extern "C" int mf_expert_meta(const mf_meta_args* a, mf_stream_t stream) {
  if (!a || a->L < 1 || a->L > mf::kMetaThreads || a->R > mf::kMetaThreads || a->block_m < 1) return -1;
  const size_t smem = (size_t)mf::meta_smem_words(a->L, mf::kMetaThreads) * sizeof(int);
  static size_t configured_all[64] = {};  // per device: the attribute belongs to (function, device)
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  size_t& configured = configured_all[dev];
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e =
        cudaFuncSetAttribute(mf::expert_meta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mf::expert_meta_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mf::expert_meta_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mf::expert_meta_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = smem;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (a->n_ctas > 1) {
    if (!a->cta_hist || !a->acc || a->n_ctas > 1024) return -2;
    if (a->xq != nullptr) return -4;  // only the one-pass kernel quantises
    cudaError_t e = mf::launch_kernel(mf::expert_meta_count_kernel, dim3(a->n_ctas), dim3(mf::kMetaThreads), smem, s,
                                      !a->plain_launch, *a);
    if (e != cudaSuccess) return (int)e;
    return (int)mf::launch_kernel(mf::expert_meta_place_kernel, dim3(a->n_ctas), dim3(mf::kMetaThreads), smem, s, true,
                                  *a);
  }
  // one CTA: the register-resident one-pass kernel when every warp's range fits one batch of steps
  const long long n_words = (long long)a->rows * a->K;
  if (n_words <= (long long)mf::kMetaThreads * mf::kMetaBatch) {
    int quant_ctas = 0;
    if (a->xq != nullptr) {
      if (!a->xs || a->H % 128 != 0) return -3;
      const long long ctas = ((long long)a->rows * (a->H / 8) + mf::kMetaThreads - 1) / mf::kMetaThreads;
      quant_ctas = (int)(ctas < a->n_sms - 1 ? ctas : a->n_sms > 1 ? a->n_sms - 1 : 1);
    }
    return (int)mf::launch_kernel(mf::expert_meta_small_kernel, dim3(1 + quant_ctas), dim3(mf::kMetaThreads), smem, s,
                                  !a->plain_launch, *a);
  }
  if (a->xq != nullptr) return -4;  // only the one-pass kernel quantises
  return (int)mf::launch_kernel(mf::expert_meta_kernel, dim3(1), dim3(mf::kMetaThreads), smem, s, !a->plain_launch, *a);
}

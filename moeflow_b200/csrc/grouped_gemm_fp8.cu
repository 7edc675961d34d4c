// Block-scaled FP8 (e4m3) grouped expert GEMMs on tcgen05, and the 1x128 activation quantiser.
//
// Checkpoint format: weights are float8_e4m3fn with one fp32 scale per 128x128 block
// (weight_scale_inv); activations are quantised on the fly to e4m3 with one fp32 scale per row and
// 128-wide K group.  These scales are arbitrary fp32 numbers, not the power-of-two per-32 scales the
// hardware block-scaling mode wants, so the kernel accumulates in two levels:
//
//   per 128-wide K block:  tmp[128, n]  = W_q[128 rows, 128 k] . X_q[n, 128 k]^T      (tcgen05 kind::f8f6f4,
//                                                                                     fp32 in tensor memory)
//                          acc[r, n]   += w_scale[block(r), kb] * x_scale[n, kb] * tmp[r, n]     (registers)
//
// The weight block of a unit (128 rows) is exactly one scale-block row, and one K block of 128 bytes is
// one TMA box row and one scale-block column, so a unit needs one weight scale per K block (two for
// gate/up) and one activation scale per token and K block.  Tensor-memory accumulators are buffered per K block so
// that the promotion of block kb overlaps the MMAs of the blocks behind it.
//
// A unit is half as long as in bf16 (32 K blocks of 32 KB: 23 us at an SM's share of the memory rate), so what a
// unit costs besides its stream weighs twice as much, and everything that sat between two units is off the promotion
// warps' path:
//   * units are handed out by a counter, and every role finds its next one ready in shared memory (work_iter.cuh);
//   * one warp fills the scale tables, a unit ahead, and reports finished token tiles for the promotion warps (a
//     device-scope fence under load takes about as long as three K blocks);
//   * the gate/up epilogue quantises the activations itself (q_out): its 128 weight rows are exactly one 128-wide
//     group of the activation row, so a token's scale is a maximum over the unit's four warps.  The bf16 activations
//     are never stored, and the down GEMM starts a token tile as soon as the tile's units have reported (tile_done),
//     as in the bf16 kernels, instead of waiting for the gate/up grid and for a quantiser launch behind it.
//
// Token tiles of 128 rows have a kernel of their own (grouped_gemm_fp8_wide.cu).
//
// Everything else (swap-AB, persistent CTAs, device-side plan, split-K with ordered fix-up, bounded
// waits) is as in grouped_gemm_tc.cu.
//
// The reference has no FP8 kernel of its own: it dequantises to bf16 (moeflow/weights.py:23-27) or calls
// the serving engine's fused experts and moe_kernel_quantize_input (moeflow/integrations/vllm_pf.py:97).
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "fp8_pipe.cuh"
#include "moeflow_b200.h"
#include "quant.cuh"
#include "work_iter.cuh"

namespace mf {

// Gather threads: warp 2, or four warps of their own (12-15) in the gate/up GEMM of 64-row tiles, where one warp's 16 copy
// instructions per K block (about 90 cycles each) took longer than the K block's promotion and its weights.  The promotion
// warps then take the registers that the others give up.  Layer, us: 1 token on 288 experts 64.6 / 61.8; 250 on 72 and 64 sequences
// of the decode model 1 to 2 % less in one run, which is what runs differ by there.  The split: 88 x 128 + 192 x 256 + 40 x 128 =
// 65536, what 512 threads start with.
template <bool kGateUp, int N_MAX>
constexpr bool kF8FourGather = kGateUp && N_MAX == 64;
constexpr int kF8Tables = 2;   // scale tables: the unit being promoted and the prefetched next one
constexpr int kF8Stage = 1024;  // per promotion warp: 16 token columns x 32 outputs of the epilogue, transposed

template <bool kGateUp, int N_MAX>
struct F8Cfg {
  static constexpr int kATiles = kGateUp ? 2 : 1;
  static constexpr int kStageA = kATiles * kF8TileA;
  static constexpr int kStageB = N_MAX * 128;
  static constexpr int kStageBytes = kStageA + kStageB;
  // Promotion warps: one group of four warps (one per tensor-memory lane quarter) per 32 token columns.
  static constexpr int kGroups = N_MAX > 32 ? 2 : 1;
  static constexpr int kCols = N_MAX / kGroups;
  static constexpr int kPromo = 4 * kGroups;             // promotion warps: 4 .. 4 + kPromo - 1
  static constexpr bool kFourGather = kF8FourGather<kGateUp, N_MAX>;
  // Gate/up units of up to 32 columns go to the two groups in turn, so that one group's epilogue (activation and quantisation of
  // 16 or 32 columns take 3 to 5 us, the first one of a launch 7 with its instructions in DRAM) runs while the other
  // promotes the next unit.  With both groups at every unit (and nothing to do for the second) the four accumulators ahead
  // covered 2.7 us of it, and the weight stream stood still for the rest.
  // Calls, us: 8 tokens on 288 experts 179.7 / 177.7, 250 on 72 (inter 2048) 362 / 357, decode model of 64 246.6 / 242.8 (all before
  // both groups took part in the hand-over of every scale table, which costs up to 0.4 %).
  static constexpr bool kTurns = kGateUp && kGroups == 2;
  static constexpr int kGather = kFourGather ? 128 : 32;  // threads
  static constexpr int kThreads = 128 + 32 * kPromo + (kFourGather ? 128 : 0);
  static constexpr int kTableFloats = N_MAX * kF8MaxKb + 2 * kF8MaxKb;  // x scales [kb][n], weight scales [2][kb]
  static constexpr int kTableBytes = kF8Tables * kTableFloats * 4;
  static constexpr int kBarrierBytes = 1024;             // barriers and the segment ring
  static constexpr int kExtra = kPromo * kF8Stage + kBarrierBytes;
  static constexpr int kFree = 227 * 1024 - 1024 /*alignment*/ - kTableBytes - kExtra;
  static constexpr int kStages = kFree / kStageBytes > 8 ? 8 : kFree / kStageBytes;
  static constexpr int kTmpCols = kATiles * N_MAX;
  // One tensor-memory accumulator per K block in flight: the MMA -> promotion -> MMA round trip is about a
  // microsecond, so two stages cannot keep up with the weight stream; use all 512 columns (at most 8 stages).
  static constexpr int kTmpStages = 512 / kTmpCols > 8 ? 8 : 512 / kTmpCols;
  static constexpr int kTmemCols = kTmpStages * kTmpCols;
  static constexpr int kSmemBytes = kStages * kStageBytes + kTableBytes + kExtra + 1024;
};

template <bool kGateUp, int N_MAX>
__global__ void __launch_bounds__(F8Cfg<kGateUp, N_MAX>::kThreads, 1)
grouped_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_b,
                        const mf_gemm_args a) {
  using Cfg = F8Cfg<kGateUp, N_MAX>;
  constexpr int STAGES = Cfg::kStages;
  constexpr int GROUPS = Cfg::kGroups;
  constexpr int COLS = Cfg::kCols;
  constexpr int PROMO_WARPS = Cfg::kPromo;
  static_assert(STAGES >= 2 && Cfg::kSmemBytes <= 227 * 1024, "shared memory");
  static_assert((int)sizeof(SegRing) + (2 * STAGES + 2 * Cfg::kTmpStages + 2 * kF8Tables + GROUPS + 2) * 8 + 8 + 4 * GROUPS <=
                    Cfg::kBarrierBytes, "barriers");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * Cfg::kStageA;
  float* sTable = reinterpret_cast<float*>(smem + STAGES * Cfg::kStageBytes);  // [kF8Tables][kTableFloats]
  uint8_t* sStage = smem + STAGES * Cfg::kStageBytes + Cfg::kTableBytes;       // [PROMO_WARPS][kF8Stage]
  SegRing* ring = reinterpret_cast<SegRing*>(sStage + PROMO_WARPS * kF8Stage);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ring + 1);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmp_full = empty_bar + STAGES;
  uint64_t* tmp_empty = tmp_full + Cfg::kTmpStages;
  uint64_t* tbl_bar = tmp_empty + Cfg::kTmpStages;  // [kF8Tables] table filled
  uint64_t* tbl_free = tbl_bar + kF8Tables;         // [kF8Tables] table no longer read
  uint64_t* grp_bar = tbl_free + kF8Tables;         // [GROUPS] the group's four warps met (epilogue)
  uint64_t* epi_bar = grp_bar + GROUPS;             // [2] a unit's outputs are stored (all promotion warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(epi_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* grp_last = abort_flag + 1;          // [GROUPS] a cut unit's arrival count, seen by the group's first warp

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool b_tma = a.b_tmap != nullptr;  // token tiles by TMA (contiguous rows) instead of the 16-byte gather
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], b_tma ? 2 : 1 + Cfg::kGather);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < Cfg::kTmpStages; ++s) {
      mbar_init(&tmp_full[s], 1);
      mbar_init(&tmp_empty[s], PROMO_WARPS);
    }
    for (int s = 0; s < kF8Tables; ++s) {
      mbar_init(&tbl_bar[s], 1);
      mbar_init(&tbl_free[s], PROMO_WARPS);
    }
    for (int s = 0; s < GROUPS; ++s) mbar_init(&grp_bar[s], 4);
    for (int s = 0; s < 2; ++s) mbar_init(&epi_bar[s], PROMO_WARPS);
    ring->init(2 + (b_tma ? 1 : Cfg::kGather / 32) + PROMO_WARPS);  // UMMA, table warp, token producers, promotion warps
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    if (b_tma) tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (tid < 6) {
    // while the predecessor runs: touch the pages read right after the wait (see touch() in common.cuh)
    const void* p = tid == 0 ? (const void*)a.plan : tid == 1 ? (const void*)a.tile_e : tid == 2 ? (const void*)a.tile_s
                  : tid == 3 ? (const void*)a.tile_n : tid == 4 ? (const void*)a.b_index : (const void*)a.tile_wait;
    touch(p);
  }
  // As in the bf16 kernels: the gate/up GEMM waits for the plan and only then lets the next kernel start, so the
  // down GEMM finds the plan complete; with tile-level hand-over nothing in it waits for the gate/up grid as a whole.
  if (kGateUp || a.tile_wait == nullptr) {
    grid_dep_wait_cta();
    grid_dep_launch();
  } else {
    grid_dep_launch();
  }

  int n_tiles = __ldcg(a.plan + MF_PLAN_N_TILES);
  const int cut = __ldcg(a.plan + a.split_word);  // 0 = stream-K, else the K split
  int slot_cols = __ldcg(a.plan + MF_PLAN_SLOT_COLS);
  if (slot_cols <= 0 || slot_cols > N_MAX) slot_cols = N_MAX;
  const long long slot_floats = (long long)Cfg::kATiles * slot_cols * kF8BlockM;
  const unsigned long long wait_ns = a.wait_ns;
  WorkIter work;
  work.init(a, N_MAX, n_tiles, cut, blockIdx.x, gridDim.x);
  {
    // the plan is checked against the buffers it indexes before anything is stored (same rule as the bf16 kernel)
    bool bad = n_tiles < 0 || !(cut == 0 || cut == 1 || cut == 2 || cut == 4 || cut == 8) ||
               (cut > 1 && a.k_blocks % cut != 0);
    bad = bad || (a.max_tiles > 0 && n_tiles > a.max_tiles);
    bad = bad || (a.n_counters > 0 && (long long)n_tiles * a.m_blocks * 4 * GROUPS > (long long)a.n_counters);
    bad = bad || (a.partial_floats > 0 && work.slots_needed() * slot_floats > a.partial_floats);
    if (bad) {
      if (tid == 0) report_status(a.status, kBadArgument, 6, blockIdx.x, 0);
      n_tiles = 0;
      work.init(a, N_MAX, 0, 1, blockIdx.x, gridDim.x);
    }
  }
  auto tile_ready = [&](int tt) -> bool {  // bounded; one lane asks
    bool got = true;
    if (lane == 0) got = wait_count_ge_gpu(a.tile_wait + tt, a.tile_wait_target, wait_ns);
    got = __all_sync(0xffffffffu, got);
    if (!got && lane == 0) {
      *abort_flag = 1;
      report_status(a.status, kGemmFullTimeout, 6, blockIdx.x, 0);
    }
    return got;
  };
  SegReader reader(ring, abort_flag, wait_ns);

  // (The register split stands at the head of each warpgroup's branch: in front of a common join the compiler keeps everything
  // behind it within the smallest share.)
  if (warp < 4) {
    if (Cfg::kFourGather) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 0) {
      // ---------------------------------------------------------------- weight TMA producer, hands out the segments
      F8Pipe st;
      bool ok = true;
      SegFeed feed(work, ring, abort_flag, wait_ns);
      const uint64_t policy = l2_evict_first();  // as in grouped_gemm_tc.cu at these tile heights
      Seg sg;
      bool have = feed.first(sg);
      while (ok && have) {
        const int row0 = sg.e * a.rows_per_expert + sg.mb * kF8BlockM;
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 0, blockIdx.x, 0);
            break;
          }
          if (elect_one()) {
            mbar_arrive_expect_tx(&full_bar[st.stage], Cfg::kStageA);
            uint8_t* dst = sA + st.stage * Cfg::kStageA;
            tma_load_2d(dst, &tmap_w, &full_bar[st.stage], kb * 128, row0, policy);
            if (kGateUp) tma_load_2d(dst + kF8TileA, &tmap_w, &full_bar[st.stage], kb * 128, row0 + a.up_row_offset, policy);
          }
          __syncwarp();
          st.advance(STAGES);
          feed.advance();
        }
        if (ok) have = feed.next(sg);
      }
      if (feed.bad_tile && lane == 0) report_status(a.status, kBadArgument, 7, blockIdx.x, 0);
      if (!ok) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) __nanosleep(1000);
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- UMMA issuer (one K block per tmp stage)
      F8Pipe st, tmp;
      bool ok = true;
      Seg sg;
      while (ok && reader.next(sg, ok)) {
        uint32_t n_tile = (uint32_t)((sg.n_rows + 15) & ~15);
        if (n_tile < 16) n_tile = 16;
        const uint32_t idesc = umma_idesc(0, 0, kF8BlockM, n_tile);  // e4m3 x e4m3 -> fp32
        for (int j = 0; j < sg.nkb; ++j) {
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tmp_empty[tmp.stage], tmp.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmAccTimeout, 1, blockIdx.x, 0);
            break;
          }
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full_bar[st.stage], st.phase, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmFullTimeout, 1, blockIdx.x, 0);
            break;
          }
          tc_fence_after_sync();
          if (!b_tma) fence_proxy_async_smem();  // the gathered rows
          const uint32_t d0 = tmem_base + tmp.stage * Cfg::kTmpCols;
          const uint64_t a_desc = umma_desc_sw128(smem_u32(sA + st.stage * Cfg::kStageA));
          const uint64_t b_desc = umma_desc_sw128(smem_u32(sB + st.stage * Cfg::kStageB));
          if (kGateUp) umma_block<true>(d0, d0 + N_MAX, a_desc, a_desc + (kF8TileA >> 4), b_desc, idesc, 0u);
          else umma_block<true>(d0, a_desc, b_desc, idesc, 0u);
          umma_commit(&empty_bar[st.stage]);
          umma_commit(&tmp_full[tmp.stage]);
          st.advance(STAGES);
          tmp.advance(Cfg::kTmpStages);
        }
      }
    } else if (warp == 2 && b_tma) {
      // ---------------------------------------------------------------- token-operand producer (TMA)
      F8Pipe st;
      bool ok = true;
      Seg sg;
      int ready_tile = -1;
      while (ok && reader.next(sg, ok)) {
        if (a.tile_wait != nullptr && sg.tt != ready_tile) {
          ok = tile_ready(sg.tt);
          if (!ok) break;
          __syncwarp();
          fence_proxy_async_all();  // the TMA reads below, by whichever lane, come after the acquire
          ready_tile = sg.tt;
        }
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
            break;
          }
          if (elect_one()) {
            mbar_arrive_expect_tx(&full_bar[st.stage], Cfg::kStageB);
            tma_load_2d(sB + st.stage * Cfg::kStageB, &tmap_b, &full_bar[st.stage], kb * 128, sg.row_start);
          }
          __syncwarp();
          st.advance(STAGES);
        }
      }
      if (!ok) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) __nanosleep(1000);
      }
    } else if (warp == 2 && Cfg::kFourGather) {
    } else if (warp == 2) {
      // ---------------------------------------------------------------- token-operand producer (gathered e4m3 rows)
      const int r_in = lane >> 3, chunk = lane & 7;  // rows r_in, r_in + 4, ...: two swizzle phases
      const uint32_t sw_off[2] = {(uint32_t)((chunk ^ r_in) << 4), (uint32_t)((chunk ^ (r_in + 4)) << 4)};
      F8Pipe st;
      bool ok = true;
      Seg sg, nx;
      int ready_tile = -1;
      int idx[N_MAX / 4];  // source rows of the segment at hand, fetched during the previous one
      auto row_indices = [&](const Seg& s_) {
#pragma unroll
        for (int i = 0; i < N_MAX / 4; ++i) {
          const int n = r_in + 4 * i;
          if (n < s_.n_rows) idx[i] = a.b_index ? __ldcg(a.b_index + s_.row_start + n) : s_.row_start + n;
        }
      };
      bool have = reader.next(sg, ok), more = false;
      if (have) row_indices(sg);
      while (ok && have) {
        if (a.tile_wait != nullptr && sg.tt != ready_tile) {
          ok = tile_ready(sg.tt);
          if (!ok) break;
          ready_tile = sg.tt;
        }
        const int n_rows = sg.n_rows;
        int n_tile = (n_rows + 15) & ~15;
        if (n_tile < 16) n_tile = 16;
        const uint8_t* rp[N_MAX / 4];
#pragma unroll
        for (int i = 0; i < N_MAX / 4; ++i) {
          const int n = r_in + 4 * i;
          rp[i] = n < n_rows ? static_cast<const uint8_t*>(a.b_base) + (long long)idx[i] * a.b_pitch + chunk * 16 : nullptr;
        }
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
            break;
          }
          const uint32_t b_stage = smem_u32(sB + st.stage * Cfg::kStageB);
#pragma unroll
          for (int i = 0; i < N_MAX / 4; ++i) {
            const int n = r_in + 4 * i;
            if (n < n_tile) {
              const bool live = rp[i] != nullptr;
              cp_async_16(b_stage + n * 128 + sw_off[i & 1], live ? (const void*)(rp[i] + (long long)kb * 128) : a.b_base, live ? 16u : 0u);
            }
          }
          cp_async_mbar_arrive_noinc(&full_bar[st.stage]);
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
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 3) {
      // ---------------------------------------------------------------- scale tables (a unit ahead), finished tiles
      // Table: x scales [j][n] and weight scales [t][j] of a segment, j = kb - kb0.  A lane takes whole token rows: all of a
      // row's scales are requested before the first one is stored.
      // Finished tiles: two units behind, the outputs of a whole gate/up unit are fenced and counted for the down GEMM.
      const int row_blocks = a.rows_per_expert / kF8BlockM;
      const bool vec = (a.b_scale_pitch & 3) == 0 && (reinterpret_cast<uintptr_t>(a.b_scale) & 15) == 0;
      const bool report = kGateUp && a.tile_done != nullptr;
      bool ok = true;
      Seg sg;
      int n_it = 0, ready_tile = -1;
      int done_tile[2] = {-1, -1};  // tiles of the last two units, if this warp has to report them
      auto report_unit = [&](int k) -> bool {  // unit k of this CTA
        const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&epi_bar[k & 1], (uint32_t)(k >> 1) & 1u, abort_flag, wait_ns));
        const int tt = k & 1 ? done_tile[1] : done_tile[0];
        if (got && lane == 0 && tt >= 0) {
          __threadfence();  // the promotion warps' stores (ordered before by the barrier) are visible device-wide
          atomicAdd(a.tile_done + tt, PROMO_WARPS);
        }
        return got;
      };
      while (ok && reader.next(sg, ok)) {
        const int buf = n_it % kF8Tables;
        float* t = sTable + buf * Cfg::kTableFloats;
        float wv[kGateUp ? 2 : 1];
#pragma unroll
        for (int q = 0; q < (kGateUp ? 2 : 1); ++q) {
          const int rb = (q == 0 ? 0 : a.up_row_offset / kF8BlockM) + sg.mb;
          wv[q] = lane < sg.nkb ? __ldcg(a.w_scale + ((long long)sg.e * row_blocks + rb) * a.k_blocks + sg.kb0 + lane) : 0.f;
        }
        if (a.tile_wait != nullptr && sg.tt != ready_tile) {
          ok = tile_ready(sg.tt);
          if (!ok) break;
          ready_tile = sg.tt;
        }
        if (n_it >= kF8Tables) {
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tbl_free[buf], (uint32_t)(n_it / kF8Tables - 1) & 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmAccTimeout, 6, blockIdx.x, 0);
            break;
          }
        }
        int n_tile = (sg.n_rows + 15) & ~15;
        if (n_tile < 16) n_tile = 16;
        for (int n = lane; n < n_tile; n += 32) {
          const bool live = n < sg.n_rows;
          long long idx = 0;
          if (live) idx = a.b_index ? (long long)__ldcg(a.b_index + sg.row_start + n) : (long long)(sg.row_start + n);
          const float* src = a.b_scale + idx * a.b_scale_pitch + sg.kb0;
          float v[kF8MaxKb];
          if (vec && ((sg.kb0 | sg.nkb) & 3) == 0) {
#pragma unroll
            for (int j = 0; j < kF8MaxKb; j += 4) {
              float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
              if (live && j < sg.nkb) f = __ldcg(reinterpret_cast<const float4*>(src + j));
              v[j] = f.x;
              v[j + 1] = f.y;
              v[j + 2] = f.z;
              v[j + 3] = f.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < kF8MaxKb; ++j) v[j] = (live && j < sg.nkb) ? __ldcg(src + j) : 0.f;
          }
#pragma unroll
          for (int j = 0; j < kF8MaxKb; ++j)
            if (j < sg.nkb) t[j * N_MAX + n] = v[j];
        }
#pragma unroll
        for (int q = 0; q < (kGateUp ? 2 : 1); ++q) t[N_MAX * kF8MaxKb + q * kF8MaxKb + lane] = wv[q];
        if (report) {
          // before the table is handed over: with it the promotion warps may come back to the same barrier
          if (n_it >= 2) ok = report_unit(n_it - 2);
          if (!ok) break;
          const int tt = sg.nseg == 1 ? sg.tt : -1;
          if (n_it & 1) done_tile[1] = tt;
          else done_tile[0] = tt;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&tbl_bar[buf]);
        ++n_it;
      }
      if (report)
        for (int k = n_it < 2 ? 0 : n_it - 2; ok && k < n_it; ++k) ok = report_unit(k);
    }
  } else if (Cfg::kFourGather && warp >= 12) {
    if (Cfg::kFourGather) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    // ---------------------------------------------------------------- token-operand producers (gathered e4m3 rows, four warps)
    const int gt = tid - 384;  // rows gt / 8, + 16, ...; 16-byte chunk gt & 7
    const int r_in = gt >> 3, chunk = gt & 7;
    const uint32_t sw_off = (uint32_t)(r_in * 128 + ((chunk ^ (r_in & 7)) << 4));
    F8Pipe st;
    bool ok = true;
    Seg sg;
    int ready_tile = -1;
    while (ok && !b_tma && reader.next(sg, ok)) {
      if (a.tile_wait != nullptr && sg.tt != ready_tile) {
        ok = tile_ready(sg.tt);
        if (!ok) break;
        ready_tile = sg.tt;
      }
      int src_row[N_MAX / 16];  // rows behind the tile repeat its last one, and nobody looks at their sums
      if (sg.n_rows > 0) {  // (a tile without rows has no last one)
#pragma unroll
        for (int i = 0; i < N_MAX / 16; ++i) {
          const int n = sg.row_start + min(r_in + 16 * i, sg.n_rows - 1);
          src_row[i] = a.b_index ? __ldcg(a.b_index + n) : n;
        }
      }
      for (int j = 0; j < sg.nkb; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
          break;
        }
        const uint32_t dst = smem_u32(sB + st.stage * Cfg::kStageB) + sw_off;
        gather_chunks(dst, reinterpret_cast<uint64_t>(a.b_base) + (sg.kb0 + j) * 128 + chunk * 16, src_row, a.b_pitch, sg.n_rows);
        cp_async_mbar_arrive_noinc(&full_bar[st.stage]);
        st.advance(STAGES);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    if (Cfg::kFourGather) asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
    // ---------------------------------------------------------------- promotion + epilogue
    const int pw = warp - 4;                 // 0 .. PROMO_WARPS-1
    const int wq = pw & 3;                   // tensor-memory lane quarter
    const int grp = pw >> 2;                 // column group
    const int row = wq * 32 + lane;
    uint8_t* stage = sStage + pw * kF8Stage;
    F8Pipe tmp;
    bool ok = true;
    uint32_t grp_phase = 0;
    // The four warps of this column group meet (bounded, so not a named barrier).
    auto group_sync = [&]() -> bool {
      __syncwarp();
      if (lane == 0) mbar_arrive(&grp_bar[grp]);
      const bool k = __all_sync(0xffffffffu, mbar_wait_bounded(&grp_bar[grp], grp_phase, abort_flag, wait_ns));
      grp_phase ^= 1u;
      if (!k && lane == 0) report_status(a.status, kGemmAccTimeout, 7, blockIdx.x, 0);
      return k;
    };
    Seg sg;
    int n_it = 0;  // index of this CTA's segment
    bool skipped = false;
    while (ok && reader.next(sg, ok)) {
      const int mb = sg.mb, n_rows = sg.n_rows, row_start = sg.row_start;
      int n_tile = (n_rows + 15) & ~15;
      if (n_tile < 16) n_tile = 16;
      const int buf = n_it % kF8Tables;
      const bool alone = Cfg::kTurns && n_tile <= COLS;  // this group has the unit to itself, or nothing to do with it
      const uint32_t share = alone ? 2u : 1u;            // arrivals on accumulators and outputs: for both groups
      if (alone && grp != (n_it & 1)) {
        // The scale table is passed on by both groups all the same: tbl_free never completes a phase that one of them has not
        // looked at, so it is at most one phase ahead of anybody, and its parity says which.  (With the other group arriving for
        // both it got two ahead while this one was in its epilogue, where the next units' K blocks fit the accumulators.)  The
        // wait keeps the arrival out of the phase of the table's last unit.
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tbl_bar[buf], (uint32_t)(n_it / kF8Tables) & 1u, abort_flag, wait_ns));
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmAccTimeout, 4, blockIdx.x, 0);
          break;
        }
        if (lane == 0) mbar_arrive(&tbl_free[buf]);
        const int at = tmp.stage + sg.nkb;
        tmp.stage = at % Cfg::kTmpStages;
        tmp.phase ^= (uint32_t)(at / Cfg::kTmpStages) & 1u;
        skipped = true;
        ++n_it;
        continue;
      }
      if (Cfg::kTurns && skipped) {
        // The parities of the accumulators mean what they say only when the other group has read all of its unit.
        skipped = false;
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tbl_free[(n_it - 1) % kF8Tables], (uint32_t)((n_it - 1) / kF8Tables) & 1u,
                                                       abort_flag, wait_ns));
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmAccTimeout, 8, blockIdx.x, 0);
          break;
        }
      }
      const int col0 = alone ? 0 : grp * COLS;
      const uint32_t lane_base = tmem_base + ((uint32_t)(wq * 32) << 16) + col0;
      const float* tbl = sTable + buf * Cfg::kTableFloats;
      const float* tblW = tbl + N_MAX * kF8MaxKb;
      f32x2 acc_g[COLS / 2], acc_u[kGateUp ? COLS / 2 : 1];
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) acc_g[i] = 0ull;
      if (kGateUp) {
#pragma unroll
        for (int i = 0; i < COLS / 2; ++i) acc_u[i] = 0ull;
      }
      float row_scale[COLS / 32];  // routing weights of this group's columns, requested ahead of the K loop
      if (!kGateUp && a.row_scale != nullptr) {
#pragma unroll
        for (int i = 0; i < COLS / 32; ++i) {
          const int n = col0 + 32 * i + lane;
          row_scale[i] = n < n_rows ? __ldcg(a.row_scale + row_start + n) : 1.f;
        }
      }
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tbl_bar[buf], (uint32_t)(n_it / kF8Tables) & 1u, abort_flag, wait_ns));
      if (!ok) {
        if (lane == 0) report_status(a.status, kGemmAccTimeout, 4, blockIdx.x, 0);
        break;
      }

      // Down projection: two K blocks per trip (a K block is only 16 KB of weights there), gate/up: one.
      constexpr int kTrip = kGateUp ? 1 : 2;
      for (int j = 0; j < sg.nkb; j += kTrip) {
        const int nb = kTrip == 2 && j + 1 < sg.nkb ? 2 : 1;
        F8Pipe nxt = tmp;
        nxt.advance(Cfg::kTmpStages);
        ok = mbar_wait_warp(&tmp_full[tmp.stage], tmp.phase, abort_flag, wait_ns);
        if (ok && nb == 2) ok = mbar_wait_warp(&tmp_full[nxt.stage], nxt.phase, abort_flag, wait_ns);
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmAccTimeout, 3, blockIdx.x, 0);
          break;
        }
        tc_fence_after_sync();
        const uint32_t t0 = lane_base + tmp.stage * Cfg::kTmpCols, t1 = lane_base + nxt.stage * Cfg::kTmpCols;
        const f32x2 w0 = pack2(tblW[j], tblW[j]);
        const f32x2 w1 = kGateUp ? pack2(tblW[kF8MaxKb + j], tblW[kF8MaxKb + j])
                                 : (nb == 2 ? pack2(tblW[j + 1], tblW[j + 1]) : 0ull);
        const ulonglong2* x0 = reinterpret_cast<const ulonglong2*>(tbl + j * N_MAX + col0);
        const ulonglong2* x1 = reinterpret_cast<const ulonglong2*>(tbl + (j + 1) * N_MAX + col0);
        // 16 token columns at a time, as many as the tile has; first and second accumulator (gate and up, or two K
        // blocks) travel together.
#pragma unroll
        for (int c0 = 0; c0 < COLS; c0 += 16) {
          if (col0 + c0 < n_tile) {
            uint32_t p[16], q[16];
            tmem_ld_16(t0 + c0, p);
            if (kGateUp) tmem_ld_16(t0 + N_MAX + c0, q);
            else if (nb == 2) tmem_ld_16(t1 + c0, q);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const ulonglong2 xs = x0[c0 / 4 + i];
              f32x2* ag = acc_g + c0 / 2 + 2 * i;
              ag[0] = fma2(pack2(p[4 * i], p[4 * i + 1]), mul2(w0, xs.x), ag[0]);
              ag[1] = fma2(pack2(p[4 * i + 2], p[4 * i + 3]), mul2(w0, xs.y), ag[1]);
              if (kGateUp) {
                f32x2* au = acc_u + c0 / 2 + 2 * i;
                au[0] = fma2(pack2(q[4 * i], q[4 * i + 1]), mul2(w1, xs.x), au[0]);
                au[1] = fma2(pack2(q[4 * i + 2], q[4 * i + 3]), mul2(w1, xs.y), au[1]);
              }
            }
            if (!kGateUp && nb == 2) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const ulonglong2 xs = x1[c0 / 4 + i];
                f32x2* ag = acc_g + c0 / 2 + 2 * i;
                ag[0] = fma2(pack2(q[4 * i], q[4 * i + 1]), mul2(w1, xs.x), ag[0]);
                ag[1] = fma2(pack2(q[4 * i + 2], q[4 * i + 3]), mul2(w1, xs.y), ag[1]);
              }
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        mbar_arrive_warp(&tmp_empty[tmp.stage], share);
        if (nb == 2) mbar_arrive_warp(&tmp_empty[nxt.stage], share);
        tmp.advance(Cfg::kTmpStages);
        if (nb == 2) tmp.advance(Cfg::kTmpStages);
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(&tbl_free[buf]);  // this warp is done with the segment's table

      bool finish = true;
      if (sg.nseg > 1) {
        // The unit is cut along K: park the sums; the group that arrives last adds the segments in K order.
        float* mine = a.partial + (long long)slot_of(sg, sg.seg) * slot_floats;
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const int n = col0 + c;
          if (n < n_rows) {
            const float2 g = unpack2(acc_g[c / 2]);
            __stcg(&mine[(long long)n * kF8BlockM + row], c & 1 ? g.y : g.x);
            if (kGateUp) {
              const float2 u = unpack2(acc_u[c / 2]);
              __stcg(&mine[(long long)(slot_cols + n) * kF8BlockM + row], c & 1 ? u.y : u.x);
            }
          }
        }
        __threadfence();
        ok = group_sync();
        if (!ok) break;
        int* counter = a.counters + (long long)sg.unit * 4 * GROUPS + (alone ? 0 : grp);
        if (wq == 0 && lane == 0) grp_last[grp] = atomicAdd(counter, 1);
        ok = group_sync();
        if (!ok) break;
        finish = grp_last[grp] == sg.nseg - 1;
        if (finish) {
          __threadfence();
          if (wq == 0 && lane == 0) *counter = 0;
#pragma unroll
          for (int i = 0; i < COLS / 2; ++i) acc_g[i] = 0ull;
          if (kGateUp) {
#pragma unroll
            for (int i = 0; i < COLS / 2; ++i) acc_u[i] = 0ull;
          }
          const f32x2 one = pack2(1.f, 1.f);
          for (int s_ = 0; s_ < sg.nseg; ++s_) {
            const float* p = a.partial + (long long)slot_of(sg, s_) * slot_floats + row;
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16) {
              if (col0 + c0 < n_rows) {
                float v[16], w[kGateUp ? 16 : 1];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                  const int n = col0 + c0 + c;
                  v[c] = n < n_rows ? __ldcg(&p[(long long)n * kF8BlockM]) : 0.f;
                  if (kGateUp) w[c] = n < n_rows ? __ldcg(&p[(long long)(slot_cols + n) * kF8BlockM]) : 0.f;
                }
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                  acc_g[(c0 + c) / 2] = fma2(pack2(v[c], v[c + 1]), one, acc_g[(c0 + c) / 2]);
                  if (kGateUp) acc_u[(c0 + c) / 2] = fma2(pack2(w[c], w[c + 1]), one, acc_u[(c0 + c) / 2]);
                }
              }
            }
          }
        }
      }

      if (finish) {
        const bool quantise = kGateUp && a.q_out != nullptr;
        unsigned peak[COLS / 32];  // quantise: lane l keeps the maximum of columns l (and l + 32) over this warp's rows
        // values of 16 columns at a time; gate/up: after the activation
        auto values = [&](int c0, float (&v)[16]) {
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            float2 g = unpack2(acc_g[(c0 + c) / 2]);
            if (kGateUp) {
              float2 u = unpack2(acc_u[(c0 + c) / 2]);
              if (a.round_h) {
                g.x = bf16_round(g.x);
                g.y = bf16_round(g.y);
                u.x = bf16_round(u.x);
                u.y = bf16_round(u.y);
              }
              g.x = swiglu_clamped(g.x, u.x, a.limit);
              g.y = swiglu_clamped(g.y, u.y, a.limit);
            }
            v[c] = g.x;
            v[c + 1] = g.y;
          }
        };
        if (!quantise) {
          __nv_bfloat16* st = reinterpret_cast<__nv_bfloat16*>(stage);
          __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + (long long)row_start * a.out_pitch + (long long)mb * kF8BlockM +
                               wq * 32 + (lane & 3) * 8;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += 16) {
            if (col0 + c0 < n_rows) {
              float v[16];
              values(c0, v);
              if (!kGateUp && a.row_scale != nullptr) {
#pragma unroll
                for (int c = 0; c < 16; ++c) v[c] *= __shfl_sync(0xffffffffu, row_scale[c0 / 32], (c0 + c) & 31);
              }
              __syncwarp();
#pragma unroll
              for (int c = 0; c < 16; ++c) st[c * 32 + lane] = __float2bfloat16_rn(v[c]);
              __syncwarp();
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int n = col0 + c0 + 8 * h + (lane >> 2);
                const uint4 x = reinterpret_cast<const uint4*>(stage)[32 * h + lane];
                if (n < n_rows) *reinterpret_cast<uint4*>(out + (long long)n * a.out_pitch) = x;
              }
            }
          }
        } else {
          // 1. activations rounded to bf16 (what the quantiser is defined on), kept in the accumulators; column maxima
#pragma unroll
          for (int i = 0; i < COLS / 32; ++i) peak[i] = 0u;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += 16) {
            if (col0 + c0 < n_rows) {
              float v[16];
              values(c0, v);
#pragma unroll
              for (int c = 0; c < 16; ++c) {
                v[c] = bf16_round(v[c]);
                const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v[c])));
                if (lane == ((c0 + c) & 31)) peak[c0 / 32] = m;
              }
#pragma unroll
              for (int c = 0; c < 16; c += 2) acc_g[(c0 + c) / 2] = pack2(v[c], v[c + 1]);
            }
          }
          // 2. a token's group is the unit's 128 rows: maximum over the group's four warps, exchanged through the upper
          //    half of their staging buffers, which the e4m3 bytes below leave free
          auto maxima = [&](int q) { return reinterpret_cast<float*>(sStage + (grp * 4 + q) * kF8Stage + 512); };
#pragma unroll
          for (int i = 0; i < COLS / 32; ++i) maxima(wq)[32 * i + lane] = __uint_as_float(peak[i]);
          ok = group_sync();
          if (!ok) break;
          float inv[COLS / 32];
#pragma unroll
          for (int i = 0; i < COLS / 32; ++i) {
            const int at = 32 * i + lane;
            const float scale = group_scale(fmaxf(fmaxf(maxima(0)[at], maxima(1)[at]), fmaxf(maxima(2)[at], maxima(3)[at])));
            inv[i] = 1.f / scale;
            const int n = col0 + at;
            if (wq == 0 && n < n_rows) a.q_scale[(long long)(row_start + n) * a.q_scale_pitch + mb] = scale;
          }
          // A warp that runs ahead writes its next maxima a unit later; with more K blocks than accumulator stages
          // that unit needed the slowest warp's arrivals, otherwise they meet again here.
          if (sg.nseg > 1 || a.k_blocks <= 2 * Cfg::kTmpStages) {
            ok = group_sync();
            if (!ok) break;
          }
          // 3. e4m3 bytes, transposed through shared memory: 16 bytes per lane
          uint8_t* out = static_cast<uint8_t*>(a.q_out) + (long long)row_start * a.q_pitch + (long long)mb * kF8BlockM + wq * 32 +
                         (lane & 1) * 16;
#pragma unroll
          for (int c0 = 0; c0 < COLS; c0 += 16) {
            if (col0 + c0 < n_rows) {
              __syncwarp();
#pragma unroll
              for (int c = 0; c < 16; ++c) {
                const float2 v = unpack2(acc_g[(c0 + c) / 2]);
                stage[c * 32 + lane] = to_e4m3(c & 1 ? v.y : v.x, __shfl_sync(0xffffffffu, inv[c0 / 32], (c0 + c) & 31));
              }
              __syncwarp();
              const int n = col0 + c0 + (lane >> 1);
              const uint4 x = reinterpret_cast<const uint4*>(stage)[lane];
              if (n < n_rows) *reinterpret_cast<uint4*>(out + (long long)n * a.q_pitch) = x;
            }
          }
        }
        if (kGateUp && a.tile_done != nullptr && sg.nseg > 1) {  // only the group that finished a cut unit knows
          __threadfence();  // every lane's stores are visible device-wide before the count
          __syncwarp();
          if (lane == 0) atomicAdd(a.tile_done + sg.tt, (int)share);
        }
      }
      if (kGateUp && a.tile_done != nullptr) {  // warp 3 reports whole units
        __syncwarp();
        if (lane == 0) mbar_arrive(&epi_bar[n_it & 1], share);
      }
      ++n_it;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// -------------------------------------------------------------------------------------------------
// 1x128 activation quantisation: x[row, :] (bf16) -> q[row, :] (e4m3) and scales[row, g] = amax_g / 448.
// One CTA per output row; 16 threads share a 128-wide group.  Rows can be gathered (row_index), skipped
// when an int32 flag inside the source row is zero (valid_off >= 0: the received-row valid flag), and
// bounded by a device-side row count (n_rows_dev, e.g. the plan's entry count).
// -------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
quant_rows_kernel(const uint8_t* x, long long x_pitch, const int* row_index, int hidden, uint8_t* q, float* scales,
                  long long valid_off, const int* n_rows_dev) {
  // Inputs are produced by kernels that may still run while this one is resident (programmatic launch), so
  // they are read from L2 (ld.global.cg), never through the non-coherent read-only path.
  grid_dep_launch();
  grid_dep_wait_cta();
  const int r = blockIdx.x;
  if (n_rows_dev != nullptr && r >= __ldcg(n_rows_dev)) return;
  const long long src = row_index ? (long long)__ldcg(row_index + r) : (long long)r;
  const uint8_t* row = x + src * x_pitch;
  if (valid_off >= 0 && __ldcg(reinterpret_cast<const int*>(row + valid_off)) == 0) return;
  const int chunks = hidden / 8;
  const int groups = hidden / 128;
  // (chunks is a multiple of 16, so a group is either fully active or fully idle in the last sweep)
  for (int c = threadIdx.x; c < chunks; c += blockDim.x)
    quant_chunk(row, c, q + (long long)r * hidden, scales + (long long)r * groups);
}

template <bool kGateUp, int N_MAX>
static int launch_f8(const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  using Cfg = F8Cfg<kGateUp, N_MAX>;
  static bool configured[64] = {};  // per device: the attribute belongs to (function, device)
  auto kern = grouped_gemm_fp8_kernel<kGateUp, N_MAX>;
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess) return (int)de;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  CUtensorMap tm, tb;
  memcpy(&tm, tmap, sizeof(tm));
  memcpy(&tb, args->b_tmap ? args->b_tmap : tmap, sizeof(tb));
  return (int)launch_kernel(kern, dim3(grid), dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, true, tm, tb, *args);
}

// 128-row tiles (grouped_gemm_fp8_wide.cu)
int launch_fp8_wide(bool gate_up, const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream);

static int check_f8(const mf_gemm_args* a, int n_max, int grid) {
  if (!a || grid < 1) return -1;
  if (n_max != 32 && n_max != 64 && n_max != 128) return -2;
  if (a->b_tmap != nullptr && a->b_index != nullptr) return -6;  // TMA token tiles need contiguous rows
  if (n_max == 128 && (a->b_box_rows < 0 || (a->b_box_rows > 0 && (a->b_box_rows % 16 != 0 || n_max % a->b_box_rows != 0)))) return -9;
  if (a->m_blocks < 1 || a->k_blocks < 1 || a->k_blocks > kF8MaxKb) return -3;
  if ((a->b_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(a->b_base) & 15) != 0) return -4;
  if (!a->w_scale || !a->b_scale) return -5;
  if (a->q_out ? (!a->q_scale || (a->q_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(a->q_out) & 15) != 0)
               : (!a->out || (a->out_pitch & 7) != 0 || (reinterpret_cast<uintptr_t>(a->out) & 15) != 0))
    return -7;  // 16-byte stores
  return 0;
}

}  // namespace mf

extern "C" {

int mf_gemm_gate_up_fp8(const void* tmap, const mf_gemm_args* args, int n_max, int grid, mf_stream_t stream) {
  int c = mf::check_f8(args, n_max, grid);
  if (c) return c;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n_max == 32) return mf::launch_f8<true, 32>(tmap, args, grid, s);
  if (n_max == 64) return mf::launch_f8<true, 64>(tmap, args, grid, s);
  return mf::launch_fp8_wide(true, tmap, args, grid, s);
}

int mf_gemm_down_fp8(const void* tmap, const mf_gemm_args* args, int n_max, int grid, mf_stream_t stream) {
  int c = mf::check_f8(args, n_max, grid);
  if (c) return c;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n_max == 32) return mf::launch_f8<false, 32>(tmap, args, grid, s);
  if (n_max == 64) return mf::launch_f8<false, 64>(tmap, args, grid, s);
  return mf::launch_fp8_wide(false, tmap, args, grid, s);
}

int mf_quant_rows_1x128(const void* x, long long x_pitch, const int* row_index, int rows, int hidden, void* q,
                        float* scales, long long valid_off, const int* n_rows_dev, mf_stream_t stream) {
  if (rows == 0) return 0;
  if (hidden % 128 != 0 || (x_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return -1;
  return (int)mf::launch_kernel(mf::quant_rows_kernel, dim3(rows), dim3(256), 0, static_cast<cudaStream_t>(stream), true,
                                static_cast<const uint8_t*>(x), x_pitch, row_index, hidden, static_cast<uint8_t*>(q),
                                scales, valid_off, n_rows_dev);
}

}  // extern "C"

// Block-scaled FP8 (e4m3) grouped expert GEMMs for token tiles of up to 128 rows (prefill chunks).
//
// Same number format, plan, unit order and hand-over as grouped_gemm_fp8.cu, with the operands the other way round: the
// 128 token rows of a tile are the UMMA M dimension and 256 weight rows its N dimension (gate/up: 128 gate rows and the
// 128 up rows that belong to them; down: two adjacent blocks).  What that buys where a tile is full of rows:
//   * a token is a tensor-memory lane, so its activation scale is one register per K block and the weight scale is the
//     same for 128 columns: the promotion acc += (w_scale * x_scale) * tmp forms two products per lane and K block, and
//     every accumulator costs one multiply-add.  With the weight rows on the lanes each accumulator needed a product of
//     its own and its scales as broadcasts from shared memory;
//   * one instruction of 128 x 256 x 32 reads 12 KB of shared memory in the time in which two of 128 x 128 x 32 read 16;
//   * the epilogue's quantisation group (128 activations of a token) lies in two threads instead of 128.
// Promotion works on 16 columns at a time, the next load under way while one is multiplied; its eight warps (a lane
// quarter and half of the columns each) hold 128 sums and two loads in registers, which is why the other four warps
// hand registers over to them.  Single multiply-adds, not pairs: the same rate (128 a clock).  Kernels alone, 2000 tokens on 36
// experts, us, gate/up and down: 32 columns in pairs 309 / 173, 16 in pairs 320 / 153, 32 single 297 / 161, 16 single 297 / 156.
// With waits and arrivals that do not branch per lane (mbar_wait_warp): 291 / 157; the call of 2000 tokens, together with a faster
// dispatch, 595 / 589 in four alternating runs.  Registers spilled (bytes stored / loaded, before and with these waits): down by map 0 / 0 and 8 / 16, down gathered
// 28 / 44 and 72 / 84, gate/up by map 8 / 16 and 92 / 92, gate/up gathered 60 / 64 and 28 / 60.  The times do not follow the spills.
// 36 experts of 3 x 4096 x 1536, whole layer, against the 64-row kernel's form on 128-row tiles, forwards on three weight sets
// in turn, with the promotion in its first form (32 columns in pairs): 2000 tokens 917 / 581 us, 1000 tokens 524 / 353, 500 tokens
// 317 / 222.  What bounds it now: a promotion warp's own instructions per K block (loads, waits, multiply-adds), not the 48 KB that a
// block brings through L2: CTA pairs, which fetch 32, took 324 / 179 for the same bits.  Also slower: sixteen promotion warps 426 /
// 172, the columns in halves on accumulators of their own 349 / 329, the next block's loads under this one's sums 320.
//
// Warps: 0 weight TMA and segment hand-out, 1 UMMA, 2 token TMA (b_tmap: contiguous rows in boxes), 3 activation and weight
// scales (four K blocks at a time, up to 16 ahead) and finished token tiles, 4-11 promotion and epilogue, 12-15 gather
// (without b_tmap: rows by index or one after the other, 16 bytes per cp.async).  The layers gather for gate/up and use
// boxes for down.  Rows by index through the tensor copy engine (tile::gather4, 32 instructions per K block) took 66 cycles
// an instruction and bound the whole kernel.
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "fp8_pipe.cuh"
#include "moeflow_b200.h"
#include "quant.cuh"
#include "work_iter.cuh"

namespace mf {

constexpr int kFwRows = 128;                   // token rows of a tile
template <bool kGather>
constexpr int kFwThreads = kGather ? 512 : 384;
constexpr int kFwGather = 128;                 // gather threads
constexpr int kFwPromo = 8;                    // promotion warps: 4 .. 11
constexpr int kFwStageW = 2 * kF8TileA;        // 256 weight rows x one K block
constexpr int kFwStageX = kFwRows * 128;
constexpr int kFwStages = 3;                   // (four: 4 % slower)
constexpr int kFwTmp = 2;                      // tensor-memory accumulators of 256 columns
constexpr int kFwScaleSlots = 4;               // scales of four K blocks each
constexpr int kFwScaleFloats = 4 * kFwRows + 8;  // [4][128] activation scales, [2][4] weight scales
constexpr int kFwOutPitch = 80;                // 32 outputs of a row, padded: 16-byte accesses of 8 rows hit all banks
constexpr int kFwOutBytes = 32 * kFwOutPitch;
constexpr int kFwSmem = 1024 + kFwStages * (kFwStageW + kFwStageX) + kFwScaleSlots * kFwScaleFloats * 4 +
                        2 * 2 * kFwRows * 4 /*maxima*/ + kFwPromo * kFwOutBytes + 1024 /*segment ring, barriers*/;
static_assert(kFwSmem <= 227 * 1024, "shared memory");
// Registers: 384 threads are launched with 168 each (64512), 512 with 128 (65536); the promotion warps take what the
// others give up.  72 x 128 + 216 x 256 = 64512; 72 x 128 + 200 x 256 + 40 x 128 = 65536.
constexpr int kFwRegsFew = 72, kFwRegsGather = 40;
template <bool kGather>
constexpr int kFwRegsMany = kGather ? 200 : 216;

// Waits for the loads so far.  The loaded values pass through, so that nothing that uses them is moved ahead of the wait.
__device__ __forceinline__ void tmem_ld_wait_16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// Four partial sums, 16 bytes at a time or (scratch off the 16-byte grid) float by float.  A template, not a test of the address:
// with both forms in one kernel the K loop of the gate/up GEMM was 1.4 % slower, cut units or not.
template <bool kAligned>
__device__ __forceinline__ void park_4(float* p, float4 v) {
  if (kAligned) {
    __stcg(reinterpret_cast<float4*>(p), v);
  } else {
    __stcg(p, v.x);
    __stcg(p + 1, v.y);
    __stcg(p + 2, v.z);
    __stcg(p + 3, v.w);
  }
}
template <bool kAligned>
__device__ __forceinline__ float4 parked_4(const float* p) {
  if (kAligned) return __ldcg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
}

// acc[0..15] += s * p[0..15]
__device__ __forceinline__ void promote_16(float* acc, const uint32_t (&p)[16], float s) {
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = fmaf(__uint_as_float(p[i]), s, acc[i]);
}

template <bool kGateUp, bool kGather, bool kAligned>
__global__ void __launch_bounds__(kFwThreads<kGather>, 1)
grouped_gemm_fp8_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                             const mf_gemm_args a, const int blocks) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;                                // [kFwStages][kFwStageW]
  uint8_t* sX = sW + kFwStages * kFwStageW;          // [kFwStages][kFwStageX]
  uint8_t* sOut = sX + kFwStages * kFwStageX;        // [kFwPromo][kFwOutBytes]
  float* sScale = reinterpret_cast<float*>(sOut + kFwPromo * kFwOutBytes);  // [kFwScaleSlots][kFwScaleFloats]
  float* sMax = sScale + kFwScaleSlots * kFwScaleFloats;                    // [2 units][2 column halves][128 rows]
  SegRing* ring = reinterpret_cast<SegRing*>(sMax + 2 * 2 * kFwRows);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ring + 1);
  uint64_t* empty_bar = full_bar + kFwStages;
  uint64_t* tmp_full = empty_bar + kFwStages;
  uint64_t* tmp_empty = tmp_full + kFwTmp;
  uint64_t* sc_full = tmp_empty + kFwTmp;            // [kFwScaleSlots]
  uint64_t* sc_free = sc_full + kFwScaleSlots;
  uint64_t* pair_bar = sc_free + kFwScaleSlots;      // [4] the two warps of a lane quarter met (epilogue)
  uint64_t* epi_bar = pair_bar + 4;                  // [2] a unit's outputs are stored (all promotion warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(epi_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* pair_last = abort_flag + 1;          // [4] a cut unit's arrival count, for both warps of the quarter
  static_assert(sizeof(SegRing) + (2 * kFwStages + 2 * kFwTmp + 2 * kFwScaleSlots + 6) * 8 + 8 + 16 <= 1024, "barriers");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kFwStages; ++s) {
      mbar_init(&full_bar[s], kGather ? 1 + kFwGather : 2);  // weights, token rows
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < kFwTmp; ++s) {
      mbar_init(&tmp_full[s], 1);
      mbar_init(&tmp_empty[s], kFwPromo);
    }
    for (int s = 0; s < kFwScaleSlots; ++s) {
      mbar_init(&sc_full[s], 1);
      mbar_init(&sc_free[s], kFwPromo);
    }
    for (int s = 0; s < 4; ++s) mbar_init(&pair_bar[s], 2);
    for (int s = 0; s < 2; ++s) mbar_init(&epi_bar[s], kFwPromo);
    ring->init((kGather ? 2 + kFwGather / 32 : 3) + kFwPromo);  // UMMA, scale warp, token producers, promotion warps
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    if (!kGather) tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
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
  // As in the other grouped GEMMs: gate/up waits for the plan and only then lets the next kernel start, so the down
  // GEMM finds the plan complete; with tile-level hand-over nothing in it waits for the gate/up grid as a whole.
  if (kGateUp || a.tile_wait == nullptr) {
    grid_dep_wait_cta();
    grid_dep_launch();
  } else {
    grid_dep_launch();
  }

  const unsigned long long wait_ns = a.wait_ns;
  int slot_cols = __ldcg(a.plan + MF_PLAN_SLOT_COLS);
  if (slot_cols <= 0 || slot_cols > kFwRows) slot_cols = kFwRows;
  WorkIter work;
  {
    const int n_tiles = __ldcg(a.plan + MF_PLAN_N_TILES);
    const int cut = __ldcg(a.plan + a.split_word);  // 0 = stream-K, else the K split
    // Scratch in accumulators of one weight block, as much as the other tile heights need.  Stream-K on units of two blocks
    // would need twice that: where it is not there, fewer CTAs take part.
    const long long acc_floats = (long long)slot_cols * kF8BlockM, steps = (long long)n_tiles * blocks * a.k_blocks;
    long long need = cut == 0 ? 2 * min(steps, (long long)gridDim.x) : cut > 1 ? (long long)n_tiles * blocks * cut : 0;
    int ctas = gridDim.x;
    if (!kGateUp && cut == 0) {
      const long long there = a.partial_floats > 0 ? a.partial_floats / acc_floats : need;
      ctas = (int)max(1ll, min(there / 4, (long long)ctas));
    }
    work.init(a, kFwRows, n_tiles, cut, blockIdx.x, ctas);
    if (kGateUp) need = 2 * work.slots_needed();
    // the plan is checked against the buffers it indexes before anything is stored (same rule as the other kernels)
    bool bad = n_tiles < 0 || !(cut == 0 || cut == 1 || cut == 2 || cut == 4 || cut == 8) ||
               (cut > 1 && a.k_blocks % cut != 0);
    bad = bad || (a.max_tiles > 0 && n_tiles > a.max_tiles);
    bad = bad || (a.n_counters > 0 && (long long)n_tiles * a.m_blocks * 4 > (long long)a.n_counters);
    bad = bad || (a.partial_floats > 0 && need * acc_floats > a.partial_floats);
    if (bad) {
      if (tid == 0) report_status(a.status, kBadArgument, 6, blockIdx.x, 0);
      work.init(a, kFwRows, 0, 1, blockIdx.x, gridDim.x);
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
  // Weight blocks of a unit: gate and up, or two adjacent ones of the `blocks` (an odd count leaves one for the last unit).
  auto unit_row = [&](const Seg& s) { return kGateUp ? s.mb * kF8BlockM : s.mb * 2 * kF8BlockM; };
  auto two_halves = [&](const Seg& s) { return kGateUp || s.mb * 2 + 1 < blocks; };
  const int second_half = kGateUp ? a.up_row_offset : kF8BlockM;
  SegReader reader(ring, abort_flag, wait_ns);

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFwRegsFew));
    if (warp == 0) {
      // -------------------------------------------------------------- weight TMA producer, hands out the segments
      F8Pipe st;
      bool ok = true;
      SegFeed feed(work, ring, abort_flag, wait_ns);
      Seg sg;
      bool have = feed.first(sg);
      while (ok && have) {
        const int row0 = sg.e * a.rows_per_expert + unit_row(sg);
        const bool two = two_halves(sg);
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 0, blockIdx.x, 0);
            break;
          }
          if (elect_one()) {
            mbar_arrive_expect_tx(&full_bar[st.stage], two ? 2 * kF8TileA : kF8TileA);
            uint8_t* dst = sW + st.stage * kFwStageW;
            tma_load_2d(dst, &tmap_w, &full_bar[st.stage], kb * 128, row0);
            if (two) tma_load_2d(dst + kF8TileA, &tmap_w, &full_bar[st.stage], kb * 128, row0 + second_half);
          }
          __syncwarp();
          st.advance(kFwStages);
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
      // -------------------------------------------------------------- UMMA issuer (one K block per tmp stage)
      F8Pipe st, tmp;
      bool ok = true;
      Seg sg;
      while (ok && reader.next(sg, ok)) {
        const uint32_t idesc = umma_idesc(0, 0, kFwRows, two_halves(sg) ? 256 : 128);  // e4m3 x e4m3 -> fp32
        for (int j = 0; j < sg.nkb; ++j) {
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full_bar[st.stage], st.phase, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmFullTimeout, 1, blockIdx.x, 0);
            break;
          }
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tmp_empty[tmp.stage], tmp.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmAccTimeout, 1, blockIdx.x, 0);
            break;
          }
          tc_fence_after_sync();
          if (kGather) fence_proxy_async_smem();  // the gathered rows
          umma_block<true>(tmem_base + tmp.stage * 256, umma_desc_sw128(smem_u32(sX + st.stage * kFwStageX)),
                           umma_desc_sw128(smem_u32(sW + st.stage * kFwStageW)), idesc, 0u);
          umma_commit(&empty_bar[st.stage]);
          umma_commit(&tmp_full[tmp.stage]);
          st.advance(kFwStages);
          tmp.advance(kFwTmp);
        }
      }
    } else if (warp == 2) {
      // -------------------------------------------------------------- token rows in boxes
      F8Pipe st;
      bool ok = true;
      Seg sg;
      int ready_tile = -1;
      const int box_rows = a.b_box_rows > 0 ? a.b_box_rows : kFwRows;
      while (!kGather && ok && reader.next(sg, ok)) {
        if (a.tile_wait != nullptr && sg.tt != ready_tile) {
          ok = tile_ready(sg.tt);
          if (!ok) break;
          __syncwarp();
          fence_proxy_async_all();  // the TMA reads below, by whichever lane, come after the acquire
          ready_tile = sg.tt;
        }
        const int n_box = (sg.n_rows + box_rows - 1) / box_rows;
        for (int j = 0; j < sg.nkb; ++j) {
          const int kb = sg.kb0 + j;
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty_bar[st.stage], st.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmEmptyTimeout, 2, blockIdx.x, 0);
            break;
          }
          if (elect_one()) {
            // rows behind the tile (the next one's, or zero fill) end up in accumulator rows that are not looked at
            uint8_t* dst = sX + st.stage * kFwStageX;
            mbar_arrive_expect_tx(&full_bar[st.stage], n_box * box_rows * 128);
            for (int i = 0; i < n_box; ++i)
              tma_load_2d(dst + i * box_rows * 128, &tmap_x, &full_bar[st.stage], kb * 128, sg.row_start + i * box_rows);
          }
          __syncwarp();
          st.advance(kFwStages);
        }
      }
      if (!ok) {
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 100000ull) __nanosleep(1000);
      }
    } else {
      // -------------------------------------------------------------- scales (four K blocks at a time), finished tiles
      const int row_blocks = a.rows_per_expert / kF8BlockM;
      const bool vec = (a.b_scale_pitch & 3) == 0 && (reinterpret_cast<uintptr_t>(a.b_scale) & 15) == 0;
      const bool report = kGateUp && a.tile_done != nullptr;
      bool ok = true;
      Seg sg;
      F8Pipe sc;
      int n_it = 0, ready_tile = -1;
      int done_tile[2] = {-1, -1};  // tiles of the last two units, if this warp has to report them
      auto report_unit = [&](int k) -> bool {  // unit k of this CTA
        const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&epi_bar[k & 1], (uint32_t)(k >> 1) & 1u, abort_flag, wait_ns));
        const int tt = k & 1 ? done_tile[1] : done_tile[0];
        if (got && lane == 0 && tt >= 0) {
          __threadfence();  // the promotion warps' stores (ordered before by the barrier) are visible device-wide
          atomicAdd(a.tile_done + tt, kFwPromo);
        }
        return got;
      };
      while (ok && reader.next(sg, ok)) {
        if (a.tile_wait != nullptr && sg.tt != ready_tile) {
          ok = tile_ready(sg.tt);
          if (!ok) break;
          ready_tile = sg.tt;
        }
        const float* src[4];  // this lane's rows: lane, lane + 32, ...
        if (sg.n_rows > 0) {  // (a tile without rows has no last one)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int n = sg.row_start + min(lane + 32 * i, sg.n_rows - 1);
            src[i] = a.b_scale + (a.b_index ? (long long)__ldcg(a.b_index + n) : (long long)n) * a.b_scale_pitch + sg.kb0;
          }
        }
        const float* wsrc = nullptr;  // lanes 0-3: the first block's scales, 4-7: the second's
        if (lane < 4 || (lane < 8 && two_halves(sg)))
          wsrc = a.w_scale + ((long long)sg.e * row_blocks + (unit_row(sg) + (lane >> 2) * second_half) / kF8BlockM) * a.k_blocks + sg.kb0;
        if (report) {
          // before any scale of this unit is handed over: with them the promotion warps may come back to the same barrier
          if (n_it >= 2) ok = report_unit(n_it - 2);
          if (!ok) break;
          const int tt = sg.nseg == 1 ? sg.tt : -1;
          if (n_it & 1) done_tile[1] = tt;
          else done_tile[0] = tt;
        }
        for (int j0 = 0; j0 < sg.nkb; j0 += 4) {
          float v[4][4], w = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (32 * i < sg.n_rows) {
              if (vec && (sg.kb0 & 3) == 0 && j0 + 4 <= sg.nkb) {
                const float4 f = __ldcg(reinterpret_cast<const float4*>(src[i] + j0));
                v[i][0] = f.x;
                v[i][1] = f.y;
                v[i][2] = f.z;
                v[i][3] = f.w;
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[i][k] = j0 + k < sg.nkb ? __ldcg(src[i] + j0 + k) : 0.f;
              }
            }
          }
          if (wsrc != nullptr && j0 + (lane & 3) < sg.nkb) w = __ldcg(wsrc + j0 + (lane & 3));
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&sc_free[sc.stage], sc.phase ^ 1u, abort_flag, wait_ns));
          if (!ok) {
            if (lane == 0) report_status(a.status, kGemmAccTimeout, 6, blockIdx.x, 0);
            break;
          }
          float* t = sScale + sc.stage * kFwScaleFloats;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (32 * i < sg.n_rows) {
#pragma unroll
              for (int k = 0; k < 4; ++k) t[k * kFwRows + lane + 32 * i] = v[i][k];
            }
          }
          if (lane < 8) t[4 * kFwRows + lane] = w;
          __syncwarp();
          if (lane == 0) mbar_arrive(&sc_full[sc.stage]);
          sc.advance(kFwScaleSlots);
        }
        ++n_it;
      }
      if (report)
        for (int k = n_it < 2 ? 0 : n_it - 2; ok && k < n_it; ++k) ok = report_unit(k);
    }
  } else if (kGather && warp >= 4 + kFwPromo) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFwRegsGather));
    // ---------------------------------------------------------------- token rows, 16 bytes at a time
    const int gt = tid - 32 * (4 + kFwPromo);  // 0 .. 127: rows gt / 8, + 16, ...; 16-byte chunk gt & 7
    const int r_in = gt >> 3, chunk = gt & 7;
    const uint32_t sw_off = (uint32_t)(r_in * 128 + ((chunk ^ (r_in & 7)) << 4));
    F8Pipe st;
    bool ok = true;
    Seg sg;
    int ready_tile = -1;
    while (ok && reader.next(sg, ok)) {
      if (!kGateUp && a.tile_wait != nullptr && sg.tt != ready_tile) {
        ok = tile_ready(sg.tt);
        if (!ok) break;
        ready_tile = sg.tt;
      }
      int src_row[kFwRows / 16];  // (rows behind the tile repeat its last one; nobody looks at them)
      if (sg.n_rows > 0) {  // (a tile without rows has no last one)
#pragma unroll
        for (int i = 0; i < kFwRows / 16; ++i) {
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
        const uint32_t dst = smem_u32(sX + st.stage * kFwStageX) + sw_off;
        gather_chunks(dst, reinterpret_cast<uint64_t>(a.b_base) + (sg.kb0 + j) * 128 + chunk * 16, src_row, a.b_pitch, sg.n_rows);
        cp_async_mbar_arrive_noinc(&full_bar[st.stage]);
        st.advance(kFwStages);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFwRegsMany<kGather>));
    // ---------------------------------------------------------------- promotion + epilogue
    const int wq = warp & 3;           // tensor-memory lane quarter: token rows 32 wq ..
    const int grp = (warp - 4) >> 2;   // columns 64 grp .. of both halves
    const int row = wq * 32 + lane;    // token row inside the tile
    const uint32_t lane_base = tmem_base + ((uint32_t)(wq * 32) << 16) + 64 * grp;
    uint8_t* stage = sOut + (warp - 4) * kFwOutBytes;
    F8Pipe tmp, sc;
    bool ok = true;
    uint32_t pair_phase = 0;
    // The two warps of this lane quarter meet (bounded, so not a named barrier).
    auto pair_sync = [&]() -> bool {
      __syncwarp();
      if (lane == 0) mbar_arrive(&pair_bar[wq]);
      const bool k = __all_sync(0xffffffffu, mbar_wait_bounded(&pair_bar[wq], pair_phase, abort_flag, wait_ns));
      pair_phase ^= 1u;
      if (!k && lane == 0) report_status(a.status, kGemmAccTimeout, 7, blockIdx.x, 0);
      return k;
    };
    Seg sg;
    int n_it = 0;  // index of this CTA's segment
    while (ok && reader.next(sg, ok)) {
      const int n_rows = sg.n_rows, row_start = sg.row_start;
      const bool live = wq * 32 < n_rows;  // warp-uniform: this quarter holds rows
      const bool two = two_halves(sg);
      float acc0[64], acc1[64];  // 64 columns of each half (gate and up, or the two blocks)
#pragma unroll
      for (int i = 0; i < 64; ++i) acc0[i] = acc1[i] = 0.f;
      float row_scale = 1.f;  // routing weight of this lane's row, requested ahead of the K loop
      if (!kGateUp && a.row_scale != nullptr && row < n_rows) row_scale = __ldcg(a.row_scale + row_start + row);

      for (int j = 0; j < sg.nkb; ++j) {
        const int sub = j & 3;
        if (sub == 0) ok = mbar_wait_warp(&sc_full[sc.stage], sc.phase, abort_flag, wait_ns);
        if (ok) ok = mbar_wait_warp(&tmp_full[tmp.stage], tmp.phase, abort_flag, wait_ns);
        if (!ok) {
          if (lane == 0) report_status(a.status, kGemmAccTimeout, 3, blockIdx.x, 0);
          break;
        }
        tc_fence_after_sync();
        if (live) {
          const float* t = sScale + sc.stage * kFwScaleFloats;
          const uint32_t d = lane_base + tmp.stage * 256;
          const float xs = t[sub * kFwRows + row];
          const float s0 = t[4 * kFwRows + sub] * xs, s1 = t[4 * kFwRows + 4 + sub] * xs;
          uint32_t p[16], q[16];
          auto release = [&]() {  // everything is in registers
            tc_fence_before_sync();
            __syncwarp();
            mbar_arrive_warp(&tmp_empty[tmp.stage]);
          };
          tmem_ld_16(d, p);
          tmem_ld_wait_16(p);
          if (two) {
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
              tmem_ld_16(d + 128 + c, q);
              promote_16(acc0 + c, p, s0);
              tmem_ld_wait_16(q);
              if (c < 48) tmem_ld_16(d + c + 16, p);
              else release();
              promote_16(acc1 + c, q, s1);
              if (c < 48) tmem_ld_wait_16(p);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
              tmem_ld_16(d + c + 16, q);
              promote_16(acc0 + c, p, s0);
              tmem_ld_wait_16(q);
              if (c < 32) tmem_ld_16(d + c + 32, p);
              else release();
              promote_16(acc0 + c + 16, q, s0);
              if (c < 32) tmem_ld_wait_16(p);
            }
          }
        } else {
          tc_fence_before_sync();
          __syncwarp();
          mbar_arrive_warp(&tmp_empty[tmp.stage]);
        }
        tmp.advance(kFwTmp);
        if (sub == 3 || j == sg.nkb - 1) {
          __syncwarp();
          mbar_arrive_warp(&sc_free[sc.stage]);
          sc.advance(kFwScaleSlots);
        }
      }
      if (!ok) break;

      // The unit is cut along K: park the sums, [block][column / 4][row][4]; the quarter that arrives last adds the segments
      // in K order, straight into its outputs (sum_16).  Summed up in the registers of the K loop instead, these few lines
      // made the compiler spill in that loop (layer at 2000 tokens: 8 % slower).
      const bool cut_unit = sg.nseg > 1;
      bool finish = true;
      const int half = kF8BlockM * slot_cols;
      auto slot_at = [&](int s_) {  // (a last unit of one block leaves no gap behind a segment of a K split)
        const long long acc = kGateUp || sg.c_first >= 0 ? 2ll * slot_of(sg, s_)
                                                         : (long long)(sg.tt * blocks + 2 * sg.mb) * sg.nseg + (two ? 2 : 1) * s_;
        return a.partial + ((acc * 32 + 16 * grp) * slot_cols + row) * 4;
      };
      if (cut_unit) {
        if (row < n_rows) {
          float* p = slot_at(sg.seg);
#pragma unroll
          for (int i = 0; i < 16; ++i, p += 4 * slot_cols) {
            park_4<kAligned>(p, make_float4(acc0[4 * i], acc0[4 * i + 1], acc0[4 * i + 2], acc0[4 * i + 3]));
            if (two) park_4<kAligned>(p + half, make_float4(acc1[4 * i], acc1[4 * i + 1], acc1[4 * i + 2], acc1[4 * i + 3]));
          }
        }
        __threadfence();
        ok = pair_sync();
        if (!ok) break;
        int* counter = a.counters + (long long)sg.unit * 4 + wq;
        if (grp == 0 && lane == 0) pair_last[wq] = atomicAdd(counter, 1);
        ok = pair_sync();
        if (!ok) break;
        finish = pair_last[wq] == sg.nseg - 1;
        if (finish) {
          __threadfence();
          if (grp == 0 && lane == 0) *counter = 0;
        }
      }
      // Columns 16 c .. of this warp's share of half h over all segments (finish only, cut units).
      auto sum_16 = [&](int h, int c, float (&v)[16]) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
#pragma unroll 1
        for (int s_ = 0; s_ < sg.nseg; ++s_) {
          const float* p = slot_at(s_) + h * half + 16 * c * slot_cols;
          float4 x[4];
#pragma unroll
          for (int i = 0; i < 4; ++i, p += 4 * slot_cols) x[i] = row < n_rows ? parked_4<kAligned>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[4 * i] += x[i].x;
            v[4 * i + 1] += x[i].y;
            v[4 * i + 2] += x[i].z;
            v[4 * i + 3] += x[i].w;
          }
        }
      };

      if (finish) {
        auto pack_bf16 = [](float x, float y) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
          return *reinterpret_cast<const uint32_t*>(&h);
        };
        // 32 outputs (bf16 pairs) of every row of this quarter, 16 bytes per lane and four lanes per row
        auto store_32 = [&](const uint32_t* o, int col) {
          __syncwarp();  // the previous block's reads are done
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(stage + lane * kFwOutPitch + 16 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
          __syncwarp();
          __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + col + (lane & 3) * 8;
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int r = 8 * h + (lane >> 2);
            const uint4 x = *reinterpret_cast<const uint4*>(stage + r * kFwOutPitch + (lane & 3) * 16);
            if (wq * 32 + r < n_rows) *reinterpret_cast<uint4*>(out + (long long)(row_start + wq * 32 + r) * a.out_pitch) = x;
          }
        };
        if (kGateUp) {
          uint32_t act[32];  // bf16 pairs: this lane's 64 activations
          auto activate = [&](float2 g, float2 u) {
            if (a.round_h) {
              g.x = bf16_round(g.x);
              g.y = bf16_round(g.y);
              u.x = bf16_round(u.x);
              u.y = bf16_round(u.y);
            }
            return pack_bf16(swiglu_clamped(g.x, u.x, a.limit), swiglu_clamped(g.y, u.y, a.limit));
          };
#pragma unroll
          for (int i = 0; i < 32; ++i) act[i] = 0u;
          if (live && !cut_unit) {
#pragma unroll
            for (int i = 0; i < 32; ++i) act[i] = activate(make_float2(acc0[2 * i], acc0[2 * i + 1]), make_float2(acc1[2 * i], acc1[2 * i + 1]));
          } else if (live) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              float g[16], u[16];
              sum_16(0, c, g);
              sum_16(1, c, u);
#pragma unroll
              for (int i = 0; i < 8; ++i)
                act[8 * c + i] = activate(make_float2(g[2 * i], g[2 * i + 1]), make_float2(u[2 * i], u[2 * i + 1]));
            }
          }
          if (a.q_out == nullptr) {
            if (live) {
              store_32(act, sg.mb * kF8BlockM + 64 * grp);
              store_32(act + 16, sg.mb * kF8BlockM + 64 * grp + 32);
            }
          } else {
            // The quantiser is defined on the bf16 activations; a group is the unit's 128 columns of one row, half of
            // them in this lane and half in the same lane of the quarter's other warp.  The maxima of two units in a row
            // lie in different words, so a warp that runs ahead does not touch what the other one still reads.
            float* maxima = sMax + (n_it & 1) * 2 * kFwRows;
            auto value = [&](int i) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&act[i])); };
            float peak = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) peak = fmaxf(peak, fmaxf(fabsf(value(i).x), fabsf(value(i).y)));
            maxima[grp * kFwRows + row] = peak;
            ok = pair_sync();
            if (!ok) break;
            const float scale = group_scale(fmaxf(peak, maxima[(grp ^ 1) * kFwRows + row]));
            const float inv = 1.f / scale;
            if (row < n_rows) {
              if (grp == 0) a.q_scale[(long long)(row_start + row) * a.q_scale_pitch + sg.mb] = scale;
              uint4* out = reinterpret_cast<uint4*>(static_cast<uint8_t*>(a.q_out) + (long long)(row_start + row) * a.q_pitch +
                                                    (long long)sg.mb * kF8BlockM + 64 * grp);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint32_t o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  o[k] = (uint32_t)to_e4m3x2(value(8 * i + 2 * k), inv) | ((uint32_t)to_e4m3x2(value(8 * i + 2 * k + 1), inv) << 16);
                out[i] = make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
          }
        } else if (live) {
          const int col = sg.mb * 2 * kF8BlockM + 64 * grp;
          if (!cut_unit) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // 32 columns of the first half, twice, then of the second
              if (q < 2 || two) {
                uint32_t o[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const float* f = (q < 2 ? acc0 : acc1) + 32 * (q & 1) + 2 * i;
                  o[i] = pack_bf16(f[0] * row_scale, f[1] * row_scale);
                }
                store_32(o, col + (q >> 1) * kF8BlockM + (q & 1) * 32);
              }
            }
          } else {
#pragma unroll 1
            for (int q = 0; q < (two ? 8 : 4); ++q) {  // 16 columns, 32 bytes per lane
              float v[16];
              sum_16(q >> 2, q & 3, v);
              uint32_t o[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = pack_bf16(v[2 * i] * row_scale, v[2 * i + 1] * row_scale);
              if (row < n_rows) {
                uint4* out = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + (long long)(row_start + row) * a.out_pitch + col +
                                                      (q >> 2) * kF8BlockM + (q & 3) * 16);
                out[0] = make_uint4(o[0], o[1], o[2], o[3]);
                out[1] = make_uint4(o[4], o[5], o[6], o[7]);
              }
            }
          }
        }
        if (kGateUp && a.tile_done != nullptr && sg.nseg > 1) {  // only the quarter that finished a cut unit knows
          __threadfence();  // every lane's stores are visible device-wide before the count
          __syncwarp();
          if (lane == 0) atomicAdd(a.tile_done + sg.tt, 1);
        }
      }
      if (kGateUp && a.tile_done != nullptr) {  // warp 3 reports whole units
        __syncwarp();
        if (lane == 0) mbar_arrive(&epi_bar[n_it & 1]);
      }
      ++n_it;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <bool kGateUp, bool kGather, bool kAligned>
static int launch_wide(const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  static bool configured[64] = {};  // per device: the attribute belongs to (function, device)
  auto kern = grouped_gemm_fp8_wide_kernel<kGateUp, kGather, kAligned>;
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess) return (int)de;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwSmem);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  mf_gemm_args a = *args;
  const int blocks = a.m_blocks;
  if (!kGateUp) a.m_blocks = (blocks + 1) / 2;  // a unit covers two weight blocks
  CUtensorMap tm, tx;
  memcpy(&tm, tmap, sizeof(tm));
  memcpy(&tx, kGather ? tmap : a.b_tmap, sizeof(tx));
  return (int)launch_kernel(kern, dim3(grid), dim3(kFwThreads<kGather>), kFwSmem, stream, true, tm, tx, a, blocks);
}

template <bool kGateUp, bool kGather>
static int launch_wide(const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  return (reinterpret_cast<uintptr_t>(args->partial) & 15) == 0 ? launch_wide<kGateUp, kGather, true>(tmap, args, grid, stream)
                                                                : launch_wide<kGateUp, kGather, false>(tmap, args, grid, stream);
}

int launch_fp8_wide(bool gate_up, const void* tmap, const mf_gemm_args* args, int grid, cudaStream_t stream) {
  if (args->b_tmap == nullptr)
    return gate_up ? launch_wide<true, true>(tmap, args, grid, stream) : launch_wide<false, true>(tmap, args, grid, stream);
  return gate_up ? launch_wide<true, false>(tmap, args, grid, stream) : launch_wide<false, false>(tmap, args, grid, stream);
}

}  // namespace mf

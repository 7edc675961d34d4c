// Dense projections of a decode step: out[t, r] = x[t, :] . W[r, :] for up to 64 tokens per tile (sm_100a).
//
// A projection of a decode step streams tens of MB of weights past a handful of tokens: it is bound by the weight
// stream, and at these sizes (25 MB = 4 us) as much by everything around it.  One weight block (128 rows, the UMMA
// M dimension; tokens are N) is far too few units for 148 SMs, so K is cut; the pieces of a block form a thread-block
// cluster and are added through distributed shared memory in K order: no global scratch, no counters, no waiting
// between CTAs that the hardware has not scheduled together, and the same sum on every run.
//   * every CTA of the cluster parks its fp32 partial tile in its own shared memory (the pipeline stages, free by
//     then), one cluster barrier, then CTA s finishes the token columns s, s + S, ... for all 128 rows;
//   * 4 stages of 24 KB: two CTAs fit an SM, so the next projection of the chain (programmatic launch) is resident
//     and has its first weight tiles in flight while this one drains.  The weights do not depend on the
//     predecessor; only the token tiles wait for it.
// Before this kernel these projections ran on the grouped GEMM with its K steps laid over all SMs: a block cut into 13
// pieces was finished by one CTA, eight columns per L2 round trip.  Shared expert (25 + 12.6 MB) at 64 tokens:
// 118 us there.
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "moeflow_b200.h"

namespace mf {

constexpr int kSkM = 128;         // weight rows per block (gate/up: 64 gate rows and their 64 up rows)
constexpr int kSkN = 64;          // token columns per tile
constexpr int kSkTileA = 128 * 128;
constexpr int kSkTileB = kSkN * 128;
constexpr int kSkStage = kSkTileA + kSkTileB;
constexpr int kSkStages = 4;
constexpr int kSkThreads = 192;   // warp 0 TMA, warp 1 UMMA, warps 2-5 tensor memory -> shared memory; all finish
constexpr int kSkSmem = kSkStages * kSkStage + 1024 + 256;
static_assert(kSkN * kSkM * 4 <= kSkStages * kSkStage, "the partial tile is parked in the pipeline stages");

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float ldcg_bf16(const void* base, long long i) {
  return __bfloat162float(__ushort_as_bfloat16(__ldcg(static_cast<const unsigned short*>(base) + i)));
}

template <bool kGateUp>
__global__ void __launch_bounds__(kSkThreads)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const mf_skinny_args a, int S) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kSkStages * kSkStage);  // [kSkStages]
  uint64_t* empty_bar = full_bar + kSkStages;
  uint64_t* acc_bar = empty_bar + kSkStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s = S > 1 ? (int)cluster_rank() : 0;
  const int unit = blockIdx.x / S;
  const int t0 = blockIdx.y * kSkN;
  const int n_rows = min(a.T - t0, kSkN);
  const int n_tile = (n_rows + 15) & ~15;
  const int kb0 = (int)((long long)s * a.k_blocks / S), kb1 = (int)((long long)(s + 1) * a.k_blocks / S);
  const int nkb = kb1 - kb0;

  if (tid == 0) {
    for (int i = 0; i < kSkStages; ++i) {
      mbar_init(&full_bar[i], 2);   // weight bytes, token bytes
      mbar_init(&empty_bar[i], 1);  // tcgen05.commit
    }
    mbar_init(acc_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kSkN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t policy = l2_evict_first();
      auto load_w = [&](int stage, int kb) {
        mbar_arrive_expect_tx(&full_bar[stage], kSkTileA);
        uint8_t* dst = smem + stage * kSkStage;
        if (kGateUp) {  // two boxes of 64 rows: one accumulator holds gate and up of the same 64 outputs
          tma_load_2d(dst, &tmap_w, &full_bar[stage], kb * 64, unit * 64, policy);
          tma_load_2d(dst + kSkTileA / 2, &tmap_w, &full_bar[stage], kb * 64, unit * 64 + a.up_row_offset, policy);
        } else {
          tma_load_2d(dst, &tmap_w, &full_bar[stage], kb * 64, unit * kSkM, policy);
        }
      };
      auto load_x = [&](int stage, int kb) {
        mbar_arrive_expect_tx(&full_bar[stage], kSkTileB);
        tma_load_2d(smem + stage * kSkStage + kSkTileA, &tmap_x, &full_bar[stage], kb * 64, t0);
      };
      const int first = min(nkb, kSkStages);
      for (int j = 0; j < first; ++j) load_w(j, kb0 + j);
      grid_dep_wait();  // the tokens are the predecessor's output
      for (int j = 0; j < first; ++j) load_x(j, kb0 + j);
      bool ok = true;
      for (int j = first; j < nkb && ok; ++j) {
        const int stage = j % kSkStages;
        ok = mbar_wait_bounded(&empty_bar[stage], (uint32_t)(j / kSkStages + 1) & 1u, abort_flag, a.wait_ns);
        if (!ok) {
          report_status(a.status, kGemmEmptyTimeout, 8, blockIdx.x, 0);
          break;
        }
        load_w(stage, kb0 + j);
        load_x(stage, kb0 + j);
      }
      if (!ok) {  // let copies in flight land before the CTA goes away
        const unsigned long long w0 = global_timer_ns();
        while (global_timer_ns() - w0 < 100000ull) __nanosleep(1000);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc(1, 1, kSkM, (uint32_t)n_tile);
    bool ok = true;
    for (int j = 0; j < nkb; ++j) {
      const int stage = j % kSkStages;
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full_bar[stage], (uint32_t)(j / kSkStages) & 1u, abort_flag, a.wait_ns));
      if (!ok) {
        if (lane == 0) report_status(a.status, kGemmFullTimeout, 8, blockIdx.x, 0);
        break;
      }
      tc_fence_after_sync();
      const uint32_t a_addr = smem_u32(smem + stage * kSkStage);
      umma_block<false>(tmem_base, umma_desc_sw128(a_addr), umma_desc_sw128(a_addr + kSkTileA), idesc, j > 0 ? 1u : 0u);
      umma_commit(&empty_bar[stage]);
    }
    if (ok) umma_commit(acc_bar);
  } else {
    // tensor memory -> this CTA's partial tile [column][row] (a warp writes 32 consecutive words: no bank conflicts).
    // The accumulator is complete, so every stage has been read and no copy is in flight.
    const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(acc_bar, 0u, abort_flag, a.wait_ns));
    if (!ok && lane == 0) report_status(a.status, kGemmAccTimeout, 8, blockIdx.x, 0);
    if (ok) {
      tc_fence_after_sync();
      const int wq = warp & 3;  // tensor-memory lane quarter this warp may read
      float* park = reinterpret_cast<float*>(smem) + wq * 32 + lane;
      for (int c0 = 0; c0 < n_tile; c0 += 16) {
        uint32_t v[16];
        tmem_ld_16(tmem_base + ((uint32_t)(wq * 32) << 16) + c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) park[(c0 + j) * kSkM] = __uint_as_float(v[j]);
      }
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kSkN);
  }
  if (S > 1) cluster_sync_all();  // all partial tiles of the block are parked

  // This CTA's token columns: add the pieces in K order, finish, store.
  const uint32_t base = smem_u32(smem);
  constexpr int kOut = kGateUp ? 64 : kSkM;          // outputs per column
  constexpr int kCols = kSkThreads / 64;             // columns at a time, 64 threads each (gate/up)
  constexpr int kPer = kGateUp ? 1 : 2;              // rows per thread: r and r + 64
  const int r = tid & 63;
  for (int c = s + S * (tid >> 6); c < n_rows; c += S * kCols) {
    float lo = 0.f, hi = 0.f;
    for (int p = 0; p < S; ++p) {
      const uint32_t from = (S > 1 ? cluster_map(base, (uint32_t)p) : base) + (uint32_t)(c * kSkM + r) * 4u;
      lo += ld_cluster_f32(from);
      hi += ld_cluster_f32(from + 256u);
    }
    float o[2] = {kGateUp ? swiglu_clamped(lo, hi, a.limit) : lo, hi};
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
      const long long col = (long long)unit * kOut + r + 64 * h;
      if (a.out_cols > 0 && col >= a.out_cols) continue;
      const long long at = (long long)(t0 + c) * a.out_pitch + col;
      if (a.out_fp32) {
        static_cast<float*>(a.out)[at] = o[h];
      } else {
        float v = bf16_round(o[h]);
        if (a.residual != nullptr) {
          float add = ldcg_bf16(a.residual, (long long)(t0 + c) * a.residual_pitch + col);
          if (a.residual2 != nullptr) add = bf16_round(add + ldcg_bf16(a.residual2, (long long)(t0 + c) * a.residual2_pitch + col));
          v += add;
        }
        static_cast<__nv_bfloat16*>(a.out)[at] = __float2bfloat16_rn(v);
      }
    }
  }
  if (S > 1) cluster_sync_all();  // nobody leaves while its partial tile may still be read
}

}  // namespace mf

// Pieces that K is cut into: the smallest S <= 8 with the fewest K steps on the busiest SM (two CTAs fit an SM; a
// CTA's own start and finish are worth about four steps).
static int skinny_split(int units, int k_blocks, int n_sms) {
  int best = 1;
  long long best_cost = -1;
  for (int S = 1; S <= 8 && S <= k_blocks; ++S) {
    const long long per_sm = ((long long)units * S + n_sms - 1) / n_sms;
    const long long cost = per_sm * ((k_blocks + S - 1) / S) + 4 * ((per_sm + 1) / 2);
    if (best_cost < 0 || cost < best_cost) {
      best = S;
      best_cost = cost;
    }
  }
  return best;
}

extern "C" int mf_skinny_gemm(const void* tmap_w, const mf_skinny_args* a, int gate_up, int n_sms, mf_stream_t stream) {
  using namespace mf;
  if (!tmap_w || !a || !a->x || !a->out || n_sms < 1) return -1;
  if (a->T == 0) return 0;
  if (a->T < 0 || a->k_blocks < 1 || a->row_blocks < 1) return -2;
  if ((a->x_pitch & 15) != 0 || (reinterpret_cast<uintptr_t>(a->x) & 15) != 0) return -3;
  if (a->residual2 != nullptr && a->residual == nullptr) return -4;
  if (a->residual != nullptr && a->out_fp32) return -4;  // added in the bf16 epilogue only
  CUtensorMap tw, tx;
  memcpy(&tw, tmap_w, sizeof(tw));
  // The token rows may be any buffer of the caller's (no copy into a fixed one): rows past T read as zero.
  const int e = mf_make_pitched_tmap(&tx, a->x, a->T, (long long)a->k_blocks * 64, 2, a->x_pitch, kSkN);
  if (e) return e;
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess) return (int)de;
  static bool configured[64][2] = {};
  auto kern = gate_up ? skinny_gemm_kernel<true> : skinny_gemm_kernel<false>;
  if (dev < 0 || dev >= 64 || !configured[dev][gate_up != 0]) {
    de = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSkSmem);
    if (de != cudaSuccess) return (int)de;
    if (dev >= 0 && dev < 64) configured[dev][gate_up != 0] = true;
  }
  const int tiles = (a->T + kSkN - 1) / kSkN;
  const int S = skinny_split(a->row_blocks * tiles, a->k_blocks, n_sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a->row_blocks * S, tiles);
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = kSkSmem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (S > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = S;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (mf_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return (int)cudaLaunchKernelEx(&cfg, kern, tw, tx, *a, S);
}

// Block-scaled e4m3 weights -> bf16, one pass over the tensor.
//
// Used by the long-prefill path of layers that hold e4m3 experts: from 256-row token tiles on, the bf16 grouped
// GEMMs (two accumulators of 256 columns, no per-K-block promotion) are faster than the block-scaled ones, so the
// layer expands the experts of the current forward into a bf16 scratch first (three times the e4m3 bytes of HBM
// traffic, a few percent of a compute-bound forward) and runs the bf16 kernels on it.
//
// Layout: w8 [rows, K] e4m3, scale [rows / 128, K / 128] fp32 (the checkpoint's weight_scale_inv, experts
// concatenated along the rows), out [rows, K] bf16.  value = float(e4m3) * scale, rounded once to bf16.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "expand.cuh"
#include "moeflow_b200.h"

namespace mf {

// A CTA expands 16 rows of one 128-row block, 8 values (8 bytes in, 16 out) per thread and step: whole sectors both ways,
// eight loads in flight, and addresses that only grow (the rows are contiguous), so that the pass is bound by memory.
// With 16 values per step and a 64-bit division for the row in each it was bound by its instructions: 36 experts of
// 3 x 4096 x 1536 (0.68 GB in, 1.36 GB out) took 430 us, 4.7 TB/s.
constexpr int kDqThreads = 256;
constexpr int kDqRows = 16;
constexpr int kDqBatch = 8;

__global__ void __launch_bounds__(kDqThreads) dequant_block_fp8_kernel(const uint8_t* w8, const float* scale, __nv_bfloat16* out, int K, int* zero) {
  grid_dep_wait_cta();
  grid_dep_launch();
  if (zero != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero = 0;
  const int cpr = K / 8;                                  // steps of 8 values per row
  const int n = kDqRows * cpr;
  const size_t at = (size_t)blockIdx.x * n;               // rows are contiguous
  const uint2* src = reinterpret_cast<const uint2*>(w8) + at;
  uint4* dst = reinterpret_cast<uint4*>(out) + at;
  const float* sc = scale + (size_t)(blockIdx.x / (128 / kDqRows)) * (K / 128);
  const int wrap = kDqThreads % cpr;
  int c = threadIdx.x % cpr;
  for (int i = threadIdx.x; i < n; i += kDqThreads * kDqBatch) {
    uint2 q[kDqBatch];
    float s[kDqBatch];
#pragma unroll
    for (int j = 0; j < kDqBatch; ++j) {
      if (i + j * kDqThreads < n) {
        q[j] = __ldcs(src + i + j * kDqThreads);  // streamed once
        s[j] = __ldg(sc + (c >> 4));
      }
      c += wrap;
      if (c >= cpr) c -= cpr;
    }
#pragma unroll
    for (int j = 0; j < kDqBatch; ++j)
      if (i + j * kDqThreads < n) dst[i + j * kDqThreads] = expand_8(q[j], s[j]);
  }
}

}  // namespace mf

// rows % 128 == 0, K % 128 == 0; pointers 16-byte aligned.  Returns 0, a negative code for bad arguments, or the
// CUDA error of the launch.
extern "C" int mf_dequant_block_fp8_zero(const void* w8, const float* scale, void* out_bf16, long long rows, int K, int* zero,
                                         void* stream) {
  if (w8 == nullptr || scale == nullptr || out_bf16 == nullptr) return -1;
  if (rows <= 0 || K <= 0 || rows % 128 != 0 || K % 128 != 0) return -2;
  if ((reinterpret_cast<uintptr_t>(w8) | reinterpret_cast<uintptr_t>(out_bf16)) & 15) return -3;
  if (rows / mf::kDqRows > 0x7fffffffLL) return -2;
  return (int)mf::launch_kernel(mf::dequant_block_fp8_kernel, dim3((unsigned)(rows / mf::kDqRows)), dim3(mf::kDqThreads), 0,
                                static_cast<cudaStream_t>(stream), true, static_cast<const uint8_t*>(w8), scale,
                                static_cast<__nv_bfloat16*>(out_bf16), K, zero);
}

extern "C" int mf_dequant_block_fp8(const void* w8, const float* scale, void* out_bf16, long long rows, int K, void* stream) {
  return mf_dequant_block_fp8_zero(w8, scale, out_bf16, rows, K, nullptr, stream);
}

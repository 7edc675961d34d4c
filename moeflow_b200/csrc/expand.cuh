// Block-scaled e4m3 values to bf16: float(e4m3) * scale, rounded once.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "common.cuh"
#include "moeflow_b200.h"

namespace mf {

__device__ __forceinline__ uint4 expand_8(uint2 q, float s) {
  const uint32_t words[2] = {q.x, q.y};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_fp8x2_storage_t pair = (__nv_fp8x2_storage_t)((words[i >> 1] >> (16 * (i & 1))) & 0xffffu);
    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(pair, __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
    const __nv_bfloat162 b = __floats2bfloat162_rn(f.x * s, f.y * s);
    o[i] = *reinterpret_cast<const uint32_t*>(&b);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// One warp's share of a whole matrix, beside a GEMM (mf_gemm_args.expand_*): every `step`-th piece of MF_EXPAND_PIECE values from
// `first` on, 16 values per lane and load, eight loads in flight.  Returns the number of pieces.
__device__ __forceinline__ int expand_pieces(const mf_gemm_args& a, int first, int step, int lane) {
  const int K = a.expand_cols, cpr = K / 16, pieces = (int)((long long)a.expand_rows * K / MF_EXPAND_PIECE);
  int n = 0;
#pragma unroll 1
  for (int i = first; i < pieces; i += step, ++n) {
    const int at = i * (MF_EXPAND_PIECE / 16) + lane;  // in steps of 16 values
    const uint4* src = static_cast<const uint4*>(a.expand_src) + at;
    uint4* dst = static_cast<uint4*>(a.expand_out) + 2ll * at;
    uint4 q[8];
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int row = (at + 32 * j) / cpr, c = (at + 32 * j) - row * cpr;
      q[j] = __ldcs(src + 32 * j);  // streamed once
      s[j] = __ldg(a.expand_scale + (row >> 7) * (K >> 7) + (c >> 3));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dst[64 * j] = expand_8(make_uint2(q[j].x, q[j].y), s[j]);
      dst[64 * j + 1] = expand_8(make_uint2(q[j].z, q[j].w), s[j]);
    }
  }
  return n;
}

}  // namespace mf

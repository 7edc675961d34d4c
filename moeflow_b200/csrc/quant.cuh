// 1x128 activation quantisation (bf16 -> e4m3 + one fp32 scale per row and 128-wide group), shared by the stand-alone
// quantiser, the metadata kernel (received rows) and the gate/up epilogue (activations).
#pragma once

#include <cuda_fp8.h>

#include "common.cuh"

namespace mf {

// Scale of a group with absolute maximum `amax`; values are multiplied by its reciprocal.
__device__ __forceinline__ float group_scale(float amax) { return fmaxf(amax, 1e-10f) / 448.f; }
__device__ __forceinline__ uint8_t to_e4m3(float x, float inv_scale) {
  return (uint8_t)__nv_cvt_float_to_fp8(x * inv_scale, __NV_SATFINITE, __NV_E4M3);
}

__device__ __forceinline__ uint16_t to_e4m3x2(float2 v, float inv_scale) {  // v.x in the low byte
  return (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(v.x * inv_scale, v.y * inv_scale), __NV_SATFINITE, __NV_E4M3);
}

// Chunk c of one row (`v`: its 8 bf16 values).  Half a warp holds a group (threads 16 n ..): all of it calls this.
__device__ __forceinline__ void quant_chunk(const uint4& v, int c, uint8_t* q_row, float* scale_row) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
  float f[8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
    amax = fmaxf(amax, fmaxf(fabsf(t.x), fabsf(t.y)));
  }
  const unsigned group = 0xffffu << (lane_id() & 16);  // named, not taken from where the compiler lets the warp meet
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(group, amax, off));
  const float scale = group_scale(amax);
  const float inv = 1.f / scale;
  uint2 packed;
  uint8_t* pb = reinterpret_cast<uint8_t*>(&packed);
#pragma unroll
  for (int i = 0; i < 8; ++i) pb[i] = to_e4m3(f[i], inv);
  reinterpret_cast<uint2*>(q_row)[c] = packed;
  if ((c & 15) == 0) scale_row[c >> 4] = scale;
}
__device__ __forceinline__ void quant_chunk(const uint8_t* row, int c, uint8_t* q_row, float* scale_row) {
  quant_chunk(__ldcg(reinterpret_cast<const uint4*>(row) + c), c, q_row, scale_row);
}

}  // namespace mf

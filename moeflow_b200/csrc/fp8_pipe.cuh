// What the two forms of the block-scaled e4m3 GEMM share: a pipeline position, arithmetic on pairs of fp32 values, and the
// gather of a tile's rows by four warps.
#pragma once

#include "common.cuh"

namespace mf {

constexpr int kF8BlockM = 128;        // weight rows per block (a row of 128x128 scale blocks)
constexpr int kF8TileA = 128 * 128;   // bytes of 128 weight rows x one K block
constexpr int kF8MaxKb = 32;          // K <= 4096 (one unit never spans more K blocks than this)

struct F8Pipe {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance(int n) {
    if (++stage == n) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

// Two fp32 values in one 64-bit register: the promotion works on pairs of token columns (one instruction for two
// multiply-adds, each rounded like fmaf).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f32x2 pack2(uint32_t lo, uint32_t hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// first + row * pitch in one multiply-add per use: as plain arithmetic the compiler keeps the 64-bit products of all rows, which
// a gather warp has no registers for.
__device__ __forceinline__ uint64_t row_at(uint64_t first, int row, int pitch) {
  uint64_t at;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(at) : "r"(row), "r"(pitch), "l"(first));
  return at;
}
// 16 bytes of every 16th row of a tile of n_rows into rows of 128 bytes.  `first`: address of those bytes in row 0.  Rows
// 2 GiB apart and more are addressed in units of 16 bytes, two instructions more for each.
template <int kRows>
__device__ __forceinline__ void gather_chunks(uint32_t dst, uint64_t first, const int (&row)[kRows], long long pitch, int n_rows) {
  if (pitch <= 0x7fffffffll) {
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (16 * i < n_rows) cp_async_16(dst + i * 2048, reinterpret_cast<const void*>(row_at(first, row[i], (int)pitch)), 16u);
  } else {
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (16 * i < n_rows) cp_async_16(dst + i * 2048, reinterpret_cast<const void*>(row_at(first >> 4, row[i], (int)(pitch >> 4)) << 4), 16u);
  }
}

}  // namespace mf

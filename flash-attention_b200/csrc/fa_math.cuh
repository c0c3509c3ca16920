// Arithmetic helpers of the softmax / gradient loops: packed two-wide fp32 operations
// (fma / mul / add on register pairs, sm_100), three-input max, fast exp2, 16-bit packing.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace fa {

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint64_t pack_f2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// d = a * b + c on both halves
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack_lowp(float lo, float hi) {
  uint32_t r;
  if constexpr (BF16) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  } else {
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  }
  return r;
}

// A tile of 32 rows whose threads hold one row each leaves through shared memory: stored straight from the registers, every
// 16-byte store of a warp touches 32 rows, one L1 tag cycle each.  The rows are put in a warp's own piece of shared memory
// (32 rows of CH 16-byte chunks, in the 64- or 128-byte swizzle of a tensor map: neither side has bank conflicts) and leave by
// TMA, or read back CH lanes to a row where TMA would write rows that are not the warp's.  dK and dV
// of a block of 128 keys: 4096 (d = 128) and 2048 (d = 64) tag cycles -> 512 and 256, which counts where a block has few query
// tiles.  Whole backward, us, before -> now: 64 x 12 x 512 (d = 64) 305 -> 278, 16 x 12 x 1024 230 -> 218, 8 x 12 x 4096 1185
// -> 1135, with dropout 1343 -> 1330; 16 x 12 x 1000 causal (d = 128) 287 -> 271.
template <int CH>
__device__ __forceinline__ uint32_t stage_offset(int row, int chunk) {
  static_assert(CH == 4 || CH == 8, "64 or 128 bytes a row");
  return row * (CH * 16) + ((chunk ^ (CH == 8 ? row & 7 : (row >> 1) & 3)) << 4);
}
// Rows below `rows` and chunks below `chunks` of a warp's piece to global memory; `dst`: row 0, chunk 0.
template <int CH>
__device__ __forceinline__ void stage_copy_out(const uint8_t* piece, uint16_t* dst, int64_t row_stride, int rows, int chunks,
                                               int lane) {
  const int r0 = lane / CH, c = lane % CH;
#pragma unroll 4
  for (int i = 0; i < CH; ++i) {
    const int r = i * (32 / CH) + r0;
    if (r < rows && c < chunks)
      *reinterpret_cast<uint4*>(dst + r * row_stride + c * 8) = *reinterpret_cast<const uint4*>(piece + stage_offset<CH>(r, c));
  }
}

}  // namespace fa

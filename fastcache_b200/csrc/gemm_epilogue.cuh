// What the epilogues of the prompt-size GEMMs (gemm.cu, gemm_2cta.cu) share: bias and activation of 32 columns held in
// registers, and slabs of 64 output columns in shared memory (128 rows of 128 bytes, 128-byte swizzle) that TMA stores.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "gemm.h"
#include "ptx.cuh"

namespace fc {

constexpr int SLAB = 64;                          // output columns an epilogue group stores at a time
constexpr int SLAB_BYTES = 128 * SLAB * 2;

__device__ __forceinline__ float apply_act(float v, int act) {
  switch (act) {
    case ACT_RELU: return fmaxf(v, 0.f);
    case ACT_GELU: return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
    case ACT_GELU_TANH: {
      float u = 0.7978845608028654f * (v + 0.044715f * v * v * v), th;
      asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(u));
      return 0.5f * v * (1.f + th);
    }
    case ACT_QUICK_GELU: return __fdividef(v, 1.f + __expf(-1.702f * v));
    case ACT_SILU: return __fdividef(v, 1.f + __expf(-v));
    default: return v;
  }
}

// The activation of 32 values with the (uniform) selector tested once, not per element.
__device__ __forceinline__ void apply_act_chunk(float (&v)[32], int act) {
  switch (act) {
    case ACT_NONE: break;
    case ACT_RELU:
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = apply_act(v[t], ACT_RELU);
      break;
    case ACT_GELU:
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = apply_act(v[t], ACT_GELU);
      break;
    case ACT_GELU_TANH:
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = apply_act(v[t], ACT_GELU_TANH);
      break;
    case ACT_QUICK_GELU:
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = apply_act(v[t], ACT_QUICK_GELU);
      break;
    case ACT_SILU:
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = apply_act(v[t], ACT_SILU);
      break;
    default: break;
  }
}

// v += bias[col ... col + 31]; `whole`: all 32 are inside the row of n values
__device__ __forceinline__ void add_bias_chunk(float (&v)[32], const __nv_bfloat16* bias, int col, int n, bool whole) {
  if (whole && (reinterpret_cast<uintptr_t>(bias + col) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 bv = *reinterpret_cast<const uint4*>(bias + col + q * 8);
      const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {      // a bf16 is the upper half of the fp32 with the same value
        v[q * 8 + e * 2] += __uint_as_float(bw[e] << 16);
        v[q * 8 + e * 2 + 1] += __uint_as_float(bw[e] & 0xffff0000u);
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < 32; ++t)
      if (col + t < n) v[t] += __bfloat162float(bias[col + t]);
  }
}

// 32 packed columns (half 0 or 1 of a slab) of row `row`
__device__ __forceinline__ uint4* slab_piece(uint8_t* slab, int row, int half, int q) {
  return reinterpret_cast<uint4*>(slab + row * 128 + (((half * 4 + q) ^ (row & 7)) << 4));
}
__device__ __forceinline__ void slab_put(uint8_t* slab, int row, int half, const uint32_t (&u)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) *slab_piece(slab, row, half, q) = make_uint4(u[4 * q], u[4 * q + 1], u[4 * q + 2], u[4 * q + 3]);
}
__device__ __forceinline__ void slab_add(uint8_t* slab, int row, int half, float (&v)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 a = *slab_piece(slab, row, half, q);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[q * 8 + 2 * e] += __uint_as_float(w[e] << 16);
      v[q * 8 + 2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
    }
  }
}

}  // namespace fc

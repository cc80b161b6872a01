// KV quantisers: per-group absmax quantisation of bf16 rows to INT8 (symmetric / asymmetric), INT4 and NF4
// (two codes per byte, even index in the low nibble) and scaled FP8 (e4m3 / e5m2), their inverses, and the
// quantise-and-restore round trip in one pass ("fake quantisation").
//
// Up to 32 lanes own one group of `g` consecutive values of a row (g = the whole row for the INT8 and FP8 modes): a
// lane holds up to QMAX_CHUNKS 16-byte pieces in registers, the group statistics (absmax, or min and max) are a
// reduction over the lanes, and the codes go out as packed words.  The op is a single pass over the data: bound by
// bandwidth (2 bytes read, 1 / 0.5 bytes written per value), nothing to put on the tensor cores.
//
// The arithmetic matches the PyTorch statements of fastcache_b200/compress/quant.py operation for operation
// (fp32 division by the scale, round-half-to-even, the same clamps), so codes and scales are bit-identical.
//
// What bounds it: at 2 + 1 bytes a value the copy rate allows ~16 instructions per value, and a division, a
// rounding, two clamps and a conversion each are ~45: with those the kernel ran at a third of the copy rate.  The
// codes are therefore taken from x * r, r ~ 1 / a, one multiply-add that rounds, and the division is done only for the
// values whose quotient lies so close to the border between two codes that its error could matter.  INT8, 1179648 rows
// of 128 values (458 MB): 199 us with the divisions, 133 us dividing all eight values of a lane that has an unsure one
// (a fraction of a percent of the values, but half of the warps), 111 us so.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <stdexcept>
#include <string>

#include "gemm.h"
#include "kernels.h"
#include "ptx.cuh"

namespace fc {

using bf16 = __nv_bfloat16;

constexpr int QMAX_CHUNKS = 4;            // 16-byte pieces per lane: groups of up to 32 * 4 * 8 = 1024 values

__constant__ float c_nf4[16] = {-1.0f, -0.6961928f, -0.52507305f, -0.39491749f, -0.28444138f, -0.18477343f,
                                -0.09105004f, 0.0f, 0.0795803f, 0.1609302f, 0.2461123f, 0.33791524f, 0.44070983f,
                                0.562617f, 0.72295684f, 1.0f};

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]);
  u.y = pack_bf16(f[2], f[3]);
  u.z = pack_bf16(f[4], f[5]);
  u.w = pack_bf16(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// code of one value and the value it stands for; `a` = scale (INT8, FP8) or absmax (INT4, NF4), `z` = zero point
template <int MODE>
__device__ __forceinline__ int encode(float x, float a, float z) {
  static_assert(MODE != QUANT_NF4, "by nf4_code_fast");
  if (MODE == QUANT_INT8) return int(fminf(fmaxf(rintf(__fdiv_rn(x, a)), -127.f), 127.f));
  if (MODE == QUANT_INT8_ASYM) return int(fminf(fmaxf(rintf(__fdiv_rn(x - z, a)), 0.f), 255.f));
  if (MODE == QUANT_INT4) return int(fminf(fmaxf(rintf(__fdiv_rn(x, a) * 7.0f), -8.f), 7.f)) + 8;
  if (MODE == QUANT_FP8_E4M3) return int(__nv_cvt_float_to_fp8(__fdiv_rn(x, a), __NV_SATFINITE, __NV_E4M3));
  return int(__nv_cvt_float_to_fp8(__fdiv_rn(x, a), __NV_SATFINITE, __NV_E5M2));
}
template <int MODE>
__device__ __forceinline__ float decode(int q, float a, float z) {
  if (MODE == QUANT_INT8) return float(q) * a;
  if (MODE == QUANT_INT8_ASYM) return __fadd_rn(__fmul_rn(float(q), a), z);   // two roundings, like the tensor ops
  if (MODE == QUANT_INT4) return __fdiv_rn(float(q) - 8.0f, 7.0f) * a;
  if (MODE == QUANT_NF4) return c_nf4[q] * a;
  const __nv_fp8_interpretation_t kind = (MODE == QUANT_FP8_E4M3) ? __NV_E4M3 : __NV_E5M2;
  const __half_raw h = __nv_cvt_fp8_to_halfraw(__nv_fp8_storage_t(q), kind);
  return __half2float(__half(h)) * a;
}

// Codes of eight values from the quotient t = x * r, r ~ 1 / a, in place of the division.  r is off by one unit in the
// last place (2^-23) at most, t and the division that the codes are defined by by half of one, so t and fl(x / a) differ
// by less than 2^-22 |t|: 6.1e-5 for the largest quotient, 255.  Returns a bit for each value whose t is closer than 1e-4
// (INT8, INT4), 1e-6 (NF4, |t| <= 1) or 2^-20 |t| (FP8) to the border between two codes, or is no number: the caller then
// divides, as it does where 1 / a would be subnormal.
// `s_mid` (NF4 only): the 15 midpoints, with -inf before and +inf behind them.
constexpr float QROUND = 12582912.f;      // 1.5 * 2^23: adding it rounds to an integer, half to even, in the low bits
constexpr float QNEAR = 0.5f - 1e-4f;

__device__ __forceinline__ int nf4_code_fast(float t, const float* s_mid);

template <int MODE>
__device__ __forceinline__ uint32_t encode8_fast(const uint4& raw, float r, float z, const float* s_mid, uint2& w) {
  float x[8];
  unpack8(raw, x);
  uint32_t unsure = 0;
  if (MODE == QUANT_INT8 || MODE == QUANT_INT8_ASYM || MODE == QUANT_INT4) {
    // x r + QROUND rounds to an integer whose low byte is the code (two's complement; INT4 counts from 8); what the
    // rounding took off is one more multiply-add
    constexpr float OFFSET = MODE == QUANT_INT4 ? QROUND + 8.f : QROUND;
    const float q = MODE == QUANT_INT4 ? r * 7.0f : r;
    uint32_t m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float y = MODE == QUANT_INT8_ASYM ? x[i] - z : x[i];
      const float n = __fmaf_rn(y, q, OFFSET);
      if (!(fabsf(__fmaf_rn(y, q, __fsub_rn(OFFSET, n))) < QNEAR)) unsure |= 1u << i;
      m[i] = __float_as_uint(n);
    }
    w.x = __byte_perm(__byte_perm(m[0], m[1], 0x0040), __byte_perm(m[2], m[3], 0x0040), 0x5410);
    w.y = __byte_perm(__byte_perm(m[4], m[5], 0x0040), __byte_perm(m[6], m[7], 0x0040), 0x5410);
  } else if (MODE == QUANT_NF4) {
    w = make_uint2(0, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float t = x[i] * r;
      const int c = nf4_code_fast(t, s_mid);
      if (!(t - s_mid[c - 1] > 1e-6f && s_mid[c] - t > 1e-6f)) unsure |= 1u << i;
      (i < 4 ? w.x : w.y) |= uint32_t(c) << (8 * (i & 3));
    }
  } else {
    // both ends of the interval that holds the quotient have the same code
    const __nv_fp8_interpretation_t kind = (MODE == QUANT_FP8_E4M3) ? __NV_E4M3 : __NV_E5M2;
    constexpr float UP = 1.f + 0x1p-20f, DOWN = 1.f - 0x1p-20f;
    const float up = r * UP, down = r * DOWN;
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      u[i] = __nv_cvt_float2_to_fp8x2(make_float2(x[2 * i] * up, x[2 * i + 1] * up), __NV_SATFINITE, kind);
      if (u[i] != __nv_cvt_float2_to_fp8x2(make_float2(x[2 * i] * down, x[2 * i + 1] * down), __NV_SATFINITE, kind)) unsure |= 3u << (2 * i);
    }
    w.x = __byte_perm(u[0], u[1], 0x5410);
    w.y = __byte_perm(u[2], u[3], 0x5410);
  }
  return unsure;
}

// group statistics of the values a warp holds -> (a, z) as `encode` wants them
template <int MODE>
__device__ __forceinline__ void group_params(float amax, float lo, float hi, float& a, float& z) {
  z = 0.f;
  if (MODE == QUANT_INT8) a = __fdiv_rn(fmaxf(amax, 1e-8f), 127.0f);
  else if (MODE == QUANT_INT8_ASYM) {
    a = fmaxf(__fdiv_rn(hi - lo, 255.0f), 1e-8f);
    z = lo;
  } else if (MODE == QUANT_INT4 || MODE == QUANT_NF4) a = fmaxf(amax, 1e-8f);
  else a = __fdiv_rn(fmaxf(amax, 1e-8f), MODE == QUANT_FP8_E4M3 ? 448.0f : 57344.0f);
}

// the codes of the values in `which` (bits 0 ... 7) by division.  With bf16 inputs borders are met exactly and not only by
// chance (a value of half the largest one lies between 63 and 64 in INT8, between 3 and 4 in INT4), a fraction of a
// percent of all values: half of all warps come here with some lane, mostly for one value
template <int MODE>
__device__ __forceinline__ void encode_exact(uint32_t which, const uint4& raw, float a, float z, const float* s_mid, uint2& w) {
  while (which != 0u) {
    const int i = __ffs(which) - 1;
    which &= which - 1;
    const uint32_t pair = i < 4 ? (i < 2 ? raw.x : raw.y) : (i < 6 ? raw.z : raw.w);
    const float x = __uint_as_float((i & 1) ? pair & 0xffff0000u : pair << 16);
    int e;
    if constexpr (MODE == QUANT_NF4) e = nf4_code_fast(__fdiv_rn(x, a), s_mid);
    else e = encode<MODE>(x, a, z);
    const int at = 8 * (i & 3);
    const uint32_t old = i < 4 ? w.x : w.y, now = (old & ~(0xFFu << at)) | (uint32_t(e & 0xFF) << at);
    if (i < 4) w.x = now;
    else w.y = now;
  }
}

// Lanes per group: a group of g values is g / 8 pieces of 16 bytes.  W lanes share one group, CH pieces each; 32 / W
// groups sit side by side in a warp and QU such batches are in flight per iteration.  Two pieces per lane halve what a
// group costs besides its values (the shuffles of the reduction, the scale and its reciprocal); only groups of up to 32
// values have one.
// FEW groups (see launch_quantize_m): one piece per lane and one batch per warp, so that as many warps as there are share the
// work; FP8 divides there, which is a shorter chain than both ends of the interval.
constexpr int quant_batches(int ch, bool few) { return few ? 1 : ch > 2 ? 2 : 4; }

template <int W>
__device__ __forceinline__ float sub_max(float v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int W>
__device__ __forceinline__ float sub_min(float v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// the 16 restored values of the two 4-bit modes, in shared memory (an index that differs between lanes reads a
// __constant__ table one lane at a time)
template <int MODE>
__device__ __forceinline__ void fill_table4(float* s_tab) {
  if (threadIdx.x < 16)
    s_tab[threadIdx.x] = (MODE == QUANT_NF4) ? c_nf4[threadIdx.x] : __fdiv_rn(float(int(threadIdx.x)) - 8.0f, 7.0f);
  __syncthreads();
}
// NF4 code by bisection over the 15 midpoints between neighbouring table entries: the entry nearest to t, the
// lower one at a midpoint (what argmin over the distances gives)
__device__ __forceinline__ int nf4_code_fast(float t, const float* s_mid) {
  int c = (t > s_mid[7]) ? 8 : 0;
  c += (t > s_mid[c + 3]) ? 4 : 0;
  c += (t > s_mid[c + 1]) ? 2 : 0;
  c += (t > s_mid[c]) ? 1 : 0;
  return c;
}

// x [groups, g] bf16 (rows of D values cut into D / g groups).  FAKE: y = decode(encode(x)) in bf16, no codes.
// Otherwise: codes as bytes (INT8, FP8: one per value; INT4 / NF4: one per two values), `scale` [groups] (the
// scale, or the absmax for the 4-bit modes) and, for the asymmetric mode, `zero` [groups].
template <int MODE, bool FAKE, int W, int CH, bool FEW>
__global__ void __launch_bounds__(256)
quantize_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale,
                float* __restrict__ zero, bf16* __restrict__ y, long long groups, int g) {
  __shared__ float s_tab[16];
  __shared__ float s_borders[17];
  float* const s_mid = s_borders + 1;
  constexpr bool FOUR_BIT = (MODE == QUANT_INT4 || MODE == QUANT_NF4);
  if (FOUR_BIT) {
    if (MODE == QUANT_NF4) {
      if (threadIdx.x < 15) s_mid[threadIdx.x] = 0.5f * (c_nf4[threadIdx.x] + c_nf4[threadIdx.x + 1]);
      else if (threadIdx.x < 17) s_borders[threadIdx.x == 15 ? 0 : 16] = threadIdx.x == 15 ? -INFINITY : INFINITY;
    }
    fill_table4<MODE>(s_tab);
  }
  const int lane = threadIdx.x & 31;
  const int sub = lane / W, l = lane % W;
  constexpr int GPW = 32 / W;                                    // groups per warp and batch
  constexpr int QU = quant_batches(CH, FEW);
  const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int chunks = g >> 3;
  for (long long g0 = warp * (GPW * QU); g0 < groups; g0 += nwarps * (GPW * QU)) {
    uint4 raw[QU][CH];
    const long long e0 = (g0 + sub) * g + l * 8;                 // this lane's first element of the batch
    const int left = int(min(groups - g0 - sub, (long long)(GPW * QU)));   // groups u * GPW < left are there
#pragma unroll
    for (int u = 0; u < QU; ++u) {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        raw[u][c] = make_uint4(0, 0, 0, 0);
        if (u * GPW < left && l + W * c < chunks) raw[u][c] = *reinterpret_cast<const uint4*>(x + e0 + u * GPW * g + W * c * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < QU; ++u) {
      float amax = 0.f, lo = INFINITY, hi = -INFINITY;
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        if (u * GPW < left && l + W * c < chunks) {
          // two values at a time; like fminf / fmaxf these take the number of a number and a NaN
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u][c]);
          if (MODE == QUANT_INT8_ASYM) {
            const float2 a = __bfloat1622float2(__hmin2(__hmin2(h[0], h[1]), __hmin2(h[2], h[3])));
            const float2 b = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
            lo = fminf(lo, fminf(a.x, a.y));
            hi = fmaxf(hi, fmaxf(b.x, b.y));
          } else {
            const float2 a = __bfloat1622float2(
                __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3]))));
            amax = fmaxf(amax, fmaxf(a.x, a.y));
          }
        }
      }
      if (MODE == QUANT_INT8_ASYM) {
        lo = sub_min<W>(lo);
        hi = sub_max<W>(hi);
      } else {
        amax = sub_max<W>(amax);
      }
      if (u * GPW >= left) continue;
      const long long grp = g0 + u * GPW + sub, e = e0 + u * GPW * g;
      float a, z;
      group_params<MODE>(amax, lo, hi, a, z);
      float r;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
      if (!FAKE && l == 0) {
        scale[grp] = a;
        if (MODE == QUANT_INT8_ASYM) zero[grp] = z;
      }
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        if (l + W * c >= chunks) continue;
        uint2 w;                                                 // eight codes, one byte each
        if constexpr (FEW && (MODE == QUANT_FP8_E4M3 || MODE == QUANT_FP8_E5M2)) {
          float v[8];
          unpack8(raw[u][c], v);
          w = make_uint2(0, 0);
#pragma unroll
          for (int i = 0; i < 8; ++i) (i < 4 ? w.x : w.y) |= uint32_t(encode<MODE>(v[i], a, z) & 0xFF) << (8 * (i & 3));
        } else {
          const uint32_t unsure = encode8_fast<MODE>(raw[u][c], r, z, s_mid, w);
          encode_exact<MODE>(a < 0x1p125f ? unsure : 0xFFu, raw[u][c], a, z, s_mid, w);
        }
        if (FAKE) {
          float out[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int code = int(((i < 4 ? w.x : w.y) >> (8 * (i & 3))) & 0xFFu);
            out[i] = FOUR_BIT ? s_tab[code] * a : decode<MODE>((MODE == QUANT_INT8) ? int(int8_t(code)) : code, a, z);
          }
          store8(y + e + W * c * 8, out);
        } else if (FOUR_BIT) {
          // bytes 0, 2, ... hold the low nibbles, 1, 3, ... the high ones
          const uint32_t lo = (w.x | (w.x >> 4)) & 0x00FF00FFu, hi = (w.y | (w.y >> 4)) & 0x00FF00FFu;
          *reinterpret_cast<uint32_t*>(q + ((e + W * c * 8) >> 1)) = __byte_perm(lo, hi, 0x6420);
        } else {
          *reinterpret_cast<uint2*>(q + e + W * c * 8) = w;
        }
      }
    }
  }
}

// one thread per 16-byte piece of the output, grid-stride: nothing is shared between the pieces of a group but its
// scale, so no warp-level structure is needed
template <int MODE>
__global__ void __launch_bounds__(256)
dequantize_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scale, const float* __restrict__ zero,
                  bf16* __restrict__ y, long long groups, int g) {
  __shared__ float s_tab[16];
  constexpr bool FOUR_BIT = (MODE == QUANT_INT4 || MODE == QUANT_NF4);
  if (FOUR_BIT) fill_table4<MODE>(s_tab);
  const int chunks = g >> 3;
  const long long total = groups * chunks;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < total;
       p += (long long)gridDim.x * blockDim.x) {
    const long long grp = p / chunks;
    const int idx = int(p - grp * chunks);
    const float a = scale[grp];
    const float z = (MODE == QUANT_INT8_ASYM) ? zero[grp] : 0.f;
    float out[8];
    if (FOUR_BIT) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(q + grp * (g >> 1) + idx * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t b = (w >> (8 * i)) & 0xFF;
        out[2 * i] = s_tab[b & 0xF] * a;
        out[2 * i + 1] = s_tab[b >> 4] * a;
      }
    } else {
      const uint2 w = *reinterpret_cast<const uint2*>(q + grp * g + idx * 8);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t b0 = (w.x >> (8 * i)) & 0xFF, b1 = (w.y >> (8 * i)) & 0xFF;
        out[i] = decode<MODE>((MODE == QUANT_INT8) ? int(int8_t(b0)) : int(b0), a, z);
        out[4 + i] = decode<MODE>((MODE == QUANT_INT8) ? int(int8_t(b1)) : int(b1), a, z);
      }
    }
    store8(y + grp * g + idx * 8, out);
  }
}

static int quant_grid(long long work_items, int per_block) {
  const long long blocks = (work_items + per_block - 1) / per_block;
  return int(blocks < 1 ? 1 : (blocks > 148 * 16 ? 148 * 16 : blocks));
}

// Groups that the form for many would spread over at most QUANT_FEW_BLOCKS blocks an SM go one piece per lane instead.  INT8,
// many -> few, groups of 64: 1000 4.5 -> 2.6 us, 60000 6.1 -> 5.1 us; of 128: 1000 4.2 -> 2.2 us, 60000 (just under the line)
// 8.6 -> 7.8 us, 100000 11.1 -> 11.5 us; FP8 of 128: 60000 10.4 -> 8.4 us.
constexpr int QUANT_FEW_BLOCKS = 4;
constexpr long long quant_groups_per_block(int w, int ch, bool few) { return 8 * (32 / w) * quant_batches(ch, few); }

template <int MODE, int W, int CH, bool FEW = false>
static void launch_quantize_w(const bf16* x, uint8_t* q, float* scale, float* zero, bf16* y, long long groups, int g,
                              cudaStream_t s) {
  const int grid = quant_grid(groups, int(quant_groups_per_block(W, CH, FEW)));
  if (y != nullptr) quantize_kernel<MODE, true, W, CH, FEW><<<grid, 256, 0, s>>>(x, q, scale, zero, y, groups, g);
  else quantize_kernel<MODE, false, W, CH, FEW><<<grid, 256, 0, s>>>(x, q, scale, zero, y, groups, g);
}
template <int MODE>
static void launch_quantize_m(const bf16* x, uint8_t* q, float* scale, float* zero, bf16* y, long long groups, int g,
                              cudaStream_t s) {
  const int chunks = g >> 3;
  const long long line = (long long)QUANT_FEW_BLOCKS * gemm_num_sms();
  auto few = [&](int w, int ch) { return groups <= line * quant_groups_per_block(w, ch, false); };
  if (chunks <= 4) {
    if (few(4, 1)) launch_quantize_w<MODE, 4, 1, true>(x, q, scale, zero, y, groups, g, s);
    else launch_quantize_w<MODE, 4, 1>(x, q, scale, zero, y, groups, g, s);
  } else if (chunks <= 8) {
    if (few(4, 2)) launch_quantize_w<MODE, 8, 1, true>(x, q, scale, zero, y, groups, g, s);
    else launch_quantize_w<MODE, 4, 2>(x, q, scale, zero, y, groups, g, s);
  } else if (chunks <= 16) {
    if (few(8, 2)) launch_quantize_w<MODE, 16, 1, true>(x, q, scale, zero, y, groups, g, s);
    else launch_quantize_w<MODE, 8, 2>(x, q, scale, zero, y, groups, g, s);
  } else if (chunks <= 32) {
    if (few(16, 2)) launch_quantize_w<MODE, 32, 1, true>(x, q, scale, zero, y, groups, g, s);
    else launch_quantize_w<MODE, 16, 2>(x, q, scale, zero, y, groups, g, s);
  } else {
    launch_quantize_w<MODE, 32, QMAX_CHUNKS>(x, q, scale, zero, y, groups, g, s);
  }
}

void launch_quantize(const void* x, void* q, float* scale, float* zero, void* y_fake, long long groups, int g,
                     int mode, cudaStream_t s) {
  if (groups == 0) return;
  if (g % 8 != 0 || g > 32 * QMAX_CHUNKS * 8) throw std::runtime_error("quantize: group size must be a multiple of 8, at most 1024");
  const bf16* xi = (const bf16*)x;
  uint8_t* qo = (uint8_t*)q;
  bf16* yo = (bf16*)y_fake;
  switch (mode) {
    case QUANT_INT8: launch_quantize_m<QUANT_INT8>(xi, qo, scale, zero, yo, groups, g, s); break;
    case QUANT_INT8_ASYM: launch_quantize_m<QUANT_INT8_ASYM>(xi, qo, scale, zero, yo, groups, g, s); break;
    case QUANT_INT4: launch_quantize_m<QUANT_INT4>(xi, qo, scale, zero, yo, groups, g, s); break;
    case QUANT_NF4: launch_quantize_m<QUANT_NF4>(xi, qo, scale, zero, yo, groups, g, s); break;
    case QUANT_FP8_E4M3: launch_quantize_m<QUANT_FP8_E4M3>(xi, qo, scale, zero, yo, groups, g, s); break;
    case QUANT_FP8_E5M2: launch_quantize_m<QUANT_FP8_E5M2>(xi, qo, scale, zero, yo, groups, g, s); break;
    default: throw std::runtime_error("quantize: unknown mode");
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("quantize launch: ") + cudaGetErrorString(e));
}

void launch_dequantize(const void* q, const float* scale, const float* zero, void* y, long long groups, int g,
                       int mode, cudaStream_t s) {
  if (groups == 0) return;
  if (g % 8 != 0) throw std::runtime_error("dequantize: group size must be a multiple of 8");
  const uint8_t* qi = (const uint8_t*)q;
  bf16* yo = (bf16*)y;
  const int grid = quant_grid(groups * (g >> 3), 256);
  switch (mode) {
    case QUANT_INT8: dequantize_kernel<QUANT_INT8><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    case QUANT_INT8_ASYM: dequantize_kernel<QUANT_INT8_ASYM><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    case QUANT_INT4: dequantize_kernel<QUANT_INT4><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    case QUANT_NF4: dequantize_kernel<QUANT_NF4><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    case QUANT_FP8_E4M3: dequantize_kernel<QUANT_FP8_E4M3><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    case QUANT_FP8_E5M2: dequantize_kernel<QUANT_FP8_E5M2><<<grid, 256, 0, s>>>(qi, scale, zero, yo, groups, g); break;
    default: throw std::runtime_error("dequantize: unknown mode");
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("dequantize launch: ") + cudaGetErrorString(e));
}

}  // namespace fc

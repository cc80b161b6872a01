// Dense (non-causal) attention on tcgen05 for the vision towers and the resampler: head_dim up to 128.
//
// out[b, s, h, :] = softmax(q[b, s, h, :] . k[b, :, h, :]^T * scale  (+ key mask)) v[b, :, h, :]
//
// One CTA owns 128 query rows of one head of one batch element and walks the keys in tiles of 128 rows; two CTAs share an
// SM (256 columns of tensor memory and at most 98 KB of shared memory each), so one tile's products run under the
// other's softmax, and 128-row units leave less of the last wave empty than pairs of them.  S, P and O live in tensor
// memory:  S [0, 128), then P as packed bf16 over its first 64 columns;  O [128, 128 + DP)
//   warp 0       TMA: the Q tile once, then K and V tiles (128-byte swizzle; two stages each for DP = 64, one for
//                DP = 128, where the copy of the next tile has the whole softmax to arrive)
//   warp 1       tcgen05.mma issuer: S = Q K^T from shared memory, O += P V with P read from tensor memory and V as an
//                MN-major operand
//   warps 2-5    softmax, one query row per thread, O rescaled lazily
//
// What bounds it: MUFU (one exp2 per score, 1024 clocks per tile and SM) and, above that, the chain S -> softmax -> P -> PV
// -> next S of a tile, of which an SM has two.  5 x 961 rows, 16 heads of 72, ragged key mask: 80 us with two query tiles
// per CTA, one CTA per SM (320 CTAs on 148 SMs) and the mask padded by two launches of its own, 69 us so.  15 x 577 rows,
// 16 heads of 64: 63 us both ways.  Two threads per row, 64 columns each, were slower (69 us, 73 us): they have to
// meet for the maximum of a row.
//
// The operands are [B, S, H, D] views with arbitrary strides (the packed qkv output of one GEMM is read in place),
// described to TMA as 4-D tensors (D, H, S, B).  The head dimension is padded to DP = 64 or 128 columns by the
// copy itself: elements past D, and rows past S, are outside the tensor and arrive as zeros, so head_dim 72
// (SigLIP) runs as 128 with zero columns that add nothing to S and produce O columns that are not written.
// The box starts at x = 0 or 64 elements, i.e. on 16-byte boundaries.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cfloat>
#include <mutex>
#include <stdexcept>
#include <string>

#include "gemm.h"
#include "kernels.h"
#include "ptx.cuh"

namespace fc {

using bf16 = __nv_bfloat16;

constexpr int DT_BM = 128;             // query rows per CTA
constexpr int DT_BN = 128;
constexpr int DT_THREADS = 192;
constexpr int DT_SUB_BYTES = 128 * 64 * 2;              // one [128 x 64] sub-tile
constexpr float DT_RESCALE_THRESHOLD = 8.f;             // log2 units
// reference of a row's exponents until its first key comes: every score that counts is above it and rescales by 2^-inf = 0
// the zeros that are there so far
constexpr float DT_NO_KEY = -FLT_MAX;

__device__ __forceinline__ uint64_t dt_sdesc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((addr & 0x3FFFF) >> 4);
  d |= uint64_t((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}

__device__ __forceinline__ float dt_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ void dt_tma_load_4d(void* smem, const CUtensorMap* m, uint64_t* bar, int x, int y, int z,
                                               int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

struct DenseTcParams {
  bf16* out;                 // [B, Sq, H, D] contiguous
  const uint8_t* key_mask;   // [B, Sk] (0 = do not attend), or null
  int Sq, Sk, H, D;
  float scale_log2;
  uint32_t* status;
};

template <int DP>
struct DtSmem {
  static constexpr int TILE_BYTES = DP / 64 * DT_SUB_BYTES;
  static constexpr int STAGES = DP == 64 ? 2 : 1;                       // of K and of V
  static constexpr int BAR_OFF = (1 + 2 * STAGES) * TILE_BYTES;
  static constexpr int TOTAL = BAR_OFF + 128 + 1024;
};

template <int DP>
__global__ void __launch_bounds__(DT_THREADS, 2)
dense_attn_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const DenseTcParams p) {
  using L = DtSmem<DP>;
  constexpr int TILE_BYTES = L::TILE_BYTES, STAGES = L::STAGES;
  constexpr uint32_t O_BASE = 128u;                    // first column of O
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_q = smem;
  uint8_t* s_k = s_q + TILE_BYTES;
  uint8_t* s_v = s_k + STAGES * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* q_full = bars;            // [1]
  uint64_t* k_full = bars + 1;        // [2]
  uint64_t* k_empty = bars + 3;       // [2]
  uint64_t* v_full = bars + 5;        // [2]
  uint64_t* v_empty = bars + 7;       // [2]
  uint64_t* s_full = bars + 9;        // [1]
  uint64_t* p_ready = bars + 10;      // [1] (128 arrivals)
  uint64_t* o_done = bars + 11;       // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int q0 = blockIdx.x * DT_BM;
  const int n_tiles = (p.Sk + DT_BN - 1) / DT_BN;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(p_ready, 128);
    mbar_init(o_done, 1);
    *s_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loader
    if (lane == 0) {
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* full, int row) {
        mbar_expect_tx(full, TILE_BYTES);             // rows and columns outside the tensor count as copied zeros
        for (int sub = 0; sub < DP / 64; ++sub)
          dt_tma_load_4d(dst + sub * DT_SUB_BYTES, tm, full, sub * 64, h, row, b);
      };
      load(s_q, &tm_q, q_full, q0);
      int nk = 0, nv = 0;
      for (int j = 0; j < n_tiles; ++j) {
        const int st = j % STAGES;
        const uint32_t ph = ((j / STAGES) & 1) ^ 1;
        if (*s_abort || !mbar_wait(&k_empty[st], ph, p.status, ST_TIMEOUT_EMPTY)) break;
        load(s_k + st * TILE_BYTES, &tm_k, &k_full[st], j * DT_BN);
        ++nk;
        if (*s_abort || !mbar_wait(&v_empty[st], ph, p.status, ST_TIMEOUT_EMPTY)) break;
        load(s_v + st * TILE_BYTES, &tm_v, &v_full[st], j * DT_BN);
        ++nv;
      }
      if (nv < n_tiles) {
        // unwind: what was asked for lands before the CTA may exit
        *s_abort = 1;
        mbar_wait(q_full, 0, nullptr, 0);
        for (int j = max(0, nk - STAGES); j < nk; ++j) mbar_wait(&k_full[j % STAGES], (j / STAGES) & 1, nullptr, 0);
        for (int j = max(0, nv - STAGES); j < nv; ++j) mbar_wait(&v_full[j % STAGES], (j / STAGES) & 1, nullptr, 0);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      // B (= V) is MN-major; of the DP columns that the copy pads to, only the 16-column groups that hold some of D
      const int d16 = (p.D + 15) / 16;
      const uint32_t idesc_o = make_idesc_bf16(128, d16 * 16, false, true);
      const uint32_t qa = smem_u32(s_q);
      bool ok = mbar_wait(q_full, 0, p.status, ST_TIMEOUT_FULL);
      auto issue_s = [&](int j) {
        const int st = j % STAGES;
        if (!mbar_wait(&k_full[st], (j / STAGES) & 1, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        const uint32_t ka = smem_u32(s_k + st * TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < DP / 16; ++kk) {
          const uint32_t off = uint32_t(kk >> 2) * DT_SUB_BYTES + uint32_t(kk & 3) * 32;
          if (kk < d16)
            tc_mma_f16(tmem_base, dt_sdesc(qa + off, 16, 1024), dt_sdesc(ka + off, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
        }
        tc_commit(s_full);
        tc_commit(&k_empty[st]);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j % STAGES;
        ok = mbar_wait(p_ready, uint32_t(j) & 1u, p.status, ST_TIMEOUT_FULL) &&
             mbar_wait(&v_full[st], uint32_t(j / STAGES) & 1u, p.status, ST_TIMEOUT_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t va = smem_u32(s_v + st * TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t db = dt_sdesc(va + uint32_t(kk) * 2048, DT_SUB_BYTES, 1024);
          tc_mma_f16_ts(tmem_base + O_BASE, tmem_base + uint32_t(kk * 8), db, idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
        }
        tc_commit(o_done);
        tc_commit(&v_empty[st]);
        if (j + 1 < n_tiles) ok = issue_s(j + 1);      // after PV(j), whose P lies where S(j + 1) goes
      }
      if (!ok) *s_abort = 1;
    }
  } else {
    // ------------------------------------------------ softmax, one query row per thread
    const int lane_group = warp & 3;                         // TMEM lanes this warp may touch
    const int row = lane_group * 32 + lane;
    const uint32_t lane_addr = uint32_t(lane_group * 32) << 16;
    const uint32_t ts = tmem_base + lane_addr;               // S, then P
    const uint32_t to = tmem_base + lane_addr + O_BASE;      // O
    const int qrow = q0 + row;
    const uint8_t* mrow = p.key_mask != nullptr ? p.key_mask + (long long)b * p.Sk : nullptr;
    float m_ref = 0.f, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles && ok; ++j) {
      // keys that are not there or not attended to, looked up before the wait for S: lane t asks for key 32 c + t, all
      // lanes get the 32 answers
      const int col0 = j * DT_BN;
      const bool some = mrow != nullptr || col0 + DT_BN > p.Sk;
      uint32_t seen[4];
      if (some) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int key = col0 + c * 32 + lane;
          seen[c] = __ballot_sync(0xffffffffu, key < p.Sk && (mrow == nullptr || mrow[key] != 0));
        }
      }
      ok = __all_sync(0xffffffffu, !*s_abort && mbar_wait(s_full, uint32_t(j) & 1u, p.status, ST_TIMEOUT_ACC_FULL));
      if (!ok) break;
      tc_fence_after();
      uint32_t s[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(ts + uint32_t(c * 32), *reinterpret_cast<uint32_t(*)[32]>(&s[c * 32]));
      tmem_ld_wait();
      if (some) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (seen[c] != 0xffffffffu) {
#pragma unroll
            for (int t = 0; t < 32; ++t)
              if (((seen[c] >> t) & 1u) == 0u) s[c * 32 + t] = 0xff800000u;      // -inf
          }
        }
      }
      // four independent chains each (a single one is 128 dependent operations per tile)
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int t = 0; t < 128; t += 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mx4[i] = dt_max3(mx4[i], __uint_as_float(s[t + 2 * i]), __uint_as_float(s[t + 2 * i + 1]));
      }
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      mx *= p.scale_log2;
      if (j == 0) {
        m_ref = fmaxf(mx, DT_NO_KEY);
      } else if (__any_sync(0xffffffffu, mx > m_ref + DT_RESCALE_THRESHOLD)) {
        // some row of this warp outgrew its reference: bring O (complete up to tile j - 1) to the new one
        if (!__all_sync(0xffffffffu, mbar_wait(o_done, uint32_t(j - 1) & 1u, p.status, ST_TIMEOUT_ACC_FULL))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const float m_new = fmaxf(m_ref, mx);
        const float f = exp2f(m_ref - m_new);
        m_ref = m_new;
        l *= f;
#pragma unroll 1
        for (int c = 0; c < DP / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(to + uint32_t(c * 32), r);
          tmem_ld_wait();
#pragma unroll
          for (int t = 0; t < 32; ++t) r[t] = __float_as_uint(__uint_as_float(r[t]) * f);
          tmem_st_32x32(to + uint32_t(c * 32), r);
        }
        tmem_st_wait();
      }
      float rs4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t u[64];
#pragma unroll
      for (int t = 0; t < 64; ++t) {
        float e0, e1;
        const float a0 = fmaf(__uint_as_float(s[2 * t]), p.scale_log2, -m_ref);
        const float a1 = fmaf(__uint_as_float(s[2 * t + 1]), p.scale_log2, -m_ref);
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(a0));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(a1));
        rs4[t & 3] += e0 + e1;
        u[t] = pack_bf16(e0, e1);
      }
      const float rs = (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
      tmem_st_32x32(ts, *reinterpret_cast<uint32_t(*)[32]>(&u[0]));
      tmem_st_32x32(ts + 32u, *reinterpret_cast<uint32_t(*)[32]>(&u[32]));
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_ready);
      l += rs;
    }
    if (!ok) *s_abort = 1;
    if (ok && __all_sync(0xffffffffu, mbar_wait(o_done, uint32_t(n_tiles - 1) & 1u, p.status, ST_TIMEOUT_ACC_FULL))) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* dst = p.out + (((long long)b * p.Sq + qrow) * p.H + h) * p.D;
#pragma unroll 1
      for (int c = 0; c < DP / 32; ++c) {
        if (c * 32 >= p.D) break;                       // uniform over the warp
        __syncwarp();                                   // a tensor-memory load is a warp instruction
        uint32_t r[32];
        tmem_ld_32x32(to + uint32_t(c * 32), r);
        tmem_ld_wait();
        if (qrow < p.Sq) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (c * 32 + q * 8 < p.D) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[q * 8 + 0]) * inv, __uint_as_float(r[q * 8 + 1]) * inv);
              v.y = pack_bf16(__uint_as_float(r[q * 8 + 2]) * inv, __uint_as_float(r[q * 8 + 3]) * inv);
              v.z = pack_bf16(__uint_as_float(r[q * 8 + 4]) * inv, __uint_as_float(r[q * 8 + 5]) * inv);
              v.w = pack_bf16(__uint_as_float(r[q * 8 + 6]) * inv, __uint_as_float(r[q * 8 + 7]) * inv);
              reinterpret_cast<uint4*>(dst + c * 32)[q] = v;
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// 4-D bf16 view (D, H, S, B) of a [B, S, H, D] tensor with element strides (sb, ss, sh, 1); box = 64 x 1 x 128 x 1
static CUtensorMap dt_tmap(const void* base, int B, int S, int H, int D, const long long* strides) {
  typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || ptr == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  CUtensorMap m;
  cuuint64_t dims[4] = {cuuint64_t(D), cuuint64_t(H), cuuint64_t(S), cuuint64_t(B)};
  cuuint64_t str[3] = {cuuint64_t(strides[2]) * 2, cuuint64_t(strides[1]) * 2, cuuint64_t(strides[0]) * 2};
  cuuint32_t box[4] = {64, 1, 128, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, str, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw std::runtime_error("dense attention: cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return m;
}

bool dense_attention_tc_supported(int B, int Sq, int Sk, int H, int D, const long long* q_strides,
                                  const long long* k_strides, const long long* v_strides) {
  if (D % 8 != 0 || D > 128 || D < 8 || Sk < 1 || Sq < 1) return false;
  for (const long long* s : {q_strides, k_strides, v_strides}) {
    // TMA wants strides that are positive multiples of 16 bytes (an expanded view has 0), each a multiple of the
    // one below it; a dimension of extent 1 gets a stride of its own at launch
    const long long sb = s[0], ss = s[1], sh = s[2];
    if (ss <= 0 || ss % 8 != 0) return false;
    if (H > 1 && (sh <= 0 || sh % 8 != 0 || sh < D || ss % sh != 0 || ss < sh * H)) return false;
    if (H == 1 && ss < D) return false;
    if (B > 1 && (sb <= 0 || sb % ss != 0)) return false;
  }
  return true;
}

template <int DP>
static void dt_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const DenseTcParams& p,
                      dim3 grid, cudaStream_t stream) {
  constexpr int smem = DtSmem<DP>::TOTAL;
  auto kern = dense_attn_tc_kernel<DP>;
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load(std::memory_order_relaxed) & bit)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) throw std::runtime_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    configured.fetch_or(bit, std::memory_order_relaxed);
  }
  kern<<<grid, DT_THREADS, smem, stream>>>(tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("dense attention (tcgen05) launch: ") + cudaGetErrorString(e));
}

void launch_dense_attention_tc(const void* q, const void* k, const void* v, void* out, const uint8_t* key_mask,
                               int B, int Sq, int Sk, int H, int D, const long long* q_strides,
                               const long long* k_strides, const long long* v_strides, float scale,
                               uint32_t* status, cudaStream_t stream) {
  if (B == 0 || Sq == 0) return;
  if (!dense_attention_tc_supported(B, Sq, Sk, H, D, q_strides, k_strides, v_strides))
    throw std::runtime_error("dense attention (tcgen05): unsupported shape or strides");
  // a dimension of extent 1 may carry any stride in the view; give TMA the one of a packed tensor
  auto fix = [&](const long long* s, int rows, long long* o) {
    o[1] = s[1];
    o[2] = H > 1 ? s[2] : D;
    o[0] = B > 1 ? s[0] : s[1] * rows;
  };
  long long qs[3], ks[3], vs[3];
  fix(q_strides, Sq, qs);
  fix(k_strides, Sk, ks);
  fix(v_strides, Sk, vs);
  DenseTcParams p{};
  p.out = reinterpret_cast<bf16*>(out);
  p.key_mask = key_mask;
  p.Sq = Sq;
  p.Sk = Sk;
  p.H = H;
  p.D = D;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  const CUtensorMap tq = dt_tmap(q, B, Sq, H, D, qs);
  const CUtensorMap tk = dt_tmap(k, B, Sk, H, D, ks);
  const CUtensorMap tv = dt_tmap(v, B, Sk, H, D, vs);
  const dim3 grid((Sq + DT_BM - 1) / DT_BM, H, B);
  if (D <= 64) dt_launch<64>(tq, tk, tv, p, grid, stream);
  else dt_launch<128>(tq, tk, tv, p, grid, stream);
}

}  // namespace fc

// Fused CCM merge compressor operating in the paged KV pool (head_dim 128).
//
// For one (request, group of G kv heads, layer, K|V) a CTA walks the request's rows in
// ascending order, segment by segment (image rows first, then text rows, each with its own
// MLP bank): f consecutive rows of a head are concatenated (they are adjacent in the
// head-major pool, so the "concatenation" is only an addressing rule), pushed through
//        y = W3 relu(W2 relu(W1 z + b1) + b2) + b3
// and written to the leading rows of the same request; the (rows mod f) remainder of a
// segment is moved unchanged.  A tile is 128 output rows: 128 / G consecutive output rows of
// each of the G heads (the MLP weights are shared by all heads, so short segments still fill
// the 128-row tensor-core tile; the host picks G from the segment lengths).
//
//   warps 6-9  gather the A operand of GEMM1 k-block by k-block with cp.async into the 128-byte-swizzled layout
//              tcgen05 expects (a ring of four k-blocks that runs on from tile to tile)
//   warp 0     streams W1 / W2 / W3 k-blocks with TMA into a ring of three
//   warp 1     issues tcgen05.mma: GEMM1 over f*2 k-blocks (A gathered), GEMM2 and GEMM3 with the activation tile
//              as the A operand FROM TENSOR MEMORY
//   warps 2-5  epilogues: tcgen05.ld, bias, ReLU, bf16; the activation tile goes back over the accumulator it came
//              from as packed bf16 (tcgen05.st), the result rows are scattered to the pool
// The intermediates never leave the SM.  112 KB of shared memory and 256 TMEM columns: two CTAs share an SM.
//
// What bounds it: rows are read once and a quarter (1 / f) of them written; the floor is that traffic.  A tile is a
// dependent chain (gather -> GEMM1 -> epilogue -> GEMM2 -> epilogue -> GEMM3 -> scatter), so the copies of the next tile
// have to be in flight while it runs: gathering warps of their own do that (with the epilogue's threads gathering,
// an SM had no read outstanding for most of a tile), and the activation tile in tensor memory is what pays for the
// deeper ring.  LLaVA-1.5 shape, 15 requests of 576 + 64 rows, 32 layers x 32 heads,
// factor 4 (6.3 GB), the kernel alone: 4.11 ms with the epilogue's threads gathering into three shared stages, 1.97 ms so, with
// the first GEMM of a tile under the scatter of the one before and a full ring announced at once (0.49 of the copy rate; a call
// from the host with its tables takes 2.2 ms).
// In-place safety: an output row index never exceeds the index of any input row of the same head it depends on, tiles
// are processed in ascending order by one CTA, and a tile is read completely (GEMM1 is done) before it is written.
// What the gathering warps read ahead lies behind every row that is still to be written for an earlier tile.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <stdexcept>
#include <string>

#include "gemm.h"
#include "kernels.h"
#include "mma.cuh"
#include "ptx.cuh"

namespace fc {

using bf16 = __nv_bfloat16;

constexpr int CCM_D = 128;
constexpr int CCM_A_STAGES = 4;        // gathered k-blocks
constexpr int CCM_W_STAGES = 3;        // weight k-blocks
constexpr int CCM_THREADS = 320;
constexpr int CCM_TILE = 128;          // output rows per tile
constexpr int CCM_KB_BYTES = CCM_TILE * 64 * 2;   // one [128 x 64] bf16 sub-tile

struct CcmParams {
  bf16* pool;                 // [L, 2, num_blocks, Hkv, block_size, D]
  const int* block_tables;    // [n_seq, max_blocks]
  const int* dst_tables;      // [n_seq, max_blocks] blocks the result is written to, or nullptr: in place
  const int* kv_lens;         // [n_seq]
  const int* image_lens;      // [n_seq]
  const bf16 *b1, *b2, *b3;   // [Lw, 4, D]
  int num_blocks, Hkv, block_size, max_blocks;
  int layer_start;            // first pool layer handled by blockIdx.y / 2 == 0
  int weight_layer_start;     // index of that layer in the packed weights
  int factor, min_seq_len;
  int single_segment;
  int heads_per_cta;          // G: 1, 2, 4 or 8 heads share a tile
  int rj_shift;               // log2(128 / G): output rows of one head per tile
  uint32_t* status;
};

__device__ __forceinline__ int ccm_seg_out(int n, int f, int min_len) {
  if (n <= 0) return 0;
  const int s = n / f;
  return s < min_len ? n : s + n % f;
}

__global__ void __launch_bounds__(CCM_THREADS, 2)
ccm_fused_kernel(const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_w2,
                 const __grid_constant__ CUtensorMap tm_w3, const CcmParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_w = smem + CCM_A_STAGES * CCM_KB_BYTES;
  uint64_t* a_full = reinterpret_cast<uint64_t*>(s_w + CCM_W_STAGES * CCM_KB_BYTES);
  uint64_t* a_empty = a_full + CCM_A_STAGES;
  uint64_t* w_full = a_empty + CCM_A_STAGES;
  uint64_t* w_empty = w_full + CCM_W_STAGES;
  uint64_t* acc_full = w_empty + CCM_W_STAGES;  // [2]: GEMM1; GEMM2 and GEMM3 in turn
  uint64_t* h_ready = acc_full + 2;             // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(h_ready + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.heads_per_cta, rj_shift = p.rj_shift, RJ = 1 << rj_shift;
  const int h0 = blockIdx.x * G, seq = blockIdx.z;
  const int layer_off = blockIdx.y >> 1, kv = blockIdx.y & 1;
  const int layer = p.layer_start + layer_off, wlayer = p.weight_layer_start + layer_off;
  const int f = p.factor;
  const int nk1 = f * (CCM_D / 64);             // k-blocks of GEMM1
  const int nk_tile = nk1 + 4;                  // + 2 for W2 + 2 for W3

  if (threadIdx.x == 0) {
    for (int s = 0; s < CCM_A_STAGES; ++s) {
      mbar_init(&a_full[s], 128);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < CCM_W_STAGES; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
    }
    mbar_init(&acc_full[0], 1);
    mbar_init(&acc_full[1], 1);
    mbar_init(h_ready, 128);
    *s_abort = (smem_u32(smem) & 1023u) != 0u;  // the swizzled tiles need 1024-byte alignment: nothing runs without it
    if (*s_abort) report(p.status, ST_BAD_INDEX);
    fence_barrier_init();
    tma_prefetch_desc(&tm_w1);
    tma_prefetch_desc(&tm_w2);
    tma_prefetch_desc(&tm_w3);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // ---- the request's segments (identical arithmetic in every role)
  const int S = p.kv_lens[seq];
  int img = p.single_segment ? 0 : p.image_lens[seq];
  img = max(0, min(img, S));
  const int seg_in[2] = {0, img};
  const int seg_len[2] = {img, S - img};
  const int seg_out[2] = {0, ccm_seg_out(img, f, p.min_seq_len)};
  int seg_tiles[2];
  for (int s = 0; s < 2; ++s) {
    const int sp = seg_len[s] / f;
    seg_tiles[s] = (seg_len[s] > 0 && sp >= p.min_seq_len) ? (sp + RJ - 1) >> rj_shift : 0;
  }
  const int total_tiles = *s_abort ? 0 : seg_tiles[0] + seg_tiles[1];

  const int* bt = p.block_tables + (long long)seq * p.max_blocks;
  const long long plane = (((long long)layer * 2 + kv) * p.num_blocks);
  auto row_ptr = [&](int hh, int tok) -> bf16* {
    int blk = bt[tok / p.block_size];
    if (blk < 0 || blk >= p.num_blocks) {
      report(p.status, ST_BAD_INDEX);
      return nullptr;
    }
    return p.pool + (((plane + blk) * p.Hkv + hh) * p.block_size + tok % p.block_size) * CCM_D;
  };
  // destination rows: the request's own blocks (in place), or a second set of blocks, in which case the
  // source rows stay intact and the request can keep decoding over them while its layers are compressed
  const bool out_of_place = p.dst_tables != nullptr;
  const int* dbt = out_of_place ? p.dst_tables + (long long)seq * p.max_blocks : bt;
  auto dst_ptr = [&](int hh, int tok) -> bf16* {
    int blk = dbt[tok / p.block_size];
    if (blk < 0 || blk >= p.num_blocks) {
      report(p.status, ST_BAD_INDEX);
      return nullptr;
    }
    return p.pool + (((plane + blk) * p.Hkv + hh) * p.block_size + tok % p.block_size) * CCM_D;
  };

  if (warp == 0) {
    // ------------------------------------------------------------- weight producer (TMA)
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int tile = 0; tile < total_tiles && ok; ++tile) {
        const int seg = tile < seg_tiles[0] ? 0 : 1;
        const int bank = (seg == 0 ? 2 : 0) + kv;             // (tk, tv, ik, iv)
        const int wrow = (wlayer * 4 + bank) * CCM_D;
        for (int i = 0; i < nk_tile; ++i, ++it) {
          const int stage = it % CCM_W_STAGES;
          if (*s_abort || !mbar_wait(&w_empty[stage], ((it / CCM_W_STAGES) & 1) ^ 1, p.status, ST_TIMEOUT_EMPTY)) {
            *s_abort = 1;
            ok = false;
            break;
          }
          uint8_t* sw = s_w + stage * CCM_KB_BYTES;
          mbar_expect_tx(&w_full[stage], CCM_KB_BYTES);
          if (i < nk1) tma_load_2d(sw, &tm_w1, &w_full[stage], i * 64, wrow);
          else if (i < nk1 + 2) tma_load_2d(sw, &tm_w2, &w_full[stage], (i - nk1) * 64, wrow);
          else tma_load_2d(sw, &tm_w3, &w_full[stage], (i - nk1 - 2) * 64, wrow);
        }
      }
      // unwind: copies that are in flight land before the CTA may exit
      if (!ok)
        for (int n = max(0, it - CCM_W_STAGES); n < it; ++n)
          mbar_wait(&w_full[n % CCM_W_STAGES], (n / CCM_W_STAGES) & 1, nullptr, 0);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------------- MMA issuer
    // accumulators: GEMM1 in columns [0, 128), GEMM2 and GEMM3 in [128, 256).  Both activation tiles are packed into
    // [0, 64), so GEMM1 of the next tile may start as soon as GEMM3 is through and runs while this tile's rows are
    // scattered.  Products are executed in the order they are issued; h_ready of the next tile says that the second
    // accumulator has been read.
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, 128);
      int ia = 0, iw = 0;
      uint32_t h_phase = 0;
      bool ok = true;
      for (int tile = 0; tile < total_tiles && ok; ++tile) {
        for (int g = 0; g < 3 && ok; ++g) {
          const int nk = g == 0 ? nk1 : 2;
          const uint32_t d_tmem = tmem_base + (g == 0 ? 0u : 128u);
          if (g > 0) {
            ok = mbar_wait(h_ready, h_phase, p.status, ST_TIMEOUT_ACC_FULL);
            h_phase ^= 1;
            if (!ok) break;
            tc_fence_after();
          }
          for (int i = 0; i < nk && ok; ++i, ++iw) {
            const int ws = iw % CCM_W_STAGES, as = ia % CCM_A_STAGES;
            ok = mbar_wait(&w_full[ws], (iw / CCM_W_STAGES) & 1, p.status, ST_TIMEOUT_FULL);
            if (ok && g == 0) ok = mbar_wait(&a_full[as], (ia / CCM_A_STAGES) & 1, p.status, ST_TIMEOUT_FULL);
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = make_sdesc_sw128(smem_u32(s_w + ws * CCM_KB_BYTES));
            if (g == 0) {
              const uint64_t da = make_sdesc_sw128(smem_u32(smem + as * CCM_KB_BYTES));
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tc_mma_f16(d_tmem, da + uint64_t(2 * k), db + uint64_t(2 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
              tc_commit(&a_empty[as]);
              ++ia;
            } else {
              const uint32_t a_tmem = tmem_base + uint32_t(i * 32);   // 64 values of K, two to a column
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tc_mma_f16_ts(d_tmem, a_tmem + uint32_t(8 * k), db + uint64_t(2 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit(&w_empty[ws]);
          }
          if (ok) tc_commit(&acc_full[g == 0 ? 0 : 1]);
        }
      }
      if (!ok) *s_abort = 1;
    }
  } else if (warp >= 6) {
    // ---------------------------------------------------------------------- gather of GEMM1's A operand
    // Thread gt copies 16-byte piece gt & 7 of rows (gt >> 3) + 16 q of every k-block; the eight threads of a row look up
    // one row each, a row of the group ahead, and pass it on.  A stage is handed to the MMA warp when its copies have
    // landed: while stages are free CCM_A_STAGES - 1 k-blocks later, and all of them when the ring is full, so that the
    // next tile's first k-blocks are announced before they are wanted.
    const int gt = threadIdx.x - 192;              // 0..127
    const int ch = gt & 7, r0 = gt >> 3;
    const uint32_t s_dst = smem_u32(smem) + r0 * 128 + ((ch ^ (r0 & 7)) << 4);     // (16 q keeps the low bits of the row)
    constexpr uint32_t NO_ROW = 0xffffffffu;
    const bf16* base = p.pool + ch * 8;
    const int my_r = r0 + 16 * ch;                 // the tile row this thread looks up: head my_r >> rj_shift
    auto lookup = [&](int tile, int tok) -> uint32_t {       // pool row (block rows of all planes counted through)
      const int seg = tile < seg_tiles[0] ? 0 : 1;
      const int j = ((seg == 0 ? tile : tile - seg_tiles[0]) << rj_shift) + (my_r & (RJ - 1));
      if (j >= seg_len[seg] / f) return NO_ROW;
      const int t = seg_in[seg] + j * f + tok;
      const int blk = bt[t / p.block_size];
      if (blk < 0 || blk >= p.num_blocks) {
        report(p.status, ST_BAD_INDEX);
        return NO_ROW;
      }
      return uint32_t(((plane + blk) * p.Hkv + h0 + (my_r >> rj_shift)) * p.block_size + t % p.block_size);
    };
    int it = 0, told = 0;                          // k-blocks asked for, and announced
    bool ok = true;
    uint32_t next = total_tiles > 0 ? lookup(0, 0) : NO_ROW;
    for (int tile = 0; tile < total_tiles && ok; ++tile) {
      for (int tok = 0; tok < f && ok; ++tok) {
        uint32_t row[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) row[q] = __shfl_sync(0xffffffffu, next, q, 8);
        if (tok + 1 < f) next = lookup(tile, tok + 1);
        else if (tile + 1 < total_tiles) next = lookup(tile + 1, 0);
        for (int half = 0; half < CCM_D / 64; ++half, ++it) {
          const int stage = it % CCM_A_STAGES;
          const uint32_t ph = ((it / CCM_A_STAGES) & 1) ^ 1;
          if (!mbar_try_wait(&a_empty[stage], ph)) {
            cp_async_wait<0>();
            fence_proxy_async();
            for (; told < it; ++told) mbar_arrive(&a_full[told % CCM_A_STAGES]);
            if (*s_abort || !mbar_wait(&a_empty[stage], ph, p.status, ST_TIMEOUT_EMPTY)) {
              ok = false;
              break;
            }
          }
          const uint32_t sa = s_dst + stage * CCM_KB_BYTES;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const bool live = row[q] != NO_ROW;
            cp_async16(sa + q * 16 * 128, base + (live ? size_t(row[q]) * CCM_D + half * 64 : size_t(0)), live);
          }
          cp_async_commit();
          if (it - told >= CCM_A_STAGES - 1) {
            cp_async_wait<CCM_A_STAGES - 1>();
            fence_proxy_async();
            mbar_arrive(&a_full[told++ % CCM_A_STAGES]);
          }
        }
        // the shuffles above count on whole warps: a thread that gave up takes the others with it
        ok = __all_sync(0xffffffffu, ok);
      }
    }
    cp_async_wait<0>();
    if (ok) {
      fence_proxy_async();
      for (; told < it; ++told) mbar_arrive(&a_full[told % CCM_A_STAGES]);
    } else {
      *s_abort = 1;
    }
  } else {
    // ---------------------------------------------------------------------- epilogues, scatter, rows that only move
    const int wt = threadIdx.x - 64;               // 0..127
    const int lane_group = warp & 3;
    const int row = lane_group * 32 + lane;        // TMEM lane == tile row owned by this thread
    uint32_t tile_phase = 0;
    bool ok = !*s_abort;
    for (int seg = 0; seg < 2 && ok; ++seg) {
      const int n = seg_len[seg];
      if (n <= 0) continue;
      const int sp = n / f;
      const int in0 = seg_in[seg], out0 = seg_out[seg];
      if (seg_tiles[seg] == 0) {
        // too short to compress: move the rows unchanged (at most a few rows; out0 <= in0)
        if (out0 != in0 || out_of_place) {
          for (int hl = 0; hl < G; ++hl) {
            for (int base = 0; base < n; base += 8) {
              const int r = base + wt / 16, piece = wt % 16;
              uint4 v = make_uint4(0, 0, 0, 0);
              const bool live = r < n;
              if (live) {
                const bf16* src = row_ptr(h0 + hl, in0 + r);
                if (src != nullptr) v = reinterpret_cast<const uint4*>(src)[piece];
              }
              asm volatile("bar.sync 1, 128;" ::: "memory");
              if (live) {
                bf16* dst = dst_ptr(h0 + hl, out0 + r);
                if (dst != nullptr) reinterpret_cast<uint4*>(dst)[piece] = v;
              }
              asm volatile("bar.sync 1, 128;" ::: "memory");
            }
          }
        }
        continue;
      }
      const int bank = (seg == 0 ? 2 : 0) + kv;
      const bf16* b1 = p.b1 + ((long long)wlayer * 4 + bank) * CCM_D;
      const bf16* b2 = p.b2 + ((long long)wlayer * 4 + bank) * CCM_D;
      const bf16* b3 = p.b3 + ((long long)wlayer * 4 + bank) * CCM_D;
      for (int t = 0; t < seg_tiles[seg] && ok; ++t) {
        const int j0 = t << rj_shift;
        // ---- epilogues 1 and 2: bias + ReLU, activation tile as packed bf16 to columns [0, 64): over the accumulator of
        //      GEMM1 (a thread has read columns 0 ... 2 c + 31 of its row when it writes columns c ... c + 15), and over
        //      the first activation tile, which GEMM2 is done with
        for (int g = 0; g < 2 && ok; ++g) {
          if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[g], g == 0 ? tile_phase : 0u, p.status, ST_TIMEOUT_ACC_FULL))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const bf16* bias = g == 0 ? b1 : b2;
          const uint32_t h_addr = tmem_base + (uint32_t(lane_group * 32) << 16), t_addr = h_addr + (g == 1 ? 128u : 0u);
#pragma unroll 1
          for (int c4 = 0; c4 < 4; ++c4) {
            uint32_t rr[32];
            tmem_ld_32x32(t_addr + uint32_t(c4 * 32), rr);
            tmem_ld_wait();
            uint32_t u[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 bv = *reinterpret_cast<const uint4*>(bias + c4 * 32 + q * 8);
              const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                // a bf16 is the upper half of the fp32 with the same value
                const float a = fmaxf(__uint_as_float(rr[q * 8 + e * 2]) + __uint_as_float(bw[e] << 16), 0.f);
                const float b = fmaxf(__uint_as_float(rr[q * 8 + e * 2 + 1]) + __uint_as_float(bw[e] & 0xffff0000u), 0.f);
                u[q * 4 + e] = pack_bf16(a, b);
              }
            }
            tmem_st_32x16(h_addr + uint32_t(c4 * 16), u);
          }
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(h_ready);
        }
        if (!ok) break;
        // ---- epilogue 3: bias, bf16, scatter the rows of this tile
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[1], 1u, p.status, ST_TIMEOUT_ACC_FULL))) {
          ok = false;
          break;
        }
        tile_phase ^= 1;
        tc_fence_after();
        {
          const int j = j0 + (row & (RJ - 1));
          bf16* dst = (j < sp) ? dst_ptr(h0 + (row >> rj_shift), out0 + j) : nullptr;
          const uint32_t t_addr = tmem_base + (uint32_t(lane_group * 32) << 16) + 128u;
#pragma unroll 1
          for (int c4 = 0; c4 < 4; ++c4) {
            __syncwarp();                        // a tensor-memory load is a warp instruction
            uint32_t rr[32];
            tmem_ld_32x32(t_addr + uint32_t(c4 * 32), rr);
            tmem_ld_wait();
            if (dst != nullptr) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 bv = *reinterpret_cast<const uint4*>(b3 + c4 * 32 + q * 8);
                const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
                uint32_t u[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  u[e] = pack_bf16(__uint_as_float(rr[q * 8 + e * 2]) + __uint_as_float(bw[e] << 16),
                                   __uint_as_float(rr[q * 8 + e * 2 + 1]) + __uint_as_float(bw[e] & 0xffff0000u));
                }
                reinterpret_cast<uint4*>(dst)[c4 * 4 + q] = make_uint4(u[0], u[1], u[2], u[3]);
              }
            }
          }
        }
        tc_fence_before();                       // (h_ready of the next tile follows)
      }
      if (!ok) break;
      // ---- remainder rows of the segment move behind the compressed rows (fewer than f rows)
      const int rem = n - sp * f;
      if (rem > 0) {
        for (int hl = 0; hl < G; ++hl) {
          asm volatile("bar.sync 1, 128;" ::: "memory");
          const int r = wt / 16, piece = wt % 16;
          uint4 v = make_uint4(0, 0, 0, 0);
          const bool live = r < rem;
          if (live) {
            const bf16* src = row_ptr(h0 + hl, in0 + sp * f + r);
            if (src != nullptr) v = reinterpret_cast<const uint4*>(src)[piece];
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
          if (live) {
            bf16* dst = dst_ptr(h0 + hl, out0 + sp + r);
            if (dst != nullptr) reinterpret_cast<uint4*>(dst)[piece] = v;
          }
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      __threadfence_block();
    }
    if (!ok) *s_abort = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// Weights: w1 [Lw, 4, D, D*f], w2 / w3 [Lw, 4, D, D], biases [Lw, 4, D]; bf16, contiguous.
void launch_ccm_fused(void* pool, const int* block_tables, const int* kv_lens, const int* image_lens,
                      const void* w1, const void* w2, const void* w3, const void* b1, const void* b2,
                      const void* b3, int n_seq, int n_weight_layers, int layer_start, int layer_end,
                      int weight_layer_start, int num_blocks, int Hkv, int block_size, int D, int max_blocks,
                      int factor, int min_seq_len, int single_segment, int heads_per_cta, uint32_t* status,
                      cudaStream_t stream, const int* dst_block_tables) {
  if (n_seq == 0 || layer_end <= layer_start) return;
  int G = heads_per_cta <= 0 ? 1 : heads_per_cta;
  if ((G != 1 && G != 2 && G != 4 && G != 8) || Hkv % G != 0)
    throw std::runtime_error("fused CCM kernel: heads per CTA must be 1, 2, 4 or 8 and divide the KV heads");
  int rj_shift = 7;
  for (int g = G; g > 1; g >>= 1) --rj_shift;
  if (D != CCM_D) throw std::runtime_error("fused CCM kernel: head_dim must be 128");
  if (factor < 1 || factor > 8) throw std::runtime_error("fused CCM kernel: factor must be in [1, 8]");
  if ((unsigned long long)(layer_end * 2ll) * num_blocks * Hkv * block_size >= 0xffffffffull)
    throw std::runtime_error("fused CCM kernel: the pool has more rows than 32 bits count");
  CcmParams p{};
  p.pool = (bf16*)pool;
  p.block_tables = block_tables;
  p.dst_tables = dst_block_tables;
  p.kv_lens = kv_lens;
  p.image_lens = image_lens;
  p.b1 = (const bf16*)b1;
  p.b2 = (const bf16*)b2;
  p.b3 = (const bf16*)b3;
  p.num_blocks = num_blocks;
  p.Hkv = Hkv;
  p.block_size = block_size;
  p.max_blocks = max_blocks;
  p.layer_start = layer_start;
  p.weight_layer_start = weight_layer_start;
  p.factor = factor;
  p.min_seq_len = min_seq_len;
  p.single_segment = single_segment;
  p.heads_per_cta = G;
  p.rj_shift = rj_shift;
  p.status = status;
  const uint64_t wrows = (uint64_t)n_weight_layers * 4 * D;
  const CUtensorMap t1 = make_tmap_bf16_2d(w1, wrows, (uint64_t)D * factor, (uint64_t)D * factor, 128, 64);
  const CUtensorMap t2 = make_tmap_bf16_2d(w2, wrows, D, D, 128, 64);
  const CUtensorMap t3 = make_tmap_bf16_2d(w3, wrows, D, D, 128, 64);
  const int smem = (CCM_A_STAGES + CCM_W_STAGES) * CCM_KB_BYTES + 256;
  cudaFuncSetAttribute(ccm_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  dim3 grid(Hkv / G, (layer_end - layer_start) * 2, n_seq);
  ccm_fused_kernel<<<grid, CCM_THREADS, smem, stream>>>(t1, t2, t3, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("fused CCM launch: ") + cudaGetErrorString(e));
}

}  // namespace fc

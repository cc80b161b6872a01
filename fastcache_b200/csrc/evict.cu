// KV eviction in the paged pool: key-norm scoring, per-head top-k selection and
// stable in-place compaction.
//
// Pool layout [L, 2, num_blocks, Hkv, block_size, D] bf16 (rows of one head contiguous in a block).  Scores are fp32
// [n_seq, L, Hkv, s_stride], higher = keep (+inf = always keep).
//
// select_compact, two kernels.  `select_rows_kernel`: one CTA per (kv head, layer, request) turns the scores of the
// request into order-preserving 32-bit keys in shared memory, finds the k-th largest key with a 4-pass radix select and
// writes the kept rows (ties resolved toward later rows) in ascending order to `kept`.  `move_rows_kernel`: K and V
// and their 64-wide column ranges are separate CTAs (they share no byte), each moves its part of the kept rows to the
// front of the request's rows, 256 rows at a time.  A destination index never exceeds its source index, and a chunk
// is read completely into registers before it is written, so the compaction is safe in place.
// Bound by the copy of the kept rows.  Selection and moves in one kernel left 256 CTAs of 256 threads for 8 requests x 4
// layers x 8 heads, which walked all rows, kept or not, with one 64 KB chunk in flight: 235 us for 26120 rows of which
// half stay (428 MB to move); now 94 us, 19 us of them the selection.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <stdexcept>
#include <string>

#include "gemm.h"
#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"

namespace fc {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// scores[seq, layer, h, tok] = sign * ||K[tok, h, :]||      (mode 0: per head)
//                            = mean_h ||K[tok, h, :]||       (mode 1: shared by heads, largest kept)
// One CTA: 32 consecutive rows of every head; the norms pass through shared memory so that the scores are written 32
// consecutive floats at a time.  Hkv <= 32 (checked on the host).  Sixteen lanes read one 16-byte piece each of a row.
// Bound by the read of K: WIDE (head_dim 128, heads a multiple of eight) has sixteen rows in flight per group of lanes
// and forms their sixteen sums with 15 shuffles instead of 64 (lanes exchange halves of what they hold, so lane i
// ends with the sum of row i; the additions pair up as in the butterfly).  26120 rows
// in 4 layers x 8 heads (214 MB): 82 us with one row in flight per group and unrolled step, 49 us so.
constexpr int KN_ROWS = 32;

__device__ __forceinline__ float square_sum(const uint4& v, float ss) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {        // a bf16 is the upper half of the fp32 with the same value
    const float a = __uint_as_float(w[e] << 16), b = __uint_as_float(w[e] & 0xffff0000u);
    ss += a * a + b * b;
  }
  return ss;
}

template <bool WIDE>
__global__ void __launch_bounds__(256)
knorm_score_kernel(const bf16* __restrict__ pool, const int* __restrict__ block_tables,
                   const int* __restrict__ kv_lens, float* __restrict__ scores, int L, int num_blocks,
                   int block_size, int Hkv, int D, int max_blocks, int s_stride, int mode, uint32_t* status) {
  __shared__ float sn[KN_ROWS][33];
  const int seq = blockIdx.z, layer = blockIdx.y;
  const int len = kv_lens[seq];
  const int tok0 = blockIdx.x * KN_ROWS;
  if (tok0 >= len) return;
  const int sub = threadIdx.x & 15, grp = threadIdx.x >> 4;
  const long long kbase = ((long long)layer * 2 + 0) * num_blocks;
  const int* bt = block_tables + (long long)seq * max_blocks;
  const int rows = KN_ROWS * Hkv;
  if constexpr (WIDE) {
    // rows grp and grp + 16 of every head: two look-ups in the block table, then one stride from head to head
    const uint4* row[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int tok = tok0 + grp + 16 * i;
      row[i] = nullptr;
      if (tok < len) {
        const int blk = bt[tok / block_size];
        if (blk < 0 || blk >= num_blocks) report(status, ST_BAD_INDEX);
        else row[i] = reinterpret_cast<const uint4*>(pool + ((kbase + blk) * Hkv * block_size + tok % block_size) * 128) + sub;
      }
    }
    const long long head = (long long)block_size * 16;                 // 16-byte pieces from head to head
    for (int h0 = 0; h0 < Hkv; h0 += 8) {
      uint4 v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = make_uint4(0, 0, 0, 0);
        if (row[i & 1] != nullptr) v[i] = row[i & 1][(h0 + (i >> 1)) * head];
      }
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = square_sum(v[i], 0.f);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const bool up = (sub & o) != 0;                                // this lane goes on with the upper half
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float give = up ? x[i] : x[i + o], keep = up ? x[i + o] : x[i];
          x[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      sn[grp + 16 * (sub & 1)][h0 + (sub >> 1)] = sqrtf(x[0]);
    }
  } else {
#pragma unroll 4
    for (int r = grp; r < rows; r += 16) {
      const int h = r / KN_ROWS, tl = r % KN_ROWS;
      const int tok = tok0 + tl;
      float ss = 0.f;
      if (tok < len) {
        const int blk = bt[tok / block_size];
        if (blk < 0 || blk >= num_blocks) {
          report(status, ST_BAD_INDEX);
        } else {
          const uint4* row = reinterpret_cast<const uint4*>(
              pool + (((kbase + blk) * Hkv + h) * block_size + tok % block_size) * D);
          for (int i = sub; i < D / 8; i += 16) ss = square_sum(row[i], ss);
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (sub == 0) sn[tl][h] = sqrtf(ss);
    }
  }
  __syncthreads();
  float* out = scores + (((long long)seq * L + layer) * Hkv) * s_stride;
  for (int idx = threadIdx.x; idx < rows; idx += 256) {
    const int h = idx / KN_ROWS, tl = idx % KN_ROWS;
    const int tok = tok0 + tl;
    if (tok >= len) continue;
    float v;
    if (mode == 0) {
      v = -sn[tl][h];
    } else {
      float m = 0.f;
      for (int hh = 0; hh < Hkv; ++hh) m += sn[tl][hh];
      v = m / float(Hkv);
    }
    out[(long long)h * s_stride + tok] = v;
  }
}

// The four passes are chains of shared-memory latencies: long requests want few rows per thread (1024 threads) as long as all
// CTAs run at once, everything else more CTAs on an SM (256 threads, see launch_select_compact).
constexpr int SC_LONG = 2048;                    // rows

// kept [n_seq, L, Hkv, s_stride]: the first n_kept entries of a row are the kept rows, ascending
template <int SC_THREADS>
__global__ void __launch_bounds__(SC_THREADS)
select_rows_kernel(const float* __restrict__ scores, const int* __restrict__ kv_lens, const int* __restrict__ n_kepts,
                   int* __restrict__ kept, int L, int Hkv, int s_stride) {
  extern __shared__ uint32_t sm[];
  pdl_launch_dependents();
  const int h = blockIdx.x, layer = blockIdx.y, seq = blockIdx.z;
  const int S = kv_lens[seq];
  int k = n_kepts[seq];
  if (k >= S || S <= 0) return;
  if (k < 1) k = 1;
  uint32_t* keys = sm;                       // [S]
  uint32_t* hist = sm + s_stride;            // [256]
  int* s_misc = reinterpret_cast<int*>(hist + 256);   // [8]: bin, above, ...
  int* wsum = s_misc + 8;                    // [SC_THREADS / 32] warp partials
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const float* sc = scores + (((long long)seq * L + layer) * Hkv + h) * s_stride;
  for (int i = tid; i < S; i += SC_THREADS) keys[i] = float_key(sc[i]);
  __syncthreads();

  // ---- radix select: the k-th largest key
  uint32_t prefix = 0, mask = 0;
  int remaining = k;                         // rank still to find inside the current prefix class
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    // scores of one request share their leading bits, so most keys of a warp fall into the same bin: the lanes
    // with equal bins elect one that adds their count (one shared-memory atomic per distinct bin and warp)
    for (int i0 = 0; i0 < S; i0 += SC_THREADS) {
      const int i = i0 + tid;
      int bin = -1;
      if (i < S) {
        const uint32_t key = keys[i];
        if ((key & mask) == prefix) bin = int((key >> shift) & 0xFF);
      }
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      if (bin >= 0 && lane == __ffs(peers) - 1) atomicAdd(&hist[bin], unsigned(__popc(peers)));
    }
    __syncthreads();
    if (warp == 0) {
      // lane l owns bins 255 - 8 l ... 248 - 8 l (from the top); the lane whose bins contain rank `remaining`
      // walks its eight bins
      int mine = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) mine += int(hist[255 - 8 * lane - b]);
      int x = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      const int above = x - mine;                       // keys in higher bins than this lane's
      const bool here = above < remaining && remaining <= x;
      const unsigned found = __ballot_sync(0xffffffffu, here);
      if (found == 0) {
        if (lane == 31) {                               // fewer keys than `remaining` in this class: lowest bin
          s_misc[0] = 0;
          s_misc[1] = x - int(hist[0]);
        }
      } else if (here) {
        int acc = above, bin = 255 - 8 * lane;
        for (int b = 0; b < 7; ++b, --bin) {
          if (acc + int(hist[bin]) >= remaining) break;
          acc += int(hist[bin]);
        }
        s_misc[0] = bin;
        s_misc[1] = acc;
      }
    }
    __syncthreads();
    prefix |= uint32_t(s_misc[0]) << shift;
    mask |= 0xFFu << shift;
    remaining -= s_misc[1];
    __syncthreads();
  }
  const uint32_t thr = prefix;               // keep key > thr, plus the last `remaining` rows with key == thr
  const int need_eq = remaining;

  // total number of ties
  int eq_local = 0;
  for (int i = tid; i < S; i += SC_THREADS) eq_local += (keys[i] == thr);
  eq_local = int(warp_sum(float(eq_local)) + 0.5f);
  if (lane == 0) wsum[warp] = eq_local;
  __syncthreads();
  int eq_total = 0;
  for (int w = 0; w < SC_THREADS / 32; ++w) eq_total += wsum[w];
  __syncthreads();

  // ---- the kept rows in order: thread t owns rows [t * RPT, (t + 1) * RPT).  Two block-wide exclusive scans (ties,
  // then kept rows).
  const int RPT = (S + SC_THREADS - 1) / SC_THREADS;
  const int r_lo = min(S, tid * RPT), r_hi = min(S, r_lo + RPT);
  auto block_exclusive = [&](int local) -> int {         // exclusive prefix of `local` over the threads of the CTA
    int x = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int before = x - local;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    __syncthreads();
    return before;
  };
  int eq_mine = 0;
  for (int r = r_lo; r < r_hi; ++r) eq_mine += (keys[r] == thr);
  int eq_before = block_exclusive(eq_mine);
  // a tie is kept when it is among the last `need_eq` ties of the request
  int kept_mine = 0;
  {
    int e = eq_before;
    for (int r = r_lo; r < r_hi; ++r) {
      const uint32_t key = keys[r];
      const bool tie = key == thr;
      kept_mine += (key > thr) || (tie && (eq_total - e) <= need_eq);
      e += tie;
    }
  }
  int pos = block_exclusive(kept_mine);
  int* out = kept + (((long long)seq * L + layer) * Hkv + h) * s_stride;
  int e = eq_before;
  for (int r = r_lo; r < r_hi; ++r) {
    const uint32_t key = keys[r];
    const bool tie = key == thr;
    if ((key > thr) || (tie && (eq_total - e) <= need_eq)) out[pos++] = r;
    e += tie;
  }
}

// One CTA: 64 columns (128 bytes) of K or V of one (kv head, layer, request); eight lanes read a row's part.  Lane j of
// such a group looks up the addresses of the group's j-th row of the chunk, the others get them by shuffle: two block
// table look-ups per row instead of one per 16-byte piece.
constexpr int MV_THREADS = 256;
constexpr int MV_ROWS = 8;                       // rows per group of eight lanes and chunk
constexpr int MV_CHUNK = MV_THREADS / 8 * MV_ROWS;
constexpr uint32_t MV_NONE = 0xffffffffu;

template <int D>
__global__ void __launch_bounds__(MV_THREADS)
move_rows_kernel(bf16* __restrict__ pool, const int* kept, const int* __restrict__ block_tables,
                 const int* __restrict__ kv_lens, const int* __restrict__ n_kepts, int L, int num_blocks, int block_size,
                 int Hkv, int max_blocks, int s_stride, uint32_t* status) {
  constexpr int COLS = D / 64;
  pdl_wait();
  const int part = blockIdx.x % (2 * COLS), h = blockIdx.x / (2 * COLS), layer = blockIdx.y, seq = blockIdx.z;
  const int S = kv_lens[seq];
  int k = n_kepts[seq];
  if (k >= S || S <= 0) return;
  if (k < 1) k = 1;
  const int lane = threadIdx.x & 7, grp = threadIdx.x >> 3;
  const int* rows = kept + (((long long)seq * L + layer) * Hkv + h) * s_stride;
  const int* bt = block_tables + (long long)seq * max_blocks;
  // rows of a plane are numbered (block * Hkv + head) * block_size + row: 32 bits count 512 GB of 64-wide rows
  bf16* base = pool + ((long long)layer * 2 + part / COLS) * num_blocks * Hkv * block_size * D + (part % COLS) * 64 + lane * 8;
  auto number = [&](int tok) -> uint32_t {
    const int blk = bt[tok / block_size];
    if (blk < 0 || blk >= num_blocks) {
      report(status, ST_BAD_INDEX);
      return MV_NONE;
    }
    return (uint32_t(blk) * Hkv + h) * block_size + tok % block_size;
  };
  auto look_up = [&](int c0, uint32_t& src, uint32_t& dst) {
    src = dst = MV_NONE;
    const int j = c0 + grp * MV_ROWS + lane;
    if (j < k) {
      const int r = __ldcg(rows + j);            // written by the kernel before this one: not through the read-only path
      if (r != j) {                              // a row that stays is neither read nor written
        src = number(r);
        dst = number(j);
      }
    }
  };
  uint32_t src, dst, next_src, next_dst;
  look_up(0, src, dst);
  for (int c0 = 0; c0 < k; c0 += MV_CHUNK, src = next_src, dst = next_dst) {
    uint4 v[MV_ROWS];
#pragma unroll
    for (int u = 0; u < MV_ROWS; ++u) {
      const uint32_t from = __shfl_sync(0xffffffffu, src, u, 8);
      v[u] = make_uint4(0, 0, 0, 0);
      if (from != MV_NONE) v[u] = *reinterpret_cast<const uint4*>(base + (long long)from * D);
    }
    look_up(c0 + MV_CHUNK, next_src, next_dst);  // two look-ups in a row, while this chunk's rows arrive
    // every row of this chunk has been read (and of the chunks before) when the first one is written; rows only move
    // towards the front, so what is written here lies before the rows of every later chunk
    __syncthreads();
#pragma unroll
    for (int u = 0; u < MV_ROWS; ++u) {
      const uint32_t to = __shfl_sync(0xffffffffu, dst, u, 8);
      if (to != MV_NONE) *reinterpret_cast<uint4*>(base + (long long)to * D) = v[u];
    }
  }
}

void launch_knorm_scores(const void* pool, const int* block_tables, const int* kv_lens, float* scores, int n_seq,
                         int L, int num_blocks, int block_size, int Hkv, int D, int max_blocks, int max_len,
                         int s_stride, int mode, uint32_t* status, cudaStream_t stream) {
  if (n_seq == 0 || max_len == 0) return;
  if (Hkv > 32 || D % 8 != 0) throw std::runtime_error("knorm scores: at most 32 KV heads, head_dim a multiple of 8");
  dim3 grid((max_len + KN_ROWS - 1) / KN_ROWS, L, n_seq);
  auto kern = (D == 128 && Hkv % 8 == 0) ? knorm_score_kernel<true> : knorm_score_kernel<false>;
  kern<<<grid, 256, 0, stream>>>((const bf16*)pool, block_tables, kv_lens, scores, L, num_blocks, block_size, Hkv, D,
                                 max_blocks, s_stride, mode, status);
}

void launch_select_compact(void* pool, const float* scores, const int* block_tables, const int* kv_lens,
                           const int* n_kepts, int* kept, int n_seq, int L, int num_blocks, int block_size, int Hkv, int D,
                           int max_blocks, int s_stride, uint32_t* status, cudaStream_t stream) {
  if (n_seq == 0) return;
  const int smem = (s_stride + 256 + 8 + 1024 / 32) * 4;
  if (smem > 220 * 1024) throw std::runtime_error("select_compact: request too long for one CTA's shared memory");
  if (D != 64 && D != 128) throw std::runtime_error("select_compact: head_dim must be 64 or 128");
  if ((long long)num_blocks * Hkv * block_size >= (long long)MV_NONE)
    throw std::runtime_error("select_compact: too many rows in one plane of the pool");
  // 1024 -> 256 threads: 32 layers x 8 heads, 4 requests of 100 rows 38.8 -> 16.2 us (the moves included), of 800 rows 81 -> 60
  // us; 4 layers, 8 requests of 3000 rows 55 us both; 8 layers, 2 requests of 6000 rows 65 -> 72 us
  const bool wide = s_stride > SC_LONG && (long long)Hkv * L * n_seq <= 2ll * gemm_num_sms();
  auto select = wide ? select_rows_kernel<1024> : select_rows_kernel<256>;
  cudaFuncSetAttribute(select, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  select<<<dim3(Hkv, L, n_seq), wide ? 1024 : 256, smem, stream>>>(scores, kv_lens, n_kepts, kept, L, Hkv, s_stride);
  auto move = D == 128 ? move_rows_kernel<128> : move_rows_kernel<64>;
  launch_pdl(PDL_EVICT, move, dim3(Hkv * 2 * (D / 64), L, n_seq), dim3(MV_THREADS), 0, stream, (bf16*)pool, (const int*)kept,
             block_tables, kv_lens, n_kepts, L, num_blocks, block_size, Hkv, max_blocks, s_stride, status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("select_compact launch: ") + cudaGetErrorString(e));
}

}  // namespace fc

// bf16 GEMM for prefill sizes on CTA pairs: D[i, j] = act(sum_k A[i, k] * B[j, k] + bias[j]), tokens on the row
// operand, 256 x 256 output tile per pair of CTAs (a thread-block cluster of two, one CTA per SM).
//
// With one CTA per 128 x 256 tile (gemm.cu) every SM copies a whole 256 x 64 B tile per K block into its shared
// memory and its tensor core reads all of it back: shared-memory traffic, not the tensor pipe, bounds that kernel
// (81 % tensor-pipe activity).  Here the two CTAs of a pair issue ONE tcgen05.mma.cta_group::2 of M = 256, N = 256:
// each CTA holds 128 rows of A and 128 of the 256 rows of B, the tensor cores exchange the B halves between the
// two SMs, and each CTA's tensor memory receives its 128 x 256 half of the accumulator.  Per FLOP a CTA copies and
// reads two thirds of the operand bytes, and six pipeline stages fit where four did.
//
//   warp 0   TMA producer in BOTH CTAs: its own A tile and B half per stage (plain 2-D tiled loads from this
//            GPU's memory; every CTA fetches its own tiles), completion counted on the LEADER's (rank 0) barrier
//   warp 1   leader only: tcgen05.mma.cta_group::2 (4 x K = 16 per stage); tcgen05.commit to both CTAs' barriers
//            frees the stage in both and publishes the accumulator to both epilogues
//   warps 2-9 epilogue in both CTAs, two groups of four as in the staged form of gemm.cu: tcgen05.ld of the CTA's own
//            128 x 256 fp32 half, bias / activation / SwiGLU / residual, slabs of 64 columns through shared memory and
//            TMA; the 512 epilogue threads of the pair hand the accumulator back to the leader
// Two accumulators (2 x 256 TMEM columns per CTA) let the epilogue overlap the next tile's main loop.
//
// Every wait is bounded; both CTAs always reach the closing cluster barrier, so neither exits while its partner
// may still signal one of its barriers.
//
// Measured (32768 x 6144 x 4096): tensor pipe 88.5 % active against 81.1 % for gemm.cu, but both kernels run into
// the board's power limit (SM clock about 1.44 GHz) and take the same time within noise, so sizes like that come here
// only when asked to (FC_GEMM_PAIRS=1 / set_gemm_pairs(1)).  Asking for tiles 16 K blocks ahead to be brought into L2
// (cp.async.bulk.prefetch.tensor) made the K = 12288 shape 30 % slower and was taken out.  Short products run at full
// clock, where gemm.cu's four stages do not cover the latency of its 94 bytes per clock and SM: see gemm_pairs_faster.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <stdexcept>
#include <string>

#include "gemm.h"
#include "gemm_epilogue.cuh"
#include "ptx.cuh"

namespace fc {

namespace {

constexpr int P2_BM = 128;          // rows of A per CTA (256 per pair)
constexpr int P2_BNH = 128;         // rows of B per CTA (256 per pair)
constexpr int P2_BN = 256;
constexpr int P2_BK = 64;
constexpr int P2_STAGES = 6;
constexpr long long PAIRS_MIN = 2 * 1024, PAIRS_MAX = 64 * 1024;      // waves x K, see gemm_pairs_faster
constexpr int PAIRS_ACT_K = 1280, PAIRS_GATED_WAVES = 8;
constexpr int P2_THREADS = 320;
constexpr int P2_A_BYTES = P2_BM * P2_BK * 2;
constexpr int P2_B_BYTES = P2_BNH * P2_BK * 2;
constexpr int P2_STAGE_BYTES = P2_A_BYTES + P2_B_BYTES;              // 32 KiB per CTA
constexpr int P2_SLAB_OFF = P2_STAGES * P2_STAGE_BYTES;
constexpr int P2_BAR_OFF = P2_SLAB_OFF + 2 * SLAB_BYTES;
constexpr int P2_SMEM = P2_BAR_OFF + 256 + 1024;

struct Pair2Params {
  int M, N, K;
  const __nv_bfloat16* bias;
  int act;
  int num_m, num_n, group_m, total_work;
  int up_row0;            // SWIGLU: row of W where the `up` half starts (= output width)
  uint32_t* status;
};

enum PairForm : int { PF_PLAIN = 0, PF_SWIGLU = 1, PF_RESIDUAL = 2 };

// 2-D tiled load whose completion is counted on a barrier of the pair's leader CTA (`bar_cluster_addr` is a
// shared::cluster address); the destination is this CTA's own shared memory
__device__ __forceinline__ void p2_tma_load(void* smem, const CUtensorMap* m, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void p2_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives (once the MMAs issued so far are done) on the barrier at this shared-memory offset in both CTAs
__device__ __forceinline__ void p2_commit_both(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask)
               : "memory");
}
__device__ __forceinline__ void p2_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

template <int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P2_THREADS, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                      const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ CUtensorMap tma_r,
                      const Pair2Params p) {
  constexpr bool SWIGLU = FORM == PF_SWIGLU;
  extern __shared__ uint8_t smem_raw[];
  // the dynamic shared memory starts at the same offset in both CTAs, so the aligned base does too
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + P2_BAR_OFF);      // used in the leader
  uint64_t* empty_bar = full_bar + P2_STAGES;                               // one set per CTA
  uint64_t* acc_full = empty_bar + P2_STAGES;                               // [2], one set per CTA
  uint64_t* acc_empty = acc_full + 2;                                       // [2], used in the leader (512 arrivals)
  uint64_t* res_full = acc_empty + 2;                                       // [2], PF_RESIDUAL, one per epilogue group
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0: leader
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P2_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 512);
      mbar_init(&res_full[a], 1);
    }
    *s_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    // all 512 columns in each CTA: both allocations start at column 0, which the pair's MMA relies on
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  cluster_sync();                                   // the partner's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int num_kb = (p.K + P2_BK - 1) / P2_BK;

  auto decode_work = [&](int w, int& m_blk, int& n_blk) {
    const int per_group = p.group_m * p.num_n;
    const int g = w / per_group;
    const int first_m = g * p.group_m;
    const int gm = min(p.num_m - first_m, p.group_m);
    const int local = w - g * per_group;
    m_blk = first_m + local % gm;
    n_blk = local / gm;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = tmem_base == 0;
      if (!ok) report(p.status, ST_BAD_INDEX);      // the allocation did not start at column 0: do not run
      for (int w = pair; w < p.total_work && ok; w += num_pairs) {
        int m_blk, n_blk;
        decode_work(w, m_blk, n_blk);
        const int a_row = m_blk * (2 * P2_BM) + int(rank) * P2_BM;
        const int b_row = SWIGLU ? (rank == 0 ? n_blk * P2_BNH : p.up_row0 + n_blk * P2_BNH)
                                 : n_blk * P2_BN + int(rank) * P2_BNH;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (*s_abort || !mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_EMPTY)) {
            *s_abort = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * P2_STAGE_BYTES;
          const uint32_t bar = cluster_map_shared(smem_u32(&full_bar[stage]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * P2_STAGE_BYTES);      // both CTAs' bytes
          p2_tma_load(sa, &tma_a, bar, kb * P2_BK, a_row);
          p2_tma_load(sa + P2_A_BYTES, &tma_b, bar, kb * P2_BK, b_row);
          if (++stage == P2_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (ok) {
        // the leader's last commits also arrive on this CTA's stage barriers: let them land before the closing
        // cluster barrier (an unused stage passes at once)
        for (int n = 0; n < P2_STAGES; ++n) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_EMPTY)) break;
          if (++stage == P2_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      } else {
        // gave up: a copy requested just before may still be on its way into this CTA's shared memory
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer (leader only)
    if (lane == 0 && rank == 0 && tmem_base == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * P2_BM, P2_BN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int w = pair; w < p.total_work && ok; w += num_pairs) {
        if (*s_abort || !mbar_wait(&acc_empty[acc], acc_phase ^ 1, p.status, ST_TIMEOUT_ACC_EMPTY)) {
          *s_abort = 1;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + uint32_t(acc * P2_BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (*s_abort || !mbar_wait(&full_bar[stage], phase, p.status, ST_TIMEOUT_FULL)) {
            *s_abort = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * P2_STAGE_BYTES);
          const uint64_t da = make_sdesc_sw128(sa);
          const uint64_t db = make_sdesc_sw128(sa + P2_A_BYTES);
#pragma unroll
          for (int k = 0; k < P2_BK / 16; ++k)
            p2_mma(d_tmem, da + uint64_t(2 * k), db + uint64_t(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          p2_commit_both(&empty_bar[stage]);
          if (++stage == P2_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        p2_commit_both(&acc_full[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (both CTAs)
    const int lane_group = warp & 3;
    const int row = lane_group * 32 + lane;
    const int group = (warp - 2) >> 2;                        // takes the slabs group, group + 2, ...
    const bool leader = warp == 2 + 4 * group && lane == 0;
    uint8_t* const slab = smem + P2_SLAB_OFF + group * SLAB_BYTES;
    const int width = SWIGLU ? p.N / 2 : p.N;
    auto group_bar = [&] {                                    // a warp instruction: lanes that went ways of their own meet first
      __syncwarp();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
    };
    int acc = 0;
    uint32_t acc_phase = 0, res_phase = 0;
    for (int w = pair; w < p.total_work; w += num_pairs) {
      int m_blk, n_blk;
      decode_work(w, m_blk, n_blk);
      // a group goes on or gives up as one: its threads meet at barriers below
      if (!barrier_all(1 + group, 128, !*s_abort && mbar_wait(&acc_full[acc], acc_phase, p.status, ST_TIMEOUT_ACC_FULL))) {
        *s_abort = 1;
        break;
      }
      tc_fence_after();
      const uint32_t t_addr = tmem_base + (uint32_t(lane_group * 32) << 16) + uint32_t(acc * P2_BN);
      const uint32_t give_back = cluster_map_shared(smem_u32(&acc_empty[acc]), 0);
      const int row0 = m_blk * (2 * P2_BM) + int(rank) * P2_BM;
      const int col0 = n_blk * (SWIGLU ? P2_BNH : P2_BN);
      constexpr int SLABS = (SWIGLU ? P2_BNH : P2_BN) / SLAB;
#pragma unroll 1
      for (int sl = group; sl < SLABS; sl += 2) {
        const int col = col0 + sl * SLAB;
        const bool here = col < width && row0 < p.M;          // the same for the whole group
        if (leader) tma_store_wait_read();                    // the slab's last store has been read out of shared memory
        group_bar();
        if (FORM == PF_RESIDUAL && leader && here) {          // what is added arrives while the accumulator is read
          mbar_expect_tx(&res_full[group], SLAB_BYTES);
          tma_load_2d(slab, &tma_r, &res_full[group], col, row0);
        }
        __syncwarp();                                         // a tensor-memory load is a warp instruction
        uint32_t r[2][32];
        if constexpr (!SWIGLU) {
          tmem_ld_32x32(t_addr + uint32_t(sl * SLAB), r[0]);
          tmem_ld_32x32(t_addr + uint32_t(sl * SLAB + 32), r[1]);
          tmem_ld_wait();
          if (sl + 2 >= SLABS) {
            tc_fence_before();
            p2_arrive_cluster(give_back);
          }
        }
        if (FORM == PF_RESIDUAL && here) {
          if (!mbar_wait(&res_full[group], res_phase, p.status, ST_TIMEOUT_FULL)) *s_abort = 1;    // (no barrier is skipped)
          res_phase ^= 1;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t u[16];
          if constexpr (SWIGLU) {
            // accumulator columns [0, 128) = gate, [128, 256) = up
            const int c = sl * SLAB + half * 32;
            tmem_ld_32x32(t_addr + uint32_t(c), r[0]);
            tmem_ld_32x32(t_addr + uint32_t(P2_BNH + c), r[1]);
            tmem_ld_wait();
            if (half == 1 && sl + 2 >= SLABS) {
              tc_fence_before();
              p2_arrive_cluster(give_back);
            }
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              const float g0 = __uint_as_float(r[0][2 * t]), g1 = __uint_as_float(r[0][2 * t + 1]);
              u[t] = pack_bf16(g0 / (1.f + __expf(-g0)) * __uint_as_float(r[1][2 * t]),
                               g1 / (1.f + __expf(-g1)) * __uint_as_float(r[1][2 * t + 1]));
            }
          } else {
            float v[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) v[t] = __uint_as_float(r[half][t]);
            if (p.bias != nullptr) add_bias_chunk(v, p.bias, col + half * 32, p.N, col + SLAB <= p.N);
            if constexpr (FORM == PF_RESIDUAL) slab_add(slab, row, half, v);
            else apply_act_chunk(v, p.act);
#pragma unroll
            for (int t = 0; t < 16; ++t) u[t] = pack_bf16(v[2 * t], v[2 * t + 1]);
          }
          slab_put(slab, row, half, u);
        }
        fence_proxy_async();
        group_bar();
        if (leader && here) {
          tma_store_2d(slab, &tma_c, col, row0);
          tma_store_commit();
        }
        __syncwarp();
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (leader) tma_store_wait_all();
  }

  tc_fence_before();
  cluster_sync();                                   // nothing of the partner's is signalled after this
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

int g_pairs = -1;

template <int FORM>
void p2_launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tr, const Pair2Params& p, int pairs, cudaStream_t stream) {
  auto kern = gemm_bf16_2cta_kernel<FORM>;
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load(std::memory_order_relaxed) & bit)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P2_SMEM);
    if (e != cudaSuccess) throw std::runtime_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    configured.fetch_or(bit, std::memory_order_relaxed);
  }
  kern<<<2 * pairs, P2_THREADS, P2_SMEM, stream>>>(ta, tb, tc, tr, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("2-CTA gemm launch: ") + cudaGetErrorString(e));
}

}  // namespace

int gemm_pairs_mode() {
  if (g_pairs < 0) {
    const char* e = std::getenv("FC_GEMM_PAIRS");
    g_pairs = e != nullptr && (e[0] == '0' || e[0] == '1') ? e[0] - '0' : PAIRS_FASTER;
  }
  return g_pairs;
}
void set_gemm_pairs(int mode) { g_pairs = mode == PAIRS_NEVER || mode == PAIRS_FASTER ? mode : PAIRS_ALWAYS; }

// Whether a pair's tiles are the faster ones: short products run at full clock, where a wave of 256 x 256 pair tiles takes
// about 0.85 of a wave of 128 x 256 tiles (one CTA per tile -> pairs, kernel times inside the towers: 15 x 577 rows of CLIP:
// qkv 46.6 -> 43.3 us, out 25.2 -> 23.7 us, fc2 61.7 -> 53.8 us; 5 x 961 rows of SigLIP: 37.0 -> 34.7 us, 24.0 -> 22.3 us,
// 63.9 -> 53.5 us, fc1 48.3 -> 47.1 us), so they are taken unless they need another wave.  What a pair adds is its longer
// start and last epilogue, so the main loops have to be long enough to win that back:
//  - PAIRS_MIN (waves x K): 577 x 4096 at K = 1024 12.8 -> 13.7 us, at K = 1536 15.6 -> 16.1 us; at the line 1 to 2 %
//    either way (577 x 4096 at K = 2048 18.3 -> 18.6 us, sums with a residual a little faster); 1154 rows of CLIP: qkv 13.5 -> 14.4 us; 961 of SigLIP: qkv 14.2 -> 14.9 us, but fc2 (K = 4304) 34.5 -> 29.7 us.
//  - an activation that takes an exponential or an error function below K = PAIRS_ACT_K, where the epilogue of every tile is
//    longer than its main loop: CLIP's fc1 (quick GELU, K = 1024) 65.3 -> 68.5 us with 15 images, 29.5 -> 31.6 us with five;
//    2000 x 8192 with quick GELU at K = 1024: 3 % slower in pairs, at K = 1280: 4 % faster.
//  - SwiGLU in fewer than PAIRS_GATED_WAVES waves, against the plain epilogue of gemm.cu: 2000 rows of 2 x 4096 (four waves)
//    54.5 -> 58.6 us at K = 2048, 3000 rows (six) 63.4 -> 65.5 us at K = 1536; 6000 rows (eleven) 149.0 -> 142.7 us.
// Products of more than PAIRS_MAX (waves x K) run at the power limit, where both take the same time, and gemm_bf16 asks for
// pairs up to K = 2048 only (what it measured at K = 4096: gemm.cu).
bool gemm_pairs_faster(int M, int N, int K, int act, int sms) {
  if (M <= 256 || N < 256 || sms < 2) return false;
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long n = up(N, 256), one = up(up(M, 128) * n, sms), two = up(up(M, 256) * n, sms / 2);
  if (K < PAIRS_ACT_K && (act == ACT_GELU || act == ACT_QUICK_GELU || act == ACT_SILU || act == ACT_SWIGLU)) return false;
  if (act == ACT_SWIGLU && one < PAIRS_GATED_WAVES) return false;
  return one * K >= PAIRS_MIN && one * K <= PAIRS_MAX && two <= one;
}

// Columns [0, N) of `residual` (pitch ldr) are added where it is given.  False where the sizes or layouts do not fit.
bool gemm_bf16_2cta(const void* x, const void* w, void* c, const void* bias, const void* residual, int M, int N, int K,
                    long long ldx, long long ldw, long long ldc, long long ldr, int act, int sm_limit, uint32_t* status,
                    cudaStream_t stream) {
  const bool swiglu = act == ACT_SWIGLU;
  if (M <= 256 || N < 256 || K < P2_BK) return false;
  if (ldc % 8 != 0 || (reinterpret_cast<uintptr_t>(c) & 15) != 0) return false;
  if (swiglu && (N % 256 != 0 || bias != nullptr)) return false;
  const int sms = sm_limit > 0 ? sm_limit : gemm_num_sms();
  if (sms < 2) return false;
  Pair2Params p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.act = swiglu ? ACT_NONE : act;
  p.num_m = (M + 2 * P2_BM - 1) / (2 * P2_BM);
  p.num_n = swiglu ? N / 256 : (N + P2_BN - 1) / P2_BN;
  // raster: groups of `group_m` row blocks are finished one after the other, all column blocks of one before the
  // next.  The group's rows of A (group_m x 256 x K) stay in L2 while B streams past once per group, so larger groups
  // mean fewer passes over B; about 32 MB of A is what stays resident beside the streams (the L2 is two 63 MB halves).
  {
    const char* e = std::getenv("FC_GEMM_GROUP_M");
    const long long a_block = 2ll * 256 * K;
    p.group_m = e != nullptr ? std::max(1, std::atoi(e)) : int(std::max(8ll, std::min(32ll, (32ll << 20) / a_block)));
  }
  p.total_work = p.num_m * p.num_n;
  p.up_row0 = N / 2;
  p.status = status;
  const CUtensorMap ta = make_tmap_bf16_2d(x, M, K, ldx, P2_BM, P2_BK);
  const CUtensorMap tb = make_tmap_bf16_2d(w, N, K, ldw, P2_BNH, P2_BK);
  const int pairs = std::max(1, std::min(p.total_work, sms / 2));
  const CUtensorMap tc = make_tmap_bf16_2d(c, M, swiglu ? N / 2 : N, ldc, P2_BM, SLAB);
  if (swiglu) p2_launch<PF_SWIGLU>(ta, tb, tc, tc, p, pairs, stream);
  else if (residual == nullptr) p2_launch<PF_PLAIN>(ta, tb, tc, tc, p, pairs, stream);
  else p2_launch<PF_RESIDUAL>(ta, tb, tc, make_tmap_bf16_2d(residual, M, N, ldr, P2_BM, SLAB), p, pairs, stream);
  return true;
}

}  // namespace fc

// Flash-attention backward for sm_100a (head_dim 128).
//
// A work item is one 128-key tile of one (batch, kv-head); its CTA loops over every query head of the group and every
// query tile that can see those keys.  Scores are kept transposed (TMEM lane = key, column = query), so that P^T goes
// back to TMEM and is the A operand of its MMA there.  Per (query tile, key tile) five tcgen05 MMAs run:
//     S^T = K Q^T      dP^T = V dO^T      dV += P^T dO      dQ_part = dS K      dK += dS^T Q
// TMEM: S^T (P^T over it) | dP^T (dQ_part over it) | dK | dV, 128 columns each.  dK and dV stay in TMEM for the whole
// work item (no atomics, GQA heads accumulate in place).
//
// Roles (16 warps): two compute warpgroups form P and dS (thread <-> key row, 64 query columns), one warpgroup drains the
// dQ partial to an fp32 scratch tensor with TMA reduce-adds from a staging buffer of its own, and one warpgroup holds
// the TMA warp, which also hands out the work items, the MMA warp and the warp that brings the row statistics into shared
// memory.
//
// The MMA order is dV(j), S(j+1) | dQ(j), dK(j), dP(j+1): S(j+1) is issued while the compute warps form dS(j), so that
// P(j+1) is formed under dQ(j) and dK(j); dQ(j) is drained under dK(j); and dS(j+1) is formed under dV(j+1), S(j+2).
// What bounds it: all MMAs but one take both operands from shared memory (8 KB per 64-cycle instruction, the port's
// 128 B/clk), and with the staging of dQ and the loads about 512 KB pass the port per tile pair (4100 cycles, against
// 2560 cycles of tensor work and about 1024 cycles of MUFU work for the exponentials).
//
// All kernels of the backward, before (P and dS through shared memory, dQ drained by the compute warps, every MMA waiting for
// the previous stage of the same tile) and now: B 2, S 4096, H 32 causal 1058 -> 730 us; B 3, S 1515, H 40 / 8 464 -> 238 us;
// B 1, S 8192, H 32 / 16, window 4096, soft-cap 1858 -> 1078 us (one GPU; others at other clocks differ by a few per cent).
//
// The math is the standard recompute form: P = exp(S - lse), dS = P * (dP - delta) with the softmax scale applied to the
// sums dQ and dK, delta = rowsum(dO * O) from a pre-pass; a tanh soft-cap multiplies dS by (1 - tanh^2).
//
// Counterpart of the autodiff of `olmax/nn/attention.py:96-103` (cuDNN backward in the reference).
#include "flash_attn.h"
#include "flash_attn_noalloc.h"
#include "host_common.h"
#include "sm100.cuh"

namespace ob {

int encode_bshd_map(CUtensorMap* m, const void* ptr, int B, int S, int H, long long sb, long long ss, long long sh,
                    int box_rows);

namespace fa_bwd {

constexpr int T = 128;    // tile (queries and keys)
constexpr int HD = 128;
constexpr int BLK = 128 * 64 * 2;   // 16 KiB swizzled block [128 rows][64 elems]
constexpr int TILE = 2 * BLK;       // 32 KiB
// Q is needed from S(j) to dK(j), across S(j+1): two stages.  dO is needed for dP(j) and dV(j) only, which are
// neighbours, and its next tile loads under S(j+1), dQ(j), dK(j): one stage.
constexpr int OFF_K = 0;
constexpr int OFF_V = TILE;
constexpr int OFF_Q = 2 * TILE;
constexpr int OFF_DO = 4 * TILE;
constexpr int OFF_DS = 5 * TILE;                   // dS^T, bf16
constexpr int OFF_STAGE = 6 * TILE;                // dQ staging: per drain warp two [32 rows][32 floats] slots
constexpr int SLOT = 32 * 128;
constexpr int OFF_STATS = OFF_STAGE + 4 * 2 * SLOT;   // [2 stages][-lse * log2(e), -delta][128]
constexpr int STATS_BYTES = 2 * T * 4;
constexpr int OFF_BAR = OFF_STATS + 2 * STATS_BYTES;
constexpr int SMEM_BYTES = OFF_BAR + 256;          // no slack: the base is 1024-byte aligned (checked by the kernel)
constexpr int THREADS = 512;
constexpr int COMPUTE_WARPS = 8;
// registers per thread after the split; 2 * 168 + 88 + 88 = 512 = 4 * the 128 of the launch
constexpr int REGS_COMPUTE = 168, REGS_DRAIN = 88, REGS_ISSUE = 88;
constexpr int TMEM_COLS = 512;
constexpr int C_S = 0, C_DP = 128, C_DK = 256, C_DV = 384;

struct Params {
  int B, S, H, Hkv;
  int Sk, q_off;   // key length; key-axis position of query row 0
  int causal, window;
  int kv_tiles, group;   // key tiles per slice; (batch, kv-head) slices per scheduling group
  float scale, scale_log2, scale_over_cap, cap_log2;
  const float* lse;
  const float* delta;
  bf16* dk; long long dk_sb, dk_ss, dk_sh;
  bf16* dv; long long dv_sb, dv_ss, dv_sh;
  int* status;
};

__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int N>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// A work item: one 128-key tile of one (batch, kv-head), and the query tiles [i_lo, i_lo + n_q) that see it.
// Schedule: inside a group of `group` slices the key tiles come in order, all slices of the group for each tile, so that
// (causal) the longest loops of the group start first.
struct Item {
  int kv0, hkv, b, i_lo, n_q;
};
__device__ __forceinline__ Item decode_item(const Params& p, int w) {
  const int per_group = p.group * p.kv_tiles;
  const int grp = w / per_group;
  const int slices = min(p.group, p.B * p.Hkv - grp * p.group);
  const int in_group = w - grp * per_group;
  const int kv_tile = in_group / slices;
  const int bh = grp * p.group + in_group - kv_tile * slices;
  Item t;
  t.b = bh / p.Hkv;
  t.hkv = bh - t.b * p.Hkv;
  t.kv0 = kv_tile * T;
  // rows i with kv0 <= q_off + i (causal) and q_off + i <= kv0 + T - 1 + window
  int i_hi = (p.S + T - 1) / T - 1;
  t.i_lo = p.causal ? max(0, t.kv0 - p.q_off) / T : 0;
  if (p.window >= 0) {
    const int last = t.kv0 + T - 1 + p.window - p.q_off;
    i_hi = last < 0 ? -1 : min(i_hi, last / T);
  }
  t.n_q = max(0, i_hi - t.i_lo + 1);
  return t;
}

// CAPPED: with a soft-cap.  Its code and registers stay out of the plain kernel, and the other way round.
// PERSISTENT: the CTA that runs on an SM takes over the items of CTAs that have not started, so that the next item's loads,
// first scores and dP run under the write-out of dK / dV; else every CTA has its one item.  Without a soft-cap the three
// kernels of the backward gain by it (both sides on one GPU each time): B 64, S 1024, H 8 682 -> 618 us (4.5 query tiles
// per item), B 2, S 4096, H 32 748 -> 723, B 3, S 1515, H 40 / 8 and B 1, S 8192, H 32 / 16, window 4096 unchanged.  With
// one, the compute warps bound the loop and the longer-lived state costs them: B 1, S 8192, H 32 / 16 1364 -> 1438 us,
// with window 4096 1058 -> 1075; so the capped kernel keeps one item per CTA.
template <bool CAPPED>
__global__ void __launch_bounds__(THREADS, 1)
    flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ CUtensorMap tmDQ, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* k_full = bars + 0;
  uint64_t* v_full = bars + 1;
  uint64_t* q_full = bars + 2;     // [2]
  uint64_t* q_empty = bars + 4;    // [2]
  uint64_t* do_full = bars + 6;
  uint64_t* do_empty = bars + 7;
  uint64_t* s_full = bars + 8;
  uint64_t* dp_full = bars + 9;
  uint64_t* p_ready = bars + 10;   // one arrival per compute warp
  uint64_t* ds_ready = bars + 11;  // one arrival per compute warp
  uint64_t* dq_full = bars + 12;
  uint64_t* dq_read = bars + 13;   // one arrival per drain warp
  uint64_t* all_done = bars + 14;  // every MMA of the work item has finished
  uint64_t* st_full = bars + 15;   // [2] row statistics
  uint64_t* st_empty = bars + 17;  // [2] one arrival per compute warp
  uint64_t* acc_free = bars + 19;  // dK / dV have left TMEM: one arrival per compute warp
  uint64_t* item_full = bars + 20;   // [2]
  uint64_t* item_empty = bars + 22;  // [2] one arrival per warp that reads the item: MMA, statistics, drain, compute
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* item_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);   // [2] work item, < 0: end
  uint64_t* taken_full = bars + 26;
  uint4* taken = reinterpret_cast<uint4*>(bars + 28);   // the scheduler's last answer, see next_cta_request

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  constexpr bool PERSISTENT = !CAPPED;
  const int G = p.H / p.Hkv;

  // Swizzled tiles have to start on 1024-byte boundaries.  The kernel has no static shared memory, so its dynamic part
  // does; were it otherwise, report it and leave the results unwritten (uniform over the CTA: nothing is waited for).
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report_error(p.status, ERR_BAD_ARG, 699, (int)smem_u32(smem));
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&st_full[s], 1);
      mbar_init(&st_empty[s], COMPUTE_WARPS);
    }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, COMPUTE_WARPS);
    mbar_init(ds_ready, COMPUTE_WARPS);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, 4);
    mbar_init(all_done, 1);
    mbar_init(acc_free, COMPUTE_WARPS);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&item_full[s], 1);
      mbar_init(&item_empty[s], 2 + 4 + COMPUTE_WARPS);
    }
    mbar_init(taken_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // The next work item of a warp other than the scheduler's; < 0: none is left, or the wait gave up (`dead`).  The first is
  // the CTA's own index, known to every warp at once; the others come through the two item slots.
  auto next_item = [&](uint32_t n_item, int site, bool& dead) {
    if (n_item == 0) return (int)blockIdx.x;
    if constexpr (!PERSISTENT) return -1;
    const uint32_t k = n_item - 1;
    dead = !mbar_wait(&item_full[k & 1], (k >> 1) & 1u, abort_flag, p.status, site);
    if (dead) return -1;
    const int w = item_slot[k & 1];
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_empty[k & 1]);
    return w;
  };

  // The issuing and draining warps run their loops with all 32 lanes so that the loop state stays warp-uniform; one
  // elected lane issues.  A wait that gives up marks the warp `dead`: the loop then runs out without issuing anything.
  if (warp >= 12) {
    reg_dealloc<REGS_ISSUE>();
    if (warp == 12) {
      // ---------------- scheduler + TMA producer ----------------
      const bool leader = elect_one();
      bool dead = false;
      if (leader) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmDO);
      }
      uint32_t g = 0, n_work = 0;   // iterations so far (stages and phases run on across items); items with iterations
      for (uint32_t n_item = 0; !dead; ++n_item) {
        int w = n_item == 0 ? (int)blockIdx.x : -1;
        if (PERSISTENT && n_item > 0) {
          // not before the last dV of the current item: a CTA that still has work would take an item from one that has none
          if (g > 0) dead = !mbar_wait(do_empty, (g & 1u) ^ 1u, abort_flag, p.status, 691);
          if (dead) break;
          const uint32_t k = n_item - 1;
          if (lane == 0) next_cta_request(taken, taken_full);
          dead = !mbar_wait(taken_full, k & 1u, abort_flag, p.status, 692);
          if (dead) break;
          w = next_cta_answer(taken);
          __syncwarp();
          dead = !mbar_wait(&item_empty[k & 1], ((k >> 1) & 1u) ^ 1u, abort_flag, p.status, 690);
          if (dead) break;
          if (lane == 0) {
            item_slot[k & 1] = w;
            mbar_arrive(&item_full[k & 1]);
          }
        }
        if (w < 0) break;
        const Item t = decode_item(p, w);
        const int n_iters = t.n_q * G;
        int hq = 0, iq = 0;   // query head within the group, query tile
        for (int it = 0; it < n_iters; ++it, ++g) {
          const uint32_t s = g & 1u;
          const int h = t.hkv * G + hq;
          const int q0 = (t.i_lo + iq) * T;
          if (!dead) dead = !mbar_wait(&q_empty[s], ((g >> 1) & 1u) ^ 1u, abort_flag, p.status, 700);
          if (leader && !dead) {
            uint8_t* sq = smem + OFF_Q + s * TILE;
            mbar_arrive_expect_tx(&q_full[s], TILE);
            tma_load_4d(sq, &tmQ, &q_full[s], 0, h, q0, t.b);
            tma_load_4d(sq + BLK, &tmQ, &q_full[s], 64, h, q0, t.b);
          }
          if (it == 0) {   // K and V replace the previous item's, once its MMAs are through
            if (!dead && n_work > 0) dead = !mbar_wait(all_done, (n_work & 1u) ^ 1u, abort_flag, p.status, 702);
            if (leader && !dead) {
              mbar_arrive_expect_tx(k_full, TILE);
              tma_load_4d(smem + OFF_K, &tmK, k_full, 0, t.hkv, t.kv0, t.b);
              tma_load_4d(smem + OFF_K + BLK, &tmK, k_full, 64, t.hkv, t.kv0, t.b);
              mbar_arrive_expect_tx(v_full, TILE);
              tma_load_4d(smem + OFF_V, &tmV, v_full, 0, t.hkv, t.kv0, t.b);
              tma_load_4d(smem + OFF_V + BLK, &tmV, v_full, 64, t.hkv, t.kv0, t.b);
            }
          }
          if (!dead) dead = !mbar_wait(do_empty, (g & 1u) ^ 1u, abort_flag, p.status, 701);
          if (leader && !dead) {
            mbar_arrive_expect_tx(do_full, TILE);
            tma_load_4d(smem + OFF_DO, &tmDO, do_full, 0, h, q0, t.b);
            tma_load_4d(smem + OFF_DO + BLK, &tmDO, do_full, 64, h, q0, t.b);
          }
          if (++iq == t.n_q) {
            iq = 0;
            ++hq;
          }
        }
        if (n_iters > 0) ++n_work;
      }
    } else if (warp == 13) {
      // ---------------- MMA issue ----------------
      const bool leader = elect_one();
      constexpr uint32_t id_kk = make_idesc_bf16(T, T, 0, 0);    // both K-major
      constexpr uint32_t id_mm = make_idesc_bf16(T, HD, 1, 1);   // both MN-major
      constexpr uint32_t id_km = make_idesc_bf16(T, HD, 0, 1);   // A K-major (or in TMEM), B MN-major
      // Shared-memory descriptors: the high word depends only on the operand's major-ness, the low word is the start
      // address in 16-byte units.  A K-major [128][128] tile is two [128][64] blocks: k step kk sits at
      // (kk / 4) * BLK + (kk % 4) * 32 bytes; in an MN-major tile k step kk sits at kk * 2048 bytes.
      const uint64_t d_k = make_smem_desc(0, 0, 1024), d_mn = make_smem_desc(0, BLK, 1024);
      const uint32_t hi_k = (uint32_t)(d_k >> 32), hi_mn = (uint32_t)(d_mn >> 32);
      const uint32_t lo_flags_k = (uint32_t)d_k, lo_flags_mn = (uint32_t)d_mn;   // low-word bits above the address
      auto lo = [](uint32_t addr) { return (addr & 0x3FFFFu) >> 4; };
      const uint32_t aK = lo(smem_u32(smem + OFF_K)), aV = lo(smem_u32(smem + OFF_V)), aDS = lo(smem_u32(smem + OFF_DS));
      const uint32_t aQ0 = lo(smem_u32(smem + OFF_Q)), aDO = lo(smem_u32(smem + OFF_DO));
      constexpr uint32_t TILE16 = TILE >> 4;
      auto koff = [](int kk) { return ((uint32_t)(kk >> 2) * BLK + (uint32_t)(kk & 3) * 32) >> 4; };
      auto issue_kk = [&](uint32_t d, uint32_t a, uint32_t bb) {   // D = A B^T over the head dimension
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_ss_lohi(tmem_base + d, lo_flags_k | (a + koff(kk)), hi_k, lo_flags_k | (bb + koff(kk)), hi_k, id_kk,
                       kk != 0 ? 1u : 0u);
      };
      bool dead = false;
      uint32_t g = 0, n_work = 0;
      for (uint32_t n_item = 0; !dead; ++n_item) {
        const int w = next_item(n_item, 798, dead);
        if (w < 0) break;
        const Item t = decode_item(p, w);
        const int n_iters = t.n_q * G;
        if (n_iters == 0) continue;
        // first scores and dP of the item: they run under the previous item's dK / dV write-out
        if (!dead) dead = !mbar_wait(k_full, n_work & 1u, abort_flag, p.status, 800);
        if (!dead) dead = !mbar_wait(&q_full[g & 1], (g >> 1) & 1u, abort_flag, p.status, 801);
        tc_fence_after_sync();
        if (leader && !dead) {
          issue_kk(C_S, aK, aQ0 + (g & 1u) * TILE16);
          umma_commit(s_full);
        }
        if (!dead) dead = !mbar_wait(v_full, n_work & 1u, abort_flag, p.status, 802);
        if (!dead) dead = !mbar_wait(do_full, g & 1u, abort_flag, p.status, 803);
        if (!dead && g > 0) dead = !mbar_wait(dq_read, (g & 1u) ^ 1u, abort_flag, p.status, 809);
        tc_fence_after_sync();
        if (leader && !dead) {
          issue_kk(C_DP, aV, aDO);
          umma_commit(dp_full);
        }
        for (int it = 0; it < n_iters; ++it, ++g) {
          const uint32_t ph = g & 1u;
          const uint32_t aQ = aQ0 + ph * TILE16;
          // dV += P^T dO; P^T of queries [0, 64) is in columns [0, 32) of the S quarter, of the others in [64, 96)
          if (!dead) dead = !mbar_wait(p_ready, ph, abort_flag, p.status, 804);
          if (!dead && it == 0 && n_work > 0) dead = !mbar_wait(acc_free, (n_work & 1u) ^ 1u, abort_flag, p.status, 810);
          tc_fence_after_sync();
          if (leader && !dead) {
#pragma unroll
            for (int kk = 0; kk < T / 16; ++kk)
              umma_ts_lohi(tmem_base + C_DV, tmem_base + C_S + (uint32_t)((kk >> 2) * 64 + (kk & 3) * 8),
                           lo_flags_mn | (aDO + (uint32_t)kk * 128u), hi_mn, id_km, (it | kk) != 0 ? 1u : 0u);
            umma_commit(do_empty);
          }
          const bool more = it + 1 < n_iters;
          if (more) {   // the next scores overwrite P^T: MMAs of one thread run in order
            const uint32_t s2 = ph ^ 1u;
            if (!dead) dead = !mbar_wait(&q_full[s2], ((g + 1) >> 1) & 1u, abort_flag, p.status, 805);
            tc_fence_after_sync();
            if (leader && !dead) {
              issue_kk(C_S, aK, aQ0 + s2 * TILE16);
              umma_commit(s_full);
            }
          }
          // dQ_part = dS K over the dP columns, dK += dS^T Q
          if (!dead) dead = !mbar_wait(ds_ready, ph, abort_flag, p.status, 806);
          tc_fence_after_sync();
          if (leader && !dead) {
#pragma unroll
            for (int kk = 0; kk < T / 16; ++kk)
              umma_ss_lohi(tmem_base + C_DP, lo_flags_mn | (aDS + (uint32_t)kk * 128u), hi_mn,
                           lo_flags_mn | (aK + (uint32_t)kk * 128u), hi_mn, id_mm, kk != 0 ? 1u : 0u);
            umma_commit(dq_full);
#pragma unroll
            for (int kk = 0; kk < T / 16; ++kk)
              umma_ss_lohi(tmem_base + C_DK, lo_flags_k | (aDS + koff(kk)), hi_k, lo_flags_mn | (aQ + (uint32_t)kk * 128u),
                           hi_mn, id_km, (it | kk) != 0 ? 1u : 0u);
            umma_commit(&q_empty[ph]);
          }
          if (more) {
            if (!dead) dead = !mbar_wait(do_full, ph ^ 1u, abort_flag, p.status, 807);
            if (!dead) dead = !mbar_wait(dq_read, ph, abort_flag, p.status, 808);
            tc_fence_after_sync();
            if (leader && !dead) {
              issue_kk(C_DP, aV, aDO);
              umma_commit(dp_full);   // all MMAs that read dS(it) have finished too: its buffer may be written again
            }
          }
        }
        if (leader && !dead) umma_commit(all_done);
        ++n_work;
      }
    } else if (warp == 14) {
      // ---------------- row statistics: -lse * log2(e) and -delta of the 128 queries of each iteration ----------------
      const float LOG2E = 1.4426950408889634f;
      bool dead = false;
      uint32_t g = 0;
      for (uint32_t n_item = 0; !dead; ++n_item) {
        const int w = next_item(n_item, 848, dead);
        if (w < 0) break;
        const Item t = decode_item(p, w);
        const int n_iters = t.n_q * G;
        int hq = 0, iq = 0;
        for (int it = 0; it < n_iters; ++it, ++g) {
          const uint32_t s = g & 1u;
          const int q0 = (t.i_lo + iq) * T;
          const long long base = ((long long)t.b * p.H + (t.hkv * G + hq)) * p.S;
          float l[4], d[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {   // rows beyond S: exp2(-inf) = 0
            const int q = q0 + j * 32 + lane;
            l[j] = q < p.S ? -__ldg(p.lse + base + q) * LOG2E : -INFINITY;
            d[j] = q < p.S ? -__ldg(p.delta + base + q) : 0.f;
          }
          if (!dead) dead = !mbar_wait(&st_empty[s], ((g >> 1) & 1u) ^ 1u, abort_flag, p.status, 850);
          if (!dead) {
            float* dst = reinterpret_cast<float*>(smem + OFF_STATS + s * STATS_BYTES) + lane;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              dst[j * 32] = l[j];
              dst[T + j * 32] = d[j];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&st_full[s]);
          }
          if (++iq == t.n_q) {
            iq = 0;
            ++hq;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 8) {
    // ---------------- dQ drain: thread <-> query row; fp32 partial += into global memory ----------------
    reg_dealloc<REGS_DRAIN>();
    const int qd = warp & 3;
    const bool leader = elect_one();
    const uint32_t t_src = tmem_base + ((uint32_t)(qd * 32) << 16) + C_DP;
    uint8_t* slots = smem + OFF_STAGE + qd * 2 * SLOT;
    const int sw = lane & 7;
    bool dead = false;
    auto put = [&](int cc, const uint32_t (&r)[32], int h, int row0, int b) {
      // at most one copy of this warp may still read its slot: the other slot is free
      if (leader) tma_store_wait_read<1>();
      __syncwarp();
      uint8_t* slot = slots + (cc & 1) * SLOT;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(slot + lane * 128 + ((j ^ sw) << 4)) =
            make_uint4(r[j * 4], r[j * 4 + 1], r[j * 4 + 2], r[j * 4 + 3]);
      fence_proxy_async();
      __syncwarp();
      if (leader) {
        if (row0 < p.S) tma_reduce_add_4d(&tmDQ, slot, cc * 32, h, row0, b);
        tma_store_commit();
      }
    };
    uint32_t g = 0;
    for (uint32_t n_item = 0; !dead; ++n_item) {
      const int w = next_item(n_item, 948, dead);
      if (w < 0) break;
      const Item t = decode_item(p, w);
      const int n_iters = t.n_q * G;
      int hq = 0, iq = 0;
      for (int it = 0; it < n_iters; ++it, ++g) {
        const int h = t.hkv * G + hq;
        const int row0 = (t.i_lo + iq) * T + qd * 32;
        if (!dead) dead = !mbar_wait(dq_full, g & 1u, abort_flag, p.status, 950);
        if (!dead) {
          tc_fence_after_sync();
          uint32_t r0[32], r1[32];
          tmem_ld32(t_src, r0);
          tmem_ld32(t_src + 32, r1);
          tmem_ld_wait();
          put(0, r0, h, row0, t.b);
          put(1, r1, h, row0, t.b);
          tmem_ld32(t_src + 64, r0);
          tmem_ld32(t_src + 96, r1);
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_read);   // the columns may be overwritten by the next dP
          put(2, r0, h, row0, t.b);
          put(3, r1, h, row0, t.b);
        }
        if (++iq == t.n_q) {
          iq = 0;
          ++hq;
        }
      }
    }
    if (leader) tma_store_wait<0>();
    __syncwarp();
  } else {
    // ---------------- P / dS: 8 warps, thread <-> (key row, 64 query columns); dK / dV at the end ----------------
    // Two warps share each TMEM lane quarter and split the 128 columns, so that every scheduler has two compute warps
    // to hide TMEM-load, MUFU and shared-memory latencies behind each other.
    reg_alloc<REGS_COMPUTE>();
    const int qd = warp & 3;
    const int half = warp >> 2;
    const int row = qd * 32 + lane;
    const int col0 = half * 64;
    const uint32_t t_lane = tmem_base + ((uint32_t)(qd * 32) << 16);
    uint8_t* sDS = smem + OFF_DS + half * BLK + row * 128;   // this thread's 128-byte row of query block `half`
    const int sw = row & 7;
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    const float2 over_cap2 = make_float2(p.scale_over_cap, p.scale_over_cap), cap2 = make_float2(p.cap_log2, p.cap_log2);
    bool ok = true;
    uint32_t g = 0, n_work = 0;
    for (uint32_t n_item = 0; ok; ++n_item) {
      bool dead = false;
      const int w = next_item(n_item, 898, dead);
      if (w < 0) break;
      const Item t = decode_item(p, w);
      const int n_iters = t.n_q * G, kv0 = t.kv0;
      const int kv_idx = kv0 + row;
      const bool kv_ok = kv_idx < p.Sk;
      int iq = 0;
      for (int it = 0; it < n_iters && ok; ++it, ++g) {
        const uint32_t ph = g & 1u, ph2 = (g >> 1) & 1u;
        const int qp0 = p.q_off + (t.i_lo + iq) * T;   // position of the first query on the key axis
        if (++iq == t.n_q) iq = 0;
        const bool need_mask = (kv0 + T > p.Sk) || (p.causal && kv0 + T - 1 > qp0) ||
                               (p.window >= 0 && kv0 < qp0 + T - 1 - p.window);
        const float4* st = reinterpret_cast<const float4*>(smem + OFF_STATS + ph * STATS_BYTES) + half * 16;

        ok = mbar_wait(&st_full[ph], ph2, abort_flag, p.status, 899);
        if (!ok) break;
        ok = mbar_wait(s_full, ph, abort_flag, p.status, 900);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t r0[32], r1[32];   // scores, then P (times 1 - tanh^2 when capped): kept in fp32 until dS is formed
        {
          uint32_t pp[32];  // P of this half row, bf16x2
          tmem_ld32(t_lane + C_S + (uint32_t)col0, r0);
          tmem_ld32(t_lane + C_S + (uint32_t)(col0 + 32), r1);
          tmem_ld_wait();
          // P = exp2(s * scale * log2e - lse2), in place over the loaded scores.  The soft-cap and mask cases are
          // handled by loops of their own: a branch inside the hot loop would cut it into one basic block per element
          // pair and expose the FFMA -> EX2 -> pack latency of every pair instead of overlapping the pairs.
          int c_lo = 0, c_hi = T;   // visible columns of this key, relative to col0
          if (need_mask) {
            if (p.causal) c_lo = kv_idx - qp0 - col0;
            if (p.window >= 0) c_hi = kv_idx + p.window - qp0 - col0;
            if (!kv_ok) c_lo = T;
          }
          if constexpr (CAPPED) {
            float2 w[16];   // 1 - tanh^2
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              uint32_t(&r)[32] = hh ? r1 : r0;
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 l = st[hh * 8 + (i >> 2)];
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                  const float2 x = mul2(make_float2(__uint_as_float(r[i + j]), __uint_as_float(r[i + j + 1])), over_cap2);
                  const float2 t = make_float2(fast_tanh(x.x), fast_tanh(x.y));
                  w[(i + j) >> 1] = fma2(mul2(t, make_float2(-1.f, -1.f)), t, make_float2(1.f, 1.f));
                  const float2 a = fma2(t, cap2, j ? make_float2(l.z, l.w) : make_float2(l.x, l.y));
                  r[i + j] = __float_as_uint(fast_exp2(a.x));
                  r[i + j + 1] = __float_as_uint(fast_exp2(a.y));
                }
              }
              if (need_mask) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (hh * 32 + i < c_lo || hh * 32 + i > c_hi) r[i] = 0u;
              }
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float2 v = make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                const float2 vw = mul2(v, w[i >> 1]);
                pp[hh * 16 + (i >> 1)] = pack_bf16x2(v.x, v.y);
                r[i] = __float_as_uint(vw.x);
                r[i + 1] = __float_as_uint(vw.y);
              }
            }
          } else {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              uint32_t(&r)[32] = hh ? r1 : r0;
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 l = st[hh * 8 + (i >> 2)];
                const float2 a = fma2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), scale2, make_float2(l.x, l.y));
                const float2 c = fma2(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), scale2, make_float2(l.z, l.w));
                r[i] = __float_as_uint(fast_exp2(a.x));
                r[i + 1] = __float_as_uint(fast_exp2(a.y));
                r[i + 2] = __float_as_uint(fast_exp2(c.x));
                r[i + 3] = __float_as_uint(fast_exp2(c.y));
              }
            }
            if (need_mask) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (i < c_lo || i > c_hi) r0[i] = 0u;
                if (i + 32 < c_lo || i + 32 > c_hi) r1[i] = 0u;
              }
            }
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              pp[i >> 1] = pack_bf16x2(__uint_as_float(r0[i]), __uint_as_float(r0[i + 1]));
              pp[16 + (i >> 1)] = pack_bf16x2(__uint_as_float(r1[i]), __uint_as_float(r1[i + 1]));
            }
          }
          // each half keeps to the columns it has read itself: the other half may still be reading its scores
          tmem_st32(t_lane + C_S + (uint32_t)col0, pp);
          tmem_st_wait();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready);

        ok = mbar_wait(dp_full, ph, abort_flag, p.status, 901);   // also: the MMAs that read dS(it - 1) have finished
        if (!ok) break;
        tc_fence_after_sync();
        {
          uint32_t g0[32], g1[32];
          tmem_ld32(t_lane + C_DP + (uint32_t)col0, g0);
          tmem_ld32(t_lane + C_DP + (uint32_t)(col0 + 32), g1);
          tmem_ld_wait();
          // eight 16-byte chunks of this row; the chunk index is XOR-swizzled by row % 8 (128-byte swizzle)
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            const uint32_t* g = ch < 4 ? g0 + ch * 8 : g1 + (ch - 4) * 8;
            const uint32_t* pv = ch < 4 ? r0 + ch * 8 : r1 + (ch - 4) * 8;
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const float4 dl = st[T / 4 + ch * 2 + j];
              float2 x = add2(make_float2(__uint_as_float(g[j * 4]), __uint_as_float(g[j * 4 + 1])), make_float2(dl.x, dl.y));
              float2 y = add2(make_float2(__uint_as_float(g[j * 4 + 2]), __uint_as_float(g[j * 4 + 3])), make_float2(dl.z, dl.w));
              x = mul2(x, make_float2(__uint_as_float(pv[j * 4]), __uint_as_float(pv[j * 4 + 1])));
              y = mul2(y, make_float2(__uint_as_float(pv[j * 4 + 2]), __uint_as_float(pv[j * 4 + 3])));
              o[j * 2] = pack_bf16x2(x.x, x.y);
              o[j * 2 + 1] = pack_bf16x2(y.x, y.y);
            }
            *reinterpret_cast<uint4*>(sDS + ((ch ^ sw) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        tc_fence_before_sync();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(ds_ready);
          mbar_arrive(&st_empty[ph]);
        }
      }
      // dK, dV out (thread <-> key row, 64-column half)
      bf16* dk_row = p.dk + (long long)t.b * p.dk_sb + (long long)kv_idx * p.dk_ss + (long long)t.hkv * p.dk_sh + col0;
      bf16* dv_row = p.dv + (long long)t.b * p.dv_sb + (long long)kv_idx * p.dv_ss + (long long)t.hkv * p.dv_sh + col0;
      if (n_iters == 0) {
        if (kv_ok) {
          for (int c = 0; c < 64; c += 8) {
            *reinterpret_cast<uint4*>(dk_row + c) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(dv_row + c) = make_uint4(0, 0, 0, 0);
          }
        }
      } else {
        if (ok) ok = mbar_wait(all_done, n_work & 1u, abort_flag, p.status, 904);
        if (ok) {
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < 64; c += 32) {
            uint32_t r[32], r2[32];
            tmem_ld32(t_lane + C_DK + (uint32_t)(col0 + c), r);
            tmem_ld32(t_lane + C_DV + (uint32_t)(col0 + c), r2);
            tmem_ld_wait();
            if (c == 32) {   // the accumulators may be overwritten by the next item's first MMAs
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(acc_free);
            }
            if (kv_ok) {
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                uint4 v, w;
                uint32_t* vv = reinterpret_cast<uint32_t*>(&v);
                uint32_t* ww = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  vv[j] = pack_bf16x2(__uint_as_float(r[g * 8 + 2 * j]) * p.scale, __uint_as_float(r[g * 8 + 2 * j + 1]) * p.scale);
                  ww[j] = pack_bf16x2(__uint_as_float(r2[g * 8 + 2 * j]), __uint_as_float(r2[g * 8 + 2 * j + 1]));
                }
                *reinterpret_cast<uint4*>(dk_row + c + g * 8) = v;
                *reinterpret_cast<uint4*>(dv_row + c + g * 8) = w;
              }
            }
          }
        }
      }
      if (n_iters > 0) ++n_work;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 13) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Row kernels before and after the main one: 16 lanes per (b, s, h) row, ROWS_PT rows per thread a block's worth apart, all
// loads of a thread in flight at once.  Bound by HBM: at B 2, S 4096, H 32 one warp per row with 8-byte loads took 58 us
// (pre-pass) and 48 us (conversion) for 268 and 201 MB; now 38 and 31 us.
constexpr int ROW_THREADS = 256, ROWS_PT = 4, ROWS_PER_BLOCK = ROW_THREADS / 16 * ROWS_PT;

// 16 bytes of a tensor that no TMA map has checked: in halves where its rows are only 8-byte aligned
__device__ __forceinline__ uint4 load16(const bf16* p, bool wide) {
  if (wide) return *reinterpret_cast<const uint4*>(p);
  const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
  return make_uint4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store16(bf16* p, uint4 v, bool wide) {
  if (wide) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
    *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
  }
}

__device__ __forceinline__ void row_coords(unsigned row, int S, int H, int& b, int& s, int& h) {
  const unsigned bs = row / (unsigned)H;
  h = (int)(row - bs * (unsigned)H);
  b = (int)(bs / (unsigned)S);
  s = (int)(bs - (unsigned)b * (unsigned)S);
}

// delta[b, h, s] = sum_d dO[b, s, h, d] * O[b, s, h, d], and the row of the dQ accumulator is cleared
__global__ void __launch_bounds__(ROW_THREADS)
    attn_delta_kernel(const bf16* __restrict__ o, long long o_sb, long long o_ss, long long o_sh,
                      const bf16* __restrict__ d_o, long long do_sb, long long do_ss, long long do_sh,
                      float* __restrict__ delta, float* __restrict__ dq_acc, int S, int H, unsigned rows, bool wide_o) {
  const int l16 = threadIdx.x & 15;
  const unsigned row0 = blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 4);
  int b[ROWS_PT], s[ROWS_PT], h[ROWS_PT];
  uint4 x[ROWS_PT], g[ROWS_PT];
#pragma unroll
  for (int k = 0; k < ROWS_PT; ++k) {
    const unsigned row = row0 + k * (ROW_THREADS / 16);
    x[k] = g[k] = make_uint4(0, 0, 0, 0);
    if (row < rows) {
      row_coords(row, S, H, b[k], s[k], h[k]);
      x[k] = load16(o + b[k] * o_sb + s[k] * o_ss + h[k] * o_sh + l16 * 8, wide_o);
      g[k] = *reinterpret_cast<const uint4*>(d_o + b[k] * do_sb + s[k] * do_ss + h[k] * do_sh + l16 * 8);
    }
  }
#pragma unroll
  for (int k = 0; k < ROWS_PT; ++k) {
    const unsigned row = row0 + k * (ROW_THREADS / 16);
    const uint32_t xw[4] = {x[k].x, x[k].y, x[k].z, x[k].w}, gw[4] = {g[k].x, g[k].y, g[k].z, g[k].w};
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 u = unpack_bf16x2(xw[j]), v = unpack_bf16x2(gw[j]);
      acc += u.x * v.x + u.y * v.y;
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (row < rows) {
      if (l16 == 0) delta[((long long)b[k] * H + h[k]) * S + s[k]] = acc;
      float4* z = reinterpret_cast<float4*>(dq_acc + (long long)row * 128) + l16;
      z[0] = z[16] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// dq[b, s, h, :] (bf16, strided) = scale * dq_accum[b, s, h, :] (fp32 contiguous)
__global__ void __launch_bounds__(ROW_THREADS)
    attn_dq_convert_kernel(const float* __restrict__ acc, bf16* __restrict__ dq, long long sb, long long ss, long long sh,
                           float scale, int S, int H, unsigned rows, bool wide) {
  const int l16 = threadIdx.x & 15;
  const unsigned row0 = blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 4);
  float4 v[ROWS_PT][2];
#pragma unroll
  for (int k = 0; k < ROWS_PT; ++k) {
    const unsigned row = row0 + k * (ROW_THREADS / 16);
    if (row < rows) {
      const float4* src = reinterpret_cast<const float4*>(acc + (long long)row * 128) + l16 * 2;
      v[k][0] = src[0];
      v[k][1] = src[1];
    }
  }
#pragma unroll
  for (int k = 0; k < ROWS_PT; ++k) {
    const unsigned row = row0 + k * (ROW_THREADS / 16);
    if (row < rows) {
      int b, s, h;
      row_coords(row, S, H, b, s, h);
      uint4 w;
      w.x = pack_bf16x2(v[k][0].x * scale, v[k][0].y * scale);
      w.y = pack_bf16x2(v[k][0].z * scale, v[k][0].w * scale);
      w.z = pack_bf16x2(v[k][1].x * scale, v[k][1].y * scale);
      w.w = pack_bf16x2(v[k][1].z * scale, v[k][1].w * scale);
      store16(dq + b * sb + s * ss + h * sh + l16 * 8, w, wide);
    }
  }
}

// fp32 dQ accumulator [B, S, H, 128] contiguous -> 4-D map (d, h, s, b), box 32 x 1 x 32 x 1 (128-byte rows)
static int encode_dq_map(CUtensorMap* m, float* acc, int B, int S, int H) {
  uint64_t dims[4] = {128, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t str[3] = {128 * 4, (uint64_t)H * 128 * 4, (uint64_t)S * H * 128 * 4};
  uint32_t box[4] = {32, 1, 32, 1};
  return encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, acc, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

static bool wide_rows(const void* p, long long sb, long long ss, long long sh) {
  return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)((sb | ss | sh) * 2)) & 15) == 0;
}

}  // namespace fa_bwd
}  // namespace ob

using namespace ob;

// Everything both entry points share: argument checks (all of them before the first enqueue), tensor maps, the delta
// pre-pass (which clears the dQ accumulator), the main kernel and the fp32 -> bf16 conversion of dQ.  `delta` ([B, H, S]) and
// `dq_accum` ([B, S, H, 128], fp32) are the two work buffers, whoever owns them.
static int launch_flash_bwd(const ObAttnArgs* a, float* delta, float* dq_accum, cudaStream_t stream) {
  if (a->D != 128) OB_FAIL(-2, "flash attention kernels are built for head_dim 128 (got %d)", a->D);
  if (a->B <= 0 || a->S <= 0 || a->H <= 0 || a->Hkv <= 0) OB_FAIL(-4, "empty problem");
  if (a->H % a->Hkv != 0) OB_FAIL(-3, "H (%d) must be a multiple of Hkv (%d)", a->H, a->Hkv);
  int Sk = 0;
  if (int g = ob_attn_check_geometry(a, &Sk))
    OB_FAIL(-5, "unsupported attention geometry (rule %d): S %d Sk %d q_off %d causal %d window %d", g, a->S, Sk,
            a->q_off, a->causal, a->window);
  CUtensorMap tq, tk, tv, tdo, tdq;
  int rc;
  if ((rc = encode_bshd_map(&tq, a->q, a->B, a->S, a->H, a->q_sb, a->q_ss, a->q_sh, 128))) return rc;
  if ((rc = encode_bshd_map(&tk, a->k, a->B, Sk, a->Hkv, a->k_sb, a->k_ss, a->k_sh, 128))) return rc;
  if ((rc = encode_bshd_map(&tv, a->v, a->B, Sk, a->Hkv, a->v_sb, a->v_ss, a->v_sh, 128))) return rc;
  if ((rc = encode_bshd_map(&tdo, a->d_o, a->B, a->S, a->H, a->do_sb, a->do_ss, a->do_sh, 128))) return rc;
  if ((rc = fa_bwd::encode_dq_map(&tdq, dq_accum, a->B, a->S, a->H))) return rc;
  // the shared-memory opt-in is a per-device attribute of the function
  static bool attr_set[64] = {};
  int dev = 0;
  OB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) OB_FAIL(-6, "device ordinal %d outside the supported range [0, 64)", dev);
  if (!attr_set[dev]) {
    OB_CUDA_OK(cudaFuncSetAttribute(fa_bwd::flash_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    fa_bwd::SMEM_BYTES));
    OB_CUDA_OK(cudaFuncSetAttribute(fa_bwd::flash_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    fa_bwd::SMEM_BYTES));
    attr_set[dev] = true;
  }

  const long long rows = (long long)a->B * a->S * a->H;
  if (rows > 0x7fffffffLL) OB_FAIL(-4, "%lld query rows exceed the index range", rows);
  const int kv_tiles = (Sk + 127) / 128;
  const long long slices = (long long)a->B * a->Hkv, items = slices * kv_tiles;
  if (items > 0x7fffffffLL) OB_FAIL(-4, "%lld key tiles exceed the grid", items);
  const unsigned nblk = (unsigned)((rows + fa_bwd::ROWS_PER_BLOCK - 1) / fa_bwd::ROWS_PER_BLOCK);
  fa_bwd::attn_delta_kernel<<<nblk, fa_bwd::ROW_THREADS, 0, stream>>>(
      reinterpret_cast<const bf16*>(a->o), a->o_sb, a->o_ss, a->o_sh, reinterpret_cast<const bf16*>(a->d_o), a->do_sb,
      a->do_ss, a->do_sh, delta, dq_accum, a->S, a->H, (unsigned)rows,
      fa_bwd::wide_rows(a->o, a->o_sb, a->o_ss, a->o_sh));
  OB_CUDA_OK(cudaGetLastError());

  fa_bwd::Params p;
  p.B = a->B; p.S = a->S; p.H = a->H; p.Hkv = a->Hkv;
  p.Sk = Sk; p.q_off = a->q_off;
  p.causal = a->causal; p.window = a->window;
  const float LOG2E = 1.4426950408889634f;
  p.scale = a->scale;
  p.scale_log2 = a->scale * LOG2E;
  p.scale_over_cap = a->softcap > 0.f ? a->scale / a->softcap : 0.f;
  p.cap_log2 = a->softcap * LOG2E;
  p.lse = a->lse;
  p.delta = delta;
  p.dk = reinterpret_cast<bf16*>(a->dk); p.dk_sb = a->dk_sb; p.dk_ss = a->dk_ss; p.dk_sh = a->dk_sh;
  p.dv = reinterpret_cast<bf16*>(a->dv); p.dv_sb = a->dv_sb; p.dv_ss = a->dv_ss; p.dv_sh = a->dv_sh;
  p.status = a->status;
  p.kv_tiles = kv_tiles;
  // Few items per SM: the longest loops of all slices first, or the last ones to start set the time.  Many: groups of eight
  // slices, whose Q / dO / dQ (8 MB per 1024 rows, times the heads per kv-head) stay in L2 while their key tiles run.
  p.group = items <= 4 * sm_count() ? (int)slices : 8;
  const auto kernel = a->softcap > 0.f ? fa_bwd::flash_bwd_kernel<true> : fa_bwd::flash_bwd_kernel<false>;
  kernel<<<(unsigned)items, fa_bwd::THREADS, fa_bwd::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, tdq, p);
  OB_CUDA_OK(cudaGetLastError());
  fa_bwd::attn_dq_convert_kernel<<<nblk, fa_bwd::ROW_THREADS, 0, stream>>>(
      dq_accum, reinterpret_cast<bf16*>(a->dq), a->dq_sb, a->dq_ss, a->dq_sh, a->scale, a->S, a->H, (unsigned)rows,
      fa_bwd::wide_rows(a->dq, a->dq_sb, a->dq_ss, a->dq_sh));
  OB_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int ob_flash_attn_bwd(const ObAttnArgs* a, cudaStream_t stream) {
  if (a == nullptr) OB_FAIL(-1, "null args");
  if (a->delta == nullptr || a->dq_accum == nullptr) OB_FAIL(-4, "backward needs the delta and dq_accum scratch buffers");
  return launch_flash_bwd(a, a->delta, a->dq_accum, stream);
}

// ---------------------------------------------------------------------------------------------------------------------
// Allocation-free variant (declared in flash_attn_noalloc.h)
// ---------------------------------------------------------------------------------------------------------------------
// The backward pass needs two work buffers besides its inputs and outputs: delta[B, H, S] and the fp32 dQ accumulator
// [B, S, H, 128].  ob_flash_attn_bwd() takes them from the caller.  The variant below keeps them in a fixed array that
// is part of the library image, for callers that have no way to obtain device memory of their own.
namespace ob {
namespace fa_bwd_static {

constexpr long long MAX_ROWS = OB_FLASH_BWD_STATIC_MAX_ROWS;             // B * S * H
constexpr long long SCRATCH_FLOATS = MAX_ROWS * 128 + MAX_ROWS;          // dQ accumulator, then delta

static __device__ __align__(256) float g_scratch[SCRATCH_FLOATS];

// In host code `g_scratch` is only a handle for the runtime, not an address a kernel may use; the device address is
// looked up once per device with cudaGetSymbolAddress and cached here.
constexpr int MAX_DEVICES = 64;
static float* g_scratch_dev[MAX_DEVICES] = {nullptr};

static int scratch_for_current_device(float** out) {
  int dev = -1;
  OB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) OB_FAIL(-21, "device ordinal %d outside the supported range [0, %d)", dev, MAX_DEVICES);
  if (g_scratch_dev[dev] == nullptr) {
    float* p = nullptr;
    OB_CUDA_OK(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_scratch));
    if (p == nullptr) OB_FAIL(-22, "cudaGetSymbolAddress returned a null scratch address");
    g_scratch_dev[dev] = p;
  }
  *out = g_scratch_dev[dev];
  return 0;
}

}  // namespace fa_bwd_static
}  // namespace ob

extern "C" int ob_flash_attn_bwd_static(const ObAttnArgs* a, cudaStream_t stream) {
  using namespace ob::fa_bwd_static;
  if (a == nullptr) OB_FAIL(-1, "null args");
  if (a->B <= 0 || a->S <= 0 || a->H <= 0 || a->Hkv <= 0) OB_FAIL(-4, "empty problem");
  const long long rows = (long long)a->B * a->S * a->H;
  if (rows > MAX_ROWS)
    OB_FAIL(-20, "B*S*H = %lld exceeds the %lld rows the built-in work area holds; use ob_flash_attn_bwd with "
                 "caller-provided buffers for larger problems", rows, (long long)MAX_ROWS);
  float* scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc) return rc;
  // dQ accumulator [rows, 128] first, delta [rows] after the accumulator's full-size region
  return launch_flash_bwd(a, scratch + MAX_ROWS * 128, scratch, stream);
}

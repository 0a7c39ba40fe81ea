// Causal grouped-query FlashAttention backward on tcgen05 / TMEM / TMA for sm_100a (head_dim 64).
//
// An item is 128 keys of one (batch, KV head): a CTA visits every (query head of the group, query tile)
// at or after its keys; dK and dV of the tile accumulate in TMEM over the whole GQA group, so they are
// written once and need no atomics (as in the reference kernel, nanonemo/kernels/cuda/flash_attn.cu:
// 176-340, which keeps them in registers). Per visit, five tensor-core products, on TRANSPOSED score tiles:
//     S^T = K Q^T           dP^T = V dO^T                     (M = keys, N = queries, K = head_dim)
//     P^T = exp(S^T*scale - L) ; dS^T = P^T * (dP^T - D) * scale   (256 compute threads, two per key row)
//     dV += P^T dO          dK += dS^T Q                      (M = keys, N = head_dim, K = queries)
//     dQ  = dS K                                              (M = queries, N = head_dim, K = keys)
// Keys as rows are how dV and dK want their A operand: P^T and dS^T go back into tensor memory over the scores and products they came
// from, as 16-bit values, and are multiplied from there. Only dS^T also goes to shared memory ([key][query], 128-byte swizzle), as the
// MN-major A operand of dQ. K is read K-major (S^T) and MN-major (dQ), Q and dO K-major (scores) and MN-major (dK, dV), without any
// transposed copy. dQ partial tiles leave through a swizzled fp32 staging tile and a TMA reduce-add
// (cp.reduce.async.bulk.tensor .add.f32) into an fp32 buffer that a small kernel converts at the end. D = rowsum(dO * O) is a pre-pass
// kernel in this file.
// 512 threads: warp 0 TMA producer, warp 1 MMA issuer, warp 2 fetches L and D of the visits' queries, warps 4..7 drain dQ, warps 8..15
// compute: two threads per key row, one for queries 0..63 of the tile and one for queries 64..127 (same TMEM lanes, different columns).
//
// Software pipeline. The score tile is double buffered in tensor memory (S0 | S1 | dP | dV | dK = 512 columns). Within a visit's score
// buffer P^T takes the outer 32 columns on either side and the dQ partial product the 64 between them. The compute warps only do
// A: P^T = exp(S^T scale - L)  and  B: dS^T = P^T (dP^T - D) scale;  the dQ tile leaves through four warps of its own:
//     compute :  A(n)                    B(n)                     A(n+1)   ...
//     tensor  :        S(n+1)   dV(n)          dQ(n) dK(n) dP(n+1)
//     drain   :  dQ(n-1)                                          dQ(n)
// S(n+1) needs only the drained buffer, so it is issued before dV(n) and is complete long before A(n+1); dP(n+1) before
// B(n+1). No block barrier is left in the loop: the compute warps meet the tensor core through mbarriers alone.
// What bounds a visit, by clock counters of one thread per role (cycles): with the queries as rows, and P and dS both written to and read
// from shared memory, 2980 (waits 690, A 1660, B 620) beside 368 KB of shared-memory traffic, 2900 cycles; now 272 KB, and about
// 3050 (waits 480, A 1700, of it 1024 exponentials on the special-function unit, B 850): one chain through A and B, whose latency two
// warps a scheduler do not hide. (A quarter or half of the exponentials as polynomials on the multiply-add pipe: no change.) Whole backward,
// us, queries as rows / keys as rows: B32 H12/4 T1024 303 / 283, B128 T256 184 / 174, B64 H8/8 T200 84 / 80, B2 H12/4 T333 35 / 33, B8 H12/4 T4096
// 697 / 702, where the card's power limit (1.63 GHz under this kernel) evens them out.
// Items follow one another in a CTA without a seam, as in the forward kernel (flash_fwd.cu): a block that is running takes over blocks that have not
// started, K and V of the next item have a tile of their own, its first scores are issued beside the last products, and the drain
// warps, idle two thirds of a visit, store dV and dK while the compute warps are in the next item. A CTA per item spent 8.8 us on set-up, first
// loads, the first visit's latencies, the epilogue and its store, as long as three visits and with an SM to itself. Whole backward in a
// row (the card's power limit included), us, a CTA per item / items in sequence: B200 T64 85.9 / 74.9, B64 T300 131.5 / 119.5, B64
// T512 222 / 203, B16 T1024 147 / 133, B32 T1024 315 / 293, B8 T4096 810 / 748.
// A grid of one wave has an instance of its own, whose compute warps, free when the visits are over, store dV and dK side by side: one after the
// other in the four drain warps they took longer than a CTA per item had. 8/8 heads, us, a CTA per item / drain warps / compute warps: B1 T64 9.4 / 9.8 / 9.3,
// B2 T100 9.7 / 10.1 / 9.6, B16 T128 13.1 / 13.3 / 12.8, B4 T512 18.2 / 17.8 / 17.1.
// All waits are bounded, except two: the register hand-over, which the launcher checks before it can start (nnb_flash_bwd_registers), and, in a
// cluster, the two barriers of all its threads at the end, which every role of every CTA reaches, after a wait that ran out too.
#include <cstdlib>
#include <initializer_list>
#include <type_traits>

#define NNB_PROF_THREAD 256  // a compute thread
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BQ = 128, BKV = 128, HD = 64;
// Four warpgroups: TMA + MMA issuers (and two idle warps), drain, 2 x compute. The block is launched with 512 x 128 registers (checked before the first launch); the
// compute warps keep 64 probabilities each and need more, so the others hand registers over: 104 + 104 + 2 x 152 = 4 x 128.
constexpr int kThreads = 512;
constexpr int kComputeThreads = 256, kDrainThreads = 128;
constexpr int kDrainWarp0 = 4, kComputeWarp0 = 8;
constexpr int kRegsIssue = 104, kRegsDrain = 104, kRegsCompute = 152, kRegsLaunch = 128;
constexpr int kRegsShares = kRegsIssue + kRegsDrain + 2 * kRegsCompute;  // one warpgroup each, two for compute
static_assert(kRegsShares == kThreads / 128 * kRegsLaunch, "the shares have to be the registers that the block is launched with");
constexpr int kTile16 = 128 * 64 * 2;     // a [128 x 64] 16-bit tile = 16 KB
constexpr int kStagesQ = 3;             // a stage is released when dK / dQ of its visit are done and refilled two visits ahead
// shared memory map (bytes)
constexpr int kOffK = 0 /* V behind it */, kOffQdO = 2 * kTile16;               // ring of (Q | dO)
constexpr int kOffdS = kOffQdO + kStagesQ * 2 * kTile16;                       // dS^T: [128 keys] x two groups of 64 queries
constexpr int kOffStage = kOffdS + 2 * kTile16;                                // fp32 [128 x 64] = 32 KB
constexpr int kOffKV1 = kOffStage + 2 * kTile16;                                // K and V of the next item (every other one)
constexpr int kOffBars = kOffKV1 + 2 * kTile16;
constexpr int kOffLD = kOffBars + 512;                                         // float [2 parities][2 (-L log2e, -D scale)][128]
constexpr int kSmem = kOffLD + 2 * 2 * BQ * 4;                                 // (nothing to spare for aligning the base: the kernel checks it)
static_assert(kSmem <= 227 * 1024, "one CTA per SM");
// tensor memory columns
constexpr int kColS = 0 /* two buffers: + 128 * (visit & 1) */, kColdP = 256, kColdV = 384, kColdK = 448, kTmemCols = 512;
// A visit's S^T buffer also holds its P^T, the queries 0..63 in columns [0, 32) and 64..127 in [96, 128), and between them its dQ
constexpr int kColdQ = kColS + 32;
__device__ __forceinline__ uint32_t col_of_queries(int k) { return k < 4 ? 8 * k : 96 + 8 * (k - 4); }  // 16 queries from 16 k, of P^T and dS^T

struct BParams {
  int B, H, KVH, T, n_q_tiles, group;
  float scale, scale_log2;
  const float* lse;    // [B, H, T]
  const float* delta;  // [B, H, T]
  uint32_t idesc_s, idesc_dkv, idesc_dq;
  int* status;
  // Optional inverse RoPE on dK (and on dQ in the convert kernel): fp32 tables [T, 32] of the forward rotation. When given,
  // the attention inputs were rotated by the producer of Q / K and the gradients leave here un-rotated, i.e. with respect to
  // the projection before RoPE, so no separate inverse-RoPE pass over the packed gradient is needed.
  const float* rope_cos;
  const float* rope_sin;
  // A cluster of `split` CTAs shares one key tile: each takes a part of its visits, and they add up their dK and dV at the end.
  int split;
  void *dk, *dv;                          // split > 1: written directly, strides as the launcher's
  long long dk_sb, dk_st, dk_sh, dv_sb, dv_st, dv_sh;
};

// SPLIT: a cluster shares a key tile (BParams). TAKE: the grid has more blocks than SMs, and blocks take over others (see flash_fwd.cu); never both.
template <bool F16, bool SPLIT = false, bool TAKE = false>
__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                 const __grid_constant__ CUtensorMap tmdQacc, const __grid_constant__ CUtensorMap tmdK,
                 const __grid_constant__ CUtensorMap tmdV, const BParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t s_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBars);
  // barriers: kv_full[2], kv_empty[2], q_full[3], q_empty[3], s_full[2], dp_full, dq_full, all_done, next_full[2] | by compute: p_written, ds_written, ld_empty[2] |
  // by drain: dq_read, acc_read | ld_full[2] | next_empty[2]
  const uint32_t bar_kv = smem_u32(bars), bar_kve = bar_kv + 16, bar_qf = bar_kve + 16, bar_qe = bar_qf + 8 * kStagesQ;
  const uint32_t bar_s = bar_qe + 8 * kStagesQ, bar_dp = bar_s + 16, bar_dq = bar_dp + 8, bar_fin = bar_dq + 8, bar_nf = bar_fin + 8;
  const uint32_t bar_p = bar_nf + 16, bar_ds = bar_p + 8, bar_le = bar_ds + 8, bar_dqr = bar_le + 16, bar_acc = bar_dqr + 8, bar_lf = bar_acc + 8, bar_ne = bar_lf + 16;
  constexpr int kBars = 4 + 2 * kStagesQ + 17;
  constexpr int kNextReaders = 2 + kDrainThreads / 32 + kComputeThreads / 32;  // warps that read which item is next: MMA, L / D, drain, compute
  const uint32_t answers = s_base + kOffBars + (kBars + 1) / 2 * 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBars + (kBars + 1) / 2 * 16 + 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* never_set = abort_flag + 1;
  static_assert(kBars <= 32 && (kBars + 1) / 2 * 16 + 32 + 12 <= 512, "barriers");
  float* s_ld = reinterpret_cast<float*>(smem + kOffLD);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool aligned = (s_base & 1023) == 0;  // (swizzled tiles; nothing runs otherwise)
  // An item is a key tile of one (batch, KV head), or a part of its visits. Longest-job-first over the whole grid: key tile 0 is visited by every
  // query tile, the last one by a single tile, and the key tile is the slowest-varying block index, so the heavy items all start first and the
  // kernel ends on the short ones.
  const int split = SPLIT ? p.split : 1;
  const int part = blockIdx.x % split;  // (rank in the cluster)
  struct Item { int kt, kvh, b, first_qt, n_qt, visit0, iters; };
  auto item_at = [&](int x, int y, int z) {
    Item i;
    i.kt = z; i.kvh = x / split; i.b = y;
    i.first_qt = (z * BKV) / BQ;                            // first query tile that can see these keys
    i.n_qt = p.n_q_tiles - i.first_qt;                      // query tiles per head of the group
    // visits are numbered head by head; this CTA's are [visit0, visit0 + iters)
    i.visit0 = i.n_qt * p.group * part / split;
    i.iters = i.n_qt * p.group * (part + 1) / split - i.visit0;
    return i;
  };
  const Item item0 = item_at(blockIdx.x, blockIdx.y, blockIdx.z);
  // The item after number k of this CTA: answer k, in slot k & 1. A warp reads it with next_item and lets the slot go. False: there is none.
  auto next_item = [&](int k, Item& i) {
    int x, y, z;
    const bool more = taken_block(answers + 16 * (k & 1), x, y, z);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_ne + 8 * (k & 1));
    if (more) i = item_at(x, y, z);
    return more;
  };
  auto next_known = [&](int k, volatile int* flag) { return mbar_wait(bar_nf + 8 * (k & 1), (k >> 1) & 1, flag); };

  if (warp == 0) {  // a barrier a lane
    const uint32_t bar = bar_kv + 8 * lane;
    const uint32_t count = bar < bar_p ? 1 : bar < bar_dqr ? kComputeThreads : bar < bar_lf ? kDrainThreads : bar < bar_ne ? 32 : kNextReaders;
    if (lane < kBars) mbar_init(bar, count);
    if (lane == 0) {
      *abort_flag = aligned ? 0 : 1;
      *never_set = 0;
    }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const float *g_lse = p.lse, *g_delta = p.delta, *g_cos = p.rope_cos, *g_sin = p.rope_sin;
  nnb_after_previous(g_lse, g_delta, g_cos, g_sin);
  int fail_role = aligned ? 0 : 6;
  // dK of key position t leaves through the transpose of the forward rotation: lo' = lo c + hi s, hi' = hi c - lo s
  auto unrotate = [&](uint32_t (&lo_)[32], uint32_t (&hi_)[32], int t) {
    const float *cr = g_cos + (size_t)t * (HD / 2), *sr = g_sin + (size_t)t * (HD / 2);
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 c4 = __ldg(reinterpret_cast<const float4*>(cr + i)), s4 = __ldg(reinterpret_cast<const float4*>(sr + i));
      const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float lo = __uint_as_float(lo_[i + e]), hi = __uint_as_float(hi_[i + e]);
        lo_[i + e] = __float_as_uint(lo * cc[e] + hi * ss[e]);
        hi_[i + e] = __float_as_uint(hi * cc[e] - lo * ss[e]);
      }
    }
  };

  // a row of 64 fp32 values, rounded, into a 16-bit tile
  auto stage16 = [&](uint8_t* row_at, int sw, const uint32_t (&r0)[32], const uint32_t (&r1)[32]) {
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = (jj & 3) * 8 + 2 * e;
        w[e] = pack2_16<F16>(__uint_as_float(jj < 4 ? r0[i] : r1[i]), __uint_as_float(jj < 4 ? r0[i + 1] : r1[i + 1]));
      }
      *reinterpret_cast<uint4*>(row_at + ((jj ^ sw) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  };

  if (warp < kDrainWarp0) {
    regs_dec<kRegsIssue>();
    if (warp == 0 && lane == 0 && aligned) {
      // ---------------------------------------------------------------- TMA producer
      Item it = item0;
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (int k = 0; ok; ++k) {
        const uint32_t kv = s_base + ((k & 1) ? kOffKV1 : kOffK);
        ok = mbar_wait(bar_kve + 8 * (k & 1), ((k >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar_kv + 8 * (k & 1), 2 * kTile16);
        tma_load_4d(kv, &tmK, bar_kv + 8 * (k & 1), 0, it.kvh, it.kt * BKV, it.b);
        tma_load_4d(kv + kTile16, &tmV, bar_kv + 8 * (k & 1), 0, it.kvh, it.kt * BKV, it.b);
        for (int n = 0; n < it.iters; ++n) {
          const int hq = it.kvh * p.group + (it.visit0 + n) / it.n_qt, qt = it.first_qt + (it.visit0 + n) % it.n_qt;
          ok = mbar_wait(bar_qe + 8 * s, ph ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t dst = s_base + kOffQdO + s * 2 * kTile16;
          mbar_expect_tx(bar_qf + 8 * s, 2 * kTile16);
          tma_load_4d(dst, &tmQ, bar_qf + 8 * s, 0, hq, qt * BQ, it.b);
          tma_load_4d(dst + kTile16, &tmdO, bar_qf + 8 * s, 0, hq, qt * BQ, it.b);
          if (++s == kStagesQ) { s = 0; ph ^= 1; }
        }
        if (!TAKE || !ok) break;
        // the next item: asked for when the last operands are on their way, not earlier (the longest CTA would take it)
        ok = mbar_wait(bar_ne + 8 * (k & 1), ((k >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        take_block(answers + 16 * (k & 1), bar_nf + 8 * (k & 1));
        ok = next_known(k, never_set);  // (has to arrive before the shared memory is given up, whatever the others do)
        if (!ok) *abort_flag = 1;
        int x, y, z;
        if (!ok || !taken_block(answers + 16 * (k & 1), x, y, z)) break;
        it = item_at(x, y, z);
      }
      if (!ok) fail_role = 1;
      nnb_release_next();
    }
    if (warp == 1 && aligned) {
      // ---------------------------------------------------------------- MMA issuer (warp-uniform: see umma_f16_elect)
      // Its waits are votes: then the compiler knows the answers to be the warp's (with an answer a lane B8 T4096 took 787 us instead of 740,
      // the products being issued later), and the warp leaves as one.
      const bool el = elect_one();
      const uint32_t sdS = s_base + kOffdS;
      // ring positions of visits n (cur) and n + 1 (nxt) and the phase of nxt, counted along instead of divided out
      uint32_t cur = 0, nxt = 0, nxt_ph = 0;
      auto stage_at = [&](uint32_t s) { return s_base + kOffQdO + s * 2 * kTile16; };
      auto k_of = [&](int k) { return s_base + ((k & 1) ? kOffKV1 : kOffK); };  // K of item k, V behind it
      // S^T(n) = K Q^T into score buffer n & 1 (K-major operands, 4 k-steps of 16 over head_dim)
      auto issue_s = [&](uint32_t n, uint32_t s, uint32_t sK) {
        const uint32_t sQ = stage_at(s);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          umma_f16_elect(el, tmem_base + kColS + (n & 1) * BKV, make_smem_desc(sK + k * 32, 16, 1024), make_smem_desc(sQ + k * 32, 16, 1024), p.idesc_s, k > 0);
        umma_commit_elect(el, bar_s + 8 * (n & 1));
      };
      // dP^T(n) = V dO^T
      auto issue_dp = [&](uint32_t s, uint32_t sV) {
        const uint32_t sdO = stage_at(s) + kTile16;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k)
          umma_f16_elect(el, tmem_base + kColdP, make_smem_desc(sV + k * 32, 16, 1024), make_smem_desc(sdO + k * 32, 16, 1024), p.idesc_s, k > 0);
        umma_commit_elect(el, bar_dp);
      };
      Item it = item0;
      bool ok = it.iters == 0 || (mbar_wait_warp(bar_kv, 0, abort_flag) && mbar_wait_warp(bar_qf, 0, abort_flag));
      if (ok && it.iters > 0) {
        tc_fence_after();
        issue_s(0, 0, k_of(0));
        issue_dp(0, k_of(0) + kTile16);
      }
      int item = 0, v = 0;  // number of the item, visit within it; n counts visits on over all items
      for (uint32_t n = 0; ok && it.iters > 0; ++n) {
        const uint32_t sQ = stage_at(cur), sdO = sQ + kTile16, sK = k_of(item);
        const bool first = v == 0, last = v == it.iters - 1;
        if (++nxt == kStagesQ) { nxt = 0; nxt_ph ^= 1; }
        // S^T(n + 1) goes into the other score buffer: its scores were read before bar_p(n - 1), its P^T(n - 1) is read by dV(n - 1),
        // which is ahead in order, and its dQ(n - 1) must have been drained. (Waited for in every visit, so that bar_dq is never two
        // phases ahead of the drain.)
        if (n >= 1 && !mbar_wait_warp(bar_dqr, (n - 1) & 1, abort_flag)) { ok = false; break; }
        Item next = it;
        bool known = !last, more = !last, s_next = false;
        const uint32_t sK_next = last ? k_of(item + 1) : sK;
        auto operands = [&](bool wait) {  // of visit n + 1, when it begins an item
          const uint32_t b = bar_kv + 8 * ((item + 1) & 1), ph = ((item + 1) >> 1) & 1;
          if (!wait) return mbar_test_warp(b, ph) && mbar_test_warp(bar_qf + 8 * nxt, nxt_ph);
          return mbar_wait_warp(b, ph, abort_flag) && mbar_wait_warp(bar_qf + 8 * nxt, nxt_ph, abort_flag);
        };
        if (!last) {
          if (!mbar_wait_warp(bar_qf + 8 * nxt, nxt_ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          issue_s(n + 1, nxt, sK);
          s_next = true;
        } else if (!TAKE) {
          known = true;
        } else if (mbar_test_warp(bar_nf + 8 * (item & 1), (item >> 1) & 1)) {  // the next item, if it is there already: else after this visit's products
          known = true;
          more = __all_sync(0xffffffffu, next_known(item, abort_flag)) && next_item(item, next);
          if (more && operands(false)) {
            operands(true);
            tc_fence_after();
            issue_s(n + 1, nxt, sK_next);
            s_next = true;
          }
        }
        if (!mbar_wait_warp(bar_p, n & 1, abort_flag)) { ok = false; break; }     // P^T(n) is in tensor memory, S^T(n) has been read
        if (first && item > 0 && !mbar_wait_warp(bar_acc, (item - 1) & 1, abort_flag)) { ok = false; break; }  // the dK and dV of the item before have been read
        tc_fence_after();
        // dV += P^T dO: A = P^T in tensor memory (16 queries = 8 columns per k-step), B = [query][hd] tile read MN-major (16 query rows =
        // 2048 bytes per step)
        const uint32_t buf = tmem_base + kColS + (n & 1) * BQ, tdS = tmem_base + kColdP;
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k)
          umma_f16_ts_elect(el, tmem_base + kColdV, buf + col_of_queries(k), make_smem_desc(sdO + k * 2048, kTile16, 1024), p.idesc_dkv,
                            (!first || k > 0) ? 1u : 0u);
        if (!mbar_wait_warp(bar_ds, n & 1, abort_flag)) { ok = false; break; }    // dS^T(n) is written, dP^T(n) has been read
        tc_fence_after();
        // dQ(n) = dS K into the middle of the score buffer of this visit: A = [key][query] tile read MN-major (M = queries: two groups of 64,
        // 16 KB apart), B = K tile read MN-major; 8 k-steps of 16 key rows
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)
          umma_f16_elect(el, tmem_base + kColdQ + (n & 1) * BQ, make_smem_desc(sdS + k * 2048, kTile16, 1024), make_smem_desc(sK + k * 2048, kTile16, 1024),
                   p.idesc_dq, k > 0);
        umma_commit_elect(el, bar_dq);        // before dK(n): the drain runs beside dK(n) and dP^T(n + 1)
        // dK += dS^T Q, operands as for dV
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k)
          umma_f16_ts_elect(el, tmem_base + kColdK, tdS + col_of_queries(k), make_smem_desc(sQ + k * 2048, kTile16, 1024), p.idesc_dkv,
                            (!first || k > 0) ? 1u : 0u);
        umma_commit_elect(el, bar_qe + 8 * cur);
        if (last) {
          umma_commit_elect(el, bar_fin);                      // every product of the item has been accumulated
          umma_commit_elect(el, bar_kve + 8 * (item & 1));     // its K and V have been read
          if (!known) {
            if (!__all_sync(0xffffffffu, next_known(item, abort_flag))) { ok = false; break; }
            more = next_item(item, next);
          }
          if (!more) break;
          if (!s_next) {
            if (!operands(true)) { ok = false; break; }
            tc_fence_after();
            issue_s(n + 1, nxt, sK_next);
          }
        }
        issue_dp(nxt, sK_next + kTile16);   // over dS^T(n), which dK(n), ahead in order, reads; Q / dO of visit n + 1 were awaited above
        cur = nxt;
        ++v;
        if (last) {
          it = next;
          ++item;
          v = 0;
        }
      }
      if (!ok && lane == 0) fail_role = 2;
    }
    if (warp == 2 && aligned) {
      // ---------------------------------------------------------------- L and D of a visit's 128 queries, up to two visits ahead:
      // -L log2(e) and -D scale, the addends of the packed multiply-adds
      constexpr float kLog2e = 1.4426950408889634f;
      Item it = item0;
      uint32_t n = 0;
      bool ok = true;
      for (int k = 0; ok; ++k) {
        const float* gL = g_lse + ((size_t)it.b * p.H + it.kvh * p.group + it.visit0 / it.n_qt) * p.T;
        const float* gD = g_delta + ((size_t)it.b * p.H + it.kvh * p.group + it.visit0 / it.n_qt) * p.T;
        int qt = it.first_qt + it.visit0 % it.n_qt;
        for (int v = 0; v < it.iters; ++v, ++n) {
          float l[4], d[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int qi = qt * BQ + i * 32 + lane;
            l[i] = qi < p.T ? -gL[qi] * kLog2e : 0.f;
            d[i] = qi < p.T ? -gD[qi] * p.scale : 0.f;
          }
          if (++qt == p.n_q_tiles) { qt = it.first_qt; gL += p.T; gD += p.T; }
          if (n >= 2) ok = mbar_wait(bar_le + 8 * (n & 1), ((n >> 1) - 1) & 1, abort_flag);
          if (!ok) break;
          float* dst = s_ld + (n & 1) * 2 * BQ + lane;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            dst[i * 32] = l[i];
            dst[BQ + i * 32] = d[i];
          }
          mbar_arrive(bar_lf + 8 * (n & 1));
        }
        if (!TAKE) break;
        ok = ok && next_known(k, abort_flag);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }  // (the lanes leave together)
        if (!next_item(k, it)) break;
      }
      if (!ok) fail_role = 5;
    }
    if constexpr (SPLIT) {  // every thread of the cluster meets twice: see the compute warps
      cluster_sync();
      cluster_sync();
    }
  } else if (warp < kComputeWarp0) {
    regs_dec<kRegsDrain>();
    // ------------------------------------------------------------------ drain warps: the dQ partial tile of every visit, dV and dK of every item
    // TMEM (score buffer m & 1) -> swizzled fp32 staging (two [128 x 32] boxes) -> TMA reduce-add into the fp32 accumulator
    const int row = (warp & 3) * 32 + lane, sw = row & 7;
    const bool leader = warp == kDrainWarp0 && lane == 0;
    const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* my_stage = smem + kOffStage + row * 128;
    Item it = item0;
    uint32_t m = 0;
    for (int k = 0;; ++k) {
      int hq = it.kvh * p.group + it.visit0 / it.n_qt, qt = it.first_qt + it.visit0 % it.n_qt;
      bool left = false;
      for (int v = 0; v < it.iters; ++v, ++m) {
        const bool ok = mbar_wait(bar_dq, m & 1, abort_flag);
        tc_fence_after();
        if (leader) tma_wait_group_read<0>();      // the previous reduce has finished reading the staging tile
        if (named_barrier_or(1, kDrainThreads, !ok)) { left = true; break; }  // all leave together
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(t_row + kColdQ + (m & 1) * BQ, r0);
        tmem_ld_32x32b_x32(t_row + kColdQ + (m & 1) * BQ + 32, r1);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(bar_dqr);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          *reinterpret_cast<uint4*>(my_stage + ((jj ^ sw) << 4)) = make_uint4(r0[4 * jj], r0[4 * jj + 1], r0[4 * jj + 2], r0[4 * jj + 3]);
          *reinterpret_cast<uint4*>(my_stage + kTile16 + ((jj ^ sw) << 4)) = make_uint4(r1[4 * jj], r1[4 * jj + 1], r1[4 * jj + 2], r1[4 * jj + 3]);
        }
        fence_proxy_async_smem();
        named_barrier_sync(1, kDrainThreads);
        if (leader) {
          tma_reduce_add_4d(&tmdQacc, s_base + kOffStage, 0, hq, qt * BQ, it.b);
          tma_reduce_add_4d(&tmdQacc, s_base + kOffStage + kTile16, 32, hq, qt * BQ, it.b);
          tma_commit_group();
        }
        if (++qt == p.n_q_tiles) { qt = it.first_qt; ++hq; }
      }
      if (left) { fail_role = 4; break; }
      if (!TAKE) break;
      // The item's dV and dK: TMEM -> 16-bit tiles in the staging tile's place -> TMA store, while the other roles are in the next item
      const bool ok = mbar_wait(bar_fin, k & 1, abort_flag) && next_known(k, abort_flag);
      tc_fence_after();
      if (leader) tma_wait_group_read<0>();
      if (named_barrier_or(1, kDrainThreads, !ok)) { fail_role = 4; break; }
      Item next = it;
      const bool more = next_item(k, next);
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(t_row + (which == 0 ? kColdV : kColdK), r0);
        tmem_ld_32x32b_x32(t_row + (which == 0 ? kColdV : kColdK) + 32, r1);
        tmem_ld_wait();
        if (which == 1) {
          tc_fence_before();
          mbar_arrive(bar_acc);
          if (p.rope_cos != nullptr && it.kt * BKV + row < p.T) unrotate(r0, r1, it.kt * BKV + row);
        }
        stage16(my_stage + which * kTile16, sw, r0, r1);
      }
      fence_proxy_async_smem();
      named_barrier_sync(1, kDrainThreads);
      if (leader) {
        tma_store_4d(&tmdV, s_base + kOffStage, 0, it.kvh, it.kt * BKV, it.b);
        tma_store_4d(&tmdK, s_base + kOffStage + kTile16, 0, it.kvh, it.kt * BKV, it.b);
        tma_commit_group();
      }
      if (!more) break;
      it = next;
    }
    if (leader) tma_wait_group<0>();
    if constexpr (SPLIT) {
      cluster_sync();
      cluster_sync();
    }
  } else {
    regs_inc<kRegsCompute>();
    // ------------------------------------------------------------------ compute warps (two threads per key row)
    const int half = (warp - kComputeWarp0) >> 2;  // 0: queries 0..63 / dV; 1: queries 64..127 / dK
    const int q = warp & 3, row = q * 32 + lane, sw = row & 7;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
    uint8_t* my_ds = smem + kOffdS + half * kTile16 + row * 128;
    // A thread works on 32 of its 64 queries and then on the others, in steps of 16. Each 32 leave their P^T (and dS^T) in 16 columns that
    // this thread has read already: for the upper half that takes its last 32 queries first.
    const int first = half * 32;
    auto query = [&](int c) { return (c < 2 ? first : 32 - first) + (c & 1) * 16; };  // first query of step c
    bool ok = true;
    NNB_PROF_DECL;
    Item it = item0;
    uint32_t n = 0;
    const uint64_t scale2 = pack_f32x2(p.scale, p.scale), scale_log2_2 = pack_f32x2(p.scale_log2, p.scale_log2);
    for (int k = 0;; ++k) {
      const int key = it.kt * BKV + row;
      int qt = it.first_qt + it.visit0 % it.n_qt;
      for (int v = 0; v < it.iters && ok; ++v, ++n) {
        NNB_PROF_T0;
        const int q0 = qt * BQ + half * 64;
        if (++qt == p.n_q_tiles) qt = it.first_qt;
        // Only tiles on the diagonal, past the end of the sequence, or with padded key rows need the
        // per-element mask; every other tile takes the branch-free version.
        const bool need_mask = q0 < it.kt * BKV + BKV - 1 || q0 + 64 > p.T || it.kt * BKV + BKV > p.T;
        const uint32_t t_buf = t_lane + kColS + (n & 1) * BQ, t_s = t_buf + half * 64, t_dp = t_lane + kColdP + half * 64;
        const float* sL = s_ld + (n & 1) * 2 * BQ + half * 64;
        float prob[64];  // P^T of this thread's 64 queries, kept in fp32 from phase A to phase B
        // ---- phase A: P^T = exp2(S^T scale log2e - L log2e)
        if (!mbar_wait(bar_lf + 8 * (n & 1), (n >> 1) & 1, abort_flag)) { ok = false; break; }
        if (!mbar_wait(bar_s + 8 * (n & 1), (n >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        NNB_PROF_ADD(0);
        auto phase_a = [&](auto masked) {
          constexpr bool kMask = decltype(masked)::value;
          uint32_t rs[2][16], pk[16];  // 16 columns at a time, the next load in flight while these are worked on
          tmem_ld_32x32b_x16(t_s + query(0), rs[0]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const ulonglong2* l4 = reinterpret_cast<const ulonglong2*>(sL + query(c));
            const ulonglong2 l[4] = {l4[0], l4[1], l4[2], l4[3]};  // (arrive while the scores are waited for)
            tmem_ld_wait(rs[c & 1]);
            if (c < 3) tmem_ld_32x32b_x16(t_s + query(c + 1), rs[(c + 1) & 1]);
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const uint64_t s2 = pack_f32x2(__uint_as_float(rs[c & 1][i]), __uint_as_float(rs[c & 1][i + 1]));
              const float2 e = unpack_f32x2(fma_f32x2(s2, scale_log2_2, (i & 2) ? l[i / 4].y : l[i / 4].x));
              float p0 = exp2f(e.x), p1 = exp2f(e.y);
              if (kMask) {
                const int qi = q0 + query(c) + i;
                p0 = (key <= qi && qi < p.T && key < p.T) ? p0 : 0.f;
                p1 = (key <= qi + 1 && qi + 1 < p.T && key < p.T) ? p1 : 0.f;
              }
              prob[c * 16 + i] = p0;
              prob[c * 16 + i + 1] = p1;
              pk[(c & 1) * 8 + (i >> 1)] = pack2_16<F16>(p0, p1);
            }
            if (c & 1) tmem_st_32x32b_x16(t_buf + half * 96 + query(c - 1) / 2, pk);
          }
        };
        if (need_mask) phase_a(std::true_type{});
        else phase_a(std::false_type{});
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(bar_p);
        NNB_PROF_ADD(1);
        // ---- phase B: dS^T = P^T (dP^T scale - D scale)
        // (dP^T(n) was issued after dK(n - 1) and dQ(n - 1): once it is complete they have read dS^T)
        if (!mbar_wait(bar_dp, n & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        NNB_PROF_ADD(2);
        uint32_t rp[2][16], dk[16];
        tmem_ld_32x32b_x16(t_dp + query(0), rp[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const ulonglong2* d4 = reinterpret_cast<const ulonglong2*>(sL + BQ + query(c));
          const ulonglong2 d[4] = {d4[0], d4[1], d4[2], d4[3]};
          tmem_ld_wait(rp[c & 1]);
          if (c < 3) tmem_ld_32x32b_x16(t_dp + query(c + 1), rp[(c + 1) & 1]);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const uint64_t t = fma_f32x2(pack_f32x2(__uint_as_float(rp[c & 1][i]), __uint_as_float(rp[c & 1][i + 1])), scale2, (i & 2) ? d[i / 4].y : d[i / 4].x);
            const float2 g = unpack_f32x2(mul_f32x2(pack_f32x2(prob[c * 16 + i], prob[c * 16 + i + 1]), t));
            dk[(c & 1) * 8 + (i >> 1)] = pack2_16<F16>(g.x, g.y);
          }
#pragma unroll
          for (int jj = 0; jj < 2; ++jj)
            *reinterpret_cast<uint4*>(my_ds + (((query(c) / 8 + jj) ^ sw) << 4)) =
                make_uint4(dk[(c & 1) * 8 + 4 * jj], dk[(c & 1) * 8 + 4 * jj + 1], dk[(c & 1) * 8 + 4 * jj + 2], dk[(c & 1) * 8 + 4 * jj + 3]);
          if (c & 1) tmem_st_32x32b_x16(t_lane + kColdP + half * 96 + query(c - 1) / 2, dk);
        }
        mbar_arrive(bar_le + 8 * (n & 1));
        fence_proxy_async_smem();
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(bar_ds);
        NNB_PROF_ADD(3);
      }
      if (!TAKE) break;
      ok = ok && next_known(k, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }  // (the lanes leave together)
      if (!next_item(k, it)) break;
    }
    NNB_PROF_FLUSH_N(n);
    if (!ok) fail_role = 3;
    if constexpr (!SPLIT && !TAKE) {  // Nothing follows the CTA's one item: these warps are free, and do dV (half 0) and dK (half 1) at the same time
      ok = ok && mbar_wait(bar_fin, 0, abort_flag);
      tc_fence_after();
      if (named_barrier_or(2, kComputeThreads, !ok)) {  // all leave together
        fail_role = 3;
      } else {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(t_lane + (half == 0 ? kColdV : kColdK), r0);
        tmem_ld_32x32b_x32(t_lane + (half == 0 ? kColdV : kColdK) + 32, r1);
        tmem_ld_wait();
        if (half == 1 && p.rope_cos != nullptr && it.kt * BKV + row < p.T) unrotate(r0, r1, it.kt * BKV + row);
        stage16(my_ds, sw, r0, r1);  // (every product that read dS^T is complete)
        fence_proxy_async_smem();
        named_barrier_sync(2, kComputeThreads);
        if (half == 0 && row == 0) {
          tma_store_4d(&tmdV, s_base + kOffdS, 0, it.kvh, it.kt * BKV, it.b);
          tma_store_4d(&tmdK, s_base + kOffdS + kTile16, 0, it.kvh, it.kt * BKV, it.b);
          tma_commit_group();
          tma_wait_group<0>();
        }
      }
    }
    if constexpr (SPLIT) {
      // dV (half 0) and dK (half 1) of this CTA's visits: TMEM -> fp32 tiles in the ring, which every CTA of the cluster then reads for the rows it
      // adds up and stores
      const int iters = it.iters;
      if (ok && iters > 0 && !mbar_wait(bar_fin, 0, abort_flag)) ok = false;
      tc_fence_after();
      if (named_barrier_or(2, kComputeThreads, !ok)) {  // all leave together
        ok = false;
        fail_role = 3;
      }
      if (ok) {
        uint32_t r0[32], r1[32];
        if (iters > 0) {
          tmem_ld_32x32b_x32(t_lane + (half == 0 ? kColdV : kColdK), r0);
          tmem_ld_32x32b_x32(t_lane + (half == 0 ? kColdV : kColdK) + 32, r1);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r0[i] = r1[i] = 0u;
        }
        if (half == 1 && p.rope_cos != nullptr && it.kt * BKV + row < p.T) unrotate(r0, r1, it.kt * BKV + row);
        uint8_t* mine = smem + kOffQdO + half * 2 * kTile16 + row * 256;  // [128 x 64] fp32, 16-byte units swizzled by the row
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          *reinterpret_cast<uint4*>(mine + ((u ^ sw) << 4)) = make_uint4(r0[4 * u], r0[4 * u + 1], r0[4 * u + 2], r0[4 * u + 3]);
          *reinterpret_cast<uint4*>(mine + 128 + ((u ^ sw) << 4)) = make_uint4(r1[4 * u], r1[4 * u + 1], r1[4 * u + 2], r1[4 * u + 3]);
        }
      }
      cluster_sync();  // every CTA's tiles are written
      // 2 tensors x 128 rows x 16 units of four values, 256 units at a time, dealt out to the CTAs; added in the order of the parts
      if (ok) {
        const uint32_t tiles = s_base + kOffQdO;
        for (int u = part * kComputeThreads + (int)threadIdx.x - kComputeWarp0 * 32; u < 2 * BKV * 16; u += kComputeThreads * split) {
          const int which = u >> 11, r = (u >> 4) & (BKV - 1), c = u & 15, t = it.kt * BKV + r;
          const uint32_t at = tiles + which * 2 * kTile16 + r * 256 + (c >> 3) * 128 + (((c & 7) ^ (r & 7)) << 4);
          float4 v = load_cluster(at, 0);
          for (int k = 1; k < split; ++k) {
            const float4 w = load_cluster(at, k);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
          }
          if (t < p.T) {
            uint16_t* out = which == 0 ? static_cast<uint16_t*>(p.dv) + it.b * p.dv_sb + t * p.dv_st + it.kvh * p.dv_sh
                                       : static_cast<uint16_t*>(p.dk) + it.b * p.dk_sb + t * p.dk_st + it.kvh * p.dk_sh;
            *reinterpret_cast<uint2*>(out + c * 4) = make_uint2(pack2_16<F16>(v.x, v.y), pack2_16<F16>(v.z, v.w));
          }
        }
      }
      cluster_sync();  // ... and read
    }
  }

  if (fail_role != 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, 3) == 0) {
      p.status[1] = fail_role;
      p.status[2] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
      p.status[3] = 0;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// delta[b, h, t] = sum_d dO[b, t, h, d] * O[b, t, h, d]; 8 lanes per (b, t, h) row of 64 elements,
// 16 bytes per lane per tensor. The same pass clears the fp32 dQ accumulator (its rows are visited in the same order).
template <typename T16>
__global__ void flash_delta_kernel(const T16* __restrict__ o, const T16* __restrict__ d_o,
                                   float* __restrict__ delta, float* __restrict__ dq_acc, int B, int T, int H, long long o_sb, long long o_st,
                                   long long o_sh, long long do_sb, long long do_st, long long do_sh) {
  nnb_after_previous(o, d_o, delta, dq_acc);
  nnb_release_next();
  const long long gid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long w = gid >> 3;
  const int sub = threadIdx.x & 7;
  const long long rows = (long long)B * T * H;
  float s = 0.f;
  int h = 0, t = 0, b = 0;
  if (w < rows) {
    h = (int)(w % H);
    const long long bt = w / H;
    t = (int)(bt % T);
    b = (int)(bt / T);
    float a[8], g[8];
    Chunk8<T16>::load(o + b * o_sb + t * o_st + h * o_sh + sub * 8, a);
    Chunk8<T16>::load(d_o + b * do_sb + t * do_st + h * do_sh + sub * 8, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += a[i] * g[i];
    float4* z = reinterpret_cast<float4*>(dq_acc + w * HD + sub * 8);
    z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if (w < rows && sub == 0) delta[((size_t)b * H + h) * T + t] = s;
}

// dq[b, t, h, :] (bf16, strided) = dq_acc[b, t, h, :] (fp32, contiguous); with tables, the inverse RoPE of position t is
// applied on the way (columns j and j + 32 are partners, so one thread converts 8 + 8 elements).
template <typename T16>
__global__ void flash_dq_convert_kernel(const float* __restrict__ acc, T16* __restrict__ dq, long long rows, int H,
                                        int T, long long sb, long long st, long long sh, const float* __restrict__ rope_cos,
                                        const float* __restrict__ rope_sin) {
  nnb_after_previous(acc, dq, rope_cos, rope_sin);
  nnb_release_next();
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;  // one thread per 8 + 8 elements
  const long long total = rows * (HD / 16);
  if (idx >= total) return;
  const long long r = idx / (HD / 16);
  const int j = (int)(idx % (HD / 16)) * 8;
  const int h = (int)(r % H);
  const long long bt = r / H;
  const int t = (int)(bt % T);
  const long long b = bt / T;
  float lo[8], hi[8];
  Chunk8<float>::load(acc + r * HD + j, lo);
  Chunk8<float>::load(acc + r * HD + HD / 2 + j, hi);
  if (rope_cos != nullptr) {
    float c[8], s[8];
    Chunk8<float>::load(rope_cos + (size_t)t * (HD / 2) + j, c);
    Chunk8<float>::load(rope_sin + (size_t)t * (HD / 2) + j, s);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float a = lo[i], bb = hi[i];
      lo[i] = a * c[i] + bb * s[i];
      hi[i] = bb * c[i] - a * s[i];
    }
  }
  T16* dst = dq + b * sb + t * st + h * sh;
  Chunk8<T16>::store(dst + j, lo);
  Chunk8<T16>::store(dst + HD / 2 + j, hi);
}

}  // namespace

int nnb_flash_bwd_t_impl(int hd, const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse, void* delta,
                          void* dq_acc, void* dq, void* dk, void* dv, int B, int T, int H, int KVH, const long long* qs,
                          const long long* ks, const long long* vs, const long long* os, const long long* dos, const long long* dqs,
                          const long long* dks, const long long* dvs, float scale, int dtype, int in_order, void* status, cudaStream_t st);

#ifdef NNB_PROFILE
extern "C" int nnb_flash_bwd_prof_read(unsigned long long* out) { return (int)cudaMemcpyFromSymbol(out, g_flash_prof, sizeof(g_flash_prof)); }
#endif

// Whether a block that is launched with `regs` registers a thread can hand them over as flash_bwd_kernel does. The increase waits,
// without a limit, for registers that the other warpgroups give up: in a build with fewer of them (another compiler, a register
// limit among its flags) it would never end, so the launcher refuses such a build.
extern "C" int nnb_flash_bwd_registers(int regs) {
  NNB_REQUIRE(regs * (kThreads / 128) >= kRegsShares, "flash_bwd: built with %d registers a thread, the hand-over needs %d", regs, kRegsLaunch);
  return 0;
}

// The rule on its own (head_dim 64: 128 queries a visit, 128: 64), for tests.
extern "C" int nnb_flash_bwd_split(int T, int query_rows, long long kv_heads, int group, int sms) { return nnb_visits_split(T, query_rows, kv_heads, group, sms); }

template <bool F16>
static int configure_bwd() {
  for (auto kernel : {flash_bwd_kernel<F16>, flash_bwd_kernel<F16, true>, flash_bwd_kernel<F16, false, true>}) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) {
      nnb_set_error("flash_bwd: cannot reserve %d bytes of shared memory", kSmem);
      return -3;
    }
    if (int rc = nnb_flash_bwd_registers(a.numRegs)) return rc;
  }
  return 0;
}

// All tensors are [B, T, heads, 64] views given by element strides (contiguous last dim), bf16 or fp16 (one dtype for all).
// lse: fp32 [B, H, T] from the forward pass; delta: fp32 [B, H, T] scratch (written here);
// dq_acc: fp32 [B, T, H, hd] contiguous scratch (cleared by the delta pre-pass; partial tiles are reduce-added into it).
// in_order: dK and dV are summed in the order of the queries, one CTA a key tile, also where CTAs that share a tile and add up their parts
// would be faster.
// rope_cos / rope_sin: null, or fp32 [T, 32] tables: dQ and dK are then returned through the inverse rotation (head_dim 64).
extern "C" int nnb_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse,
                             void* delta, void* dq_acc, void* dq, void* dk, void* dv, int B, int T, int H, int KVH, int hd,
                             long long q_sb, long long q_st, long long q_sh, long long k_sb, long long k_st, long long k_sh,
                             long long v_sb, long long v_st, long long v_sh, long long o_sb, long long o_st, long long o_sh,
                             long long do_sb, long long do_st, long long do_sh, long long dq_sb, long long dq_st,
                             long long dq_sh, long long dk_sb, long long dk_st, long long dk_sh, long long dv_sb,
                             long long dv_st, long long dv_sh, float scale, int dtype, const void* rope_cos, const void* rope_sin,
                             int in_order, void* status, cudaStream_t st) {
  NNB_REQUIRE(hd == HD || hd == 128, "flash_bwd: head_dim %d not supported (64, 128)", hd);
  NNB_REQUIRE(dtype == NNB_BF16 || dtype == NNB_F16, "flash_bwd: bf16 or fp16 only (dtype code %d)", dtype);
  const bool f16 = dtype == NNB_F16;
  NNB_REQUIRE(H % KVH == 0 && B > 0 && T > 0, "flash_bwd: bad shape");
  // head_dim 128 runs on the transposed-tile kernel (flash_bwd_t.cu). It also serves head_dim 64
  // (NANONEMO_FLASH_BWD=transposed), but there the 128 x 128 tiles of this file measured faster (283 vs 361 us at
  // B32 H12/4 T1024; 702 vs 1058 us at B8 T4096): with 64-wide tiles every product has N = 64 and is bound by shared-memory operand reads.
  static const bool square = [] { const char* e = getenv("NANONEMO_FLASH_BWD"); return !(e && e[0] == 't'); }();
  NNB_REQUIRE((rope_cos == nullptr) == (rope_sin == nullptr), "flash_bwd: give both RoPE tables or neither");
  NNB_REQUIRE(rope_cos == nullptr || (hd == HD && square && nnb_aligned16(rope_cos) && nnb_aligned16(rope_sin)),
              "flash_bwd: the fused inverse RoPE exists for head_dim 64 on the 128 x 128 kernel only");
  if (hd == 128 || !square) {
    const long long qs[3] = {q_sb, q_st, q_sh}, ks[3] = {k_sb, k_st, k_sh}, vs[3] = {v_sb, v_st, v_sh}, os[3] = {o_sb, o_st, o_sh};
    const long long dos[3] = {do_sb, do_st, do_sh}, dqs[3] = {dq_sb, dq_st, dq_sh}, dks[3] = {dk_sb, dk_st, dk_sh};
    const long long dvs[3] = {dv_sb, dv_st, dv_sh};
    return nnb_flash_bwd_t_impl(hd, q, k, v, o, d_o, lse, delta, dq_acc, dq, dk, dv, B, T, H, KVH, qs, ks, vs, os, dos, dqs, dks, dvs,
                                scale, dtype, in_order, status, st);
  }
  const CUtensorMapDataType dt = f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv;
  if (!nnb_make_tmap_4d(&tq, dt, 2, q, hd, H, T, B, q_sh * 2, q_st * 2, q_sb * 2, 64, 1, BQ, "flash_bwd Q")) return -4;
  if (!nnb_make_tmap_4d(&tk, dt, 2, k, hd, KVH, T, B, k_sh * 2, k_st * 2, k_sb * 2, 64, 1, BKV, "flash_bwd K")) return -4;
  if (!nnb_make_tmap_4d(&tv, dt, 2, v, hd, KVH, T, B, v_sh * 2, v_st * 2, v_sb * 2, 64, 1, BKV, "flash_bwd V")) return -4;
  if (!nnb_make_tmap_4d(&tdo, dt, 2, d_o, hd, H, T, B, do_sh * 2, do_st * 2, do_sb * 2, 64, 1, BQ, "flash_bwd dO")) return -4;
  if (!nnb_make_tmap_4d(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dq_acc, hd, H, T, B, (uint64_t)hd * 4, (uint64_t)H * hd * 4,
                        (uint64_t)T * H * hd * 4, 32, 1, BQ, "flash_bwd dQ acc")) return -4;
  if (!nnb_make_tmap_4d(&tdk, dt, 2, dk, hd, KVH, T, B, dk_sh * 2, dk_st * 2, dk_sb * 2, 64, 1, BKV, "flash_bwd dK")) return -4;
  if (!nnb_make_tmap_4d(&tdv, dt, 2, dv, hd, KVH, T, B, dv_sh * 2, dv_st * 2, dv_sb * 2, 64, 1, BKV, "flash_bwd dV")) return -4;

  const long long rows = (long long)B * T * H;
  const unsigned delta_blocks = (unsigned)((rows * 8 + 255) / 256);
  if (f16)
    nnb_launch_pre_pass(rows * HD, flash_delta_kernel<__half>, delta_blocks, 256, st, (const __half*)o, (const __half*)d_o, (float*)delta, (float*)dq_acc, B, T, H, o_sb,
                                                            o_st, o_sh, do_sb, do_st, do_sh);
  else
    nnb_launch_pre_pass(rows * HD, flash_delta_kernel<__nv_bfloat16>, delta_blocks, 256, st, (const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, (float*)delta,
                                                                   (float*)dq_acc, B, T, H, o_sb, o_st, o_sh, do_sb, do_st, do_sh);
  NNB_LAUNCH_OK("flash_delta");

  BParams p{};
  p.B = B; p.H = H; p.KVH = KVH; p.T = T;
  p.n_q_tiles = (T + BQ - 1) / BQ;
  p.group = H / KVH;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = static_cast<const float*>(lse);
  p.delta = static_cast<const float*>(delta);
  const int fmt = f16 ? 0 : 1;
  p.idesc_s = sm100::make_idesc_f16(fmt, 0, 0, BKV, BQ);
  p.idesc_dkv = sm100::make_idesc_f16(fmt, 0, 1, BKV, HD);
  p.idesc_dq = sm100::make_idesc_f16(fmt, 1, 1, BQ, HD);
  p.status = static_cast<int*>(status);
  p.rope_cos = static_cast<const float*>(rope_cos);
  p.rope_sin = static_cast<const float*>(rope_sin);
  static bool configured = false;
  if (!configured) {
    if (int rc = configure_bwd<false>()) return rc;
    if (int rc = configure_bwd<true>()) return rc;
    configured = true;
  }
  p.split = in_order ? 1 : nnb_visits_split(T, BQ, (long long)KVH * B, p.group, nnb_num_sms());
  p.dk = dk; p.dk_sb = dk_sb; p.dk_st = dk_st; p.dk_sh = dk_sh;
  p.dv = dv; p.dv_sb = dv_sb; p.dv_st = dv_st; p.dv_sh = dv_sh;
  dim3 grid(KVH * p.split, B, (T + BKV - 1) / BKV);
  // A grid that runs at once has nothing to take over: its instance leaves dV and dK to the compute warps, which have nothing to do by then.
  const bool take = (long long)KVH * B * grid.z > nnb_num_sms();
  if (p.split > 1)
    nnb_launch_clusters(f16 ? flash_bwd_kernel<true, true> : flash_bwd_kernel<false, true>, p.split, grid, kThreads, kSmem, st, tq, tk, tv, tdo, tdq, tdk, tdv, p);
  // (full grids in plain stream order: an early start measured the same, B32 H12/4 T1024 285-287 us in either form, B128 T256 178-180 / 180)
  else if (take) (f16 ? flash_bwd_kernel<true, false, true> : flash_bwd_kernel<false, false, true>)<<<grid, kThreads, kSmem, st>>>(tq, tk, tv, tdo, tdq, tdk, tdv, p);
  else if (f16) flash_bwd_kernel<true><<<grid, kThreads, kSmem, st>>>(tq, tk, tv, tdo, tdq, tdk, tdv, p);
  else flash_bwd_kernel<false><<<grid, kThreads, kSmem, st>>>(tq, tk, tv, tdo, tdq, tdk, tdv, p);
  NNB_LAUNCH_OK("flash_bwd");
  const unsigned conv_blocks = (unsigned)((rows * (HD / 16) + 255) / 256);
  if (f16)
    nnb_launch(flash_dq_convert_kernel<__half>, conv_blocks, 256, 0, st, (const float*)dq_acc, (__half*)dq, rows, H, T, dq_sb, dq_st, dq_sh, p.rope_cos,
                                                                p.rope_sin);
  else
    nnb_launch(flash_dq_convert_kernel<__nv_bfloat16>, conv_blocks, 256, 0, st, (const float*)dq_acc, (__nv_bfloat16*)dq, rows, H, T, dq_sb, dq_st, dq_sh,
                                                                       p.rope_cos, p.rope_sin);
  NNB_LAUNCH_OK("flash_dq_convert");
  return 0;
}

// Causal grouped-query FlashAttention backward on TRANSPOSED score tiles (tcgen05 / TMEM / TMA, sm_100a), head_dim 64 and 128.
//
// One CTA owns 128 keys of one (batch, KV head) and visits every (query head of the group, 64-query block) at or after its
// keys. Per visit, on score tiles of 128 keys x 64 queries:
//     S^T  = K Q^T          dP^T = V dO^T                  (M = 128 keys,  N = 64 queries, K = head_dim)
//     P^T  = exp(S^T scale - L[q]) ; dS^T = P^T (dP^T - D[q]) scale     (256 threads: key row x half of the queries)
//     dV  += P^T dO         dK  += dS^T Q                  (M = 128 keys,  N = head_dim,   K = 64 queries)
//     dQ^T = K^T dS^T                                      (M = head_dim,  N = 64 queries, K = 128 keys)
// Why transposed: at head_dim 128 the 128 x 128 formulation of flash_bwd.cu does not fit tensor memory; here S^T is double buffered
// and everything fits in 64 + 64 (S^T) + 64 (dP^T) + 128 + 128 (dV, dK) + 64 (dQ^T) = 512 columns. And P^T, dS^T have the keys as rows,
// which is how dV and dK want their A operand: both are written back into tensor memory over the scores / products they came
// from and multiplied from there. Only dS^T also goes to shared memory (16-bit [key][query], 128-byte rows, swizzled), as the
// MN-major B operand of dQ^T. K is read K-major (S^T) and MN-major (dQ^T), Q / dO K-major (scores) and MN-major (dK, dV): no
// transposed copies. dQ^T (lanes = head_dim index; at head_dim 64 an M = 64 accumulator: row m in lane m % 16 of lane quarter
// m / 16) leaves through an fp32 [query][head_dim] staging tile — the transpose happens in the shared-memory write — and a TMA
// reduce-add into an fp32 buffer. dK / dV accumulate over the GQA group and are stored once.
// 512 threads: warp 0 TMA producer, warp 1 MMA issuer (warp-uniform, see umma_f16_elect), warp 2 fetches L and D of the visits'
// queries, warps 4..7 drain dQ^T, warps 8..15 compute. No block barrier in the loop:
//     compute :  A(n)                      B(n)                            A(n+1)  ...
//     tensor  :        S^T(n+1)   dV(n)           dQ^T(n) dK(n) dP^T(n+1)
//     drain   :  dQ^T(n-1)                                                 dQ^T(n)
// What bounded it: one chain. With single-buffered scores, the drain in the compute warps and a one-lane MMA issuer a visit
// took 5000 cycles (wait for the products 1245, P and dS 1371, wait for dQ^T 1630, drain 749) of which the tensor core needs
// about 1660. Backward at B8 H16/4 T2048 head_dim 128: 785 us then, 469 us now.
// Same contract as the reference backward (nanonemo/kernels/cuda/flash_attn.cu:176-340; head_dim 64 only).
#include <type_traits>

#define NNB_PROF_THREAD 256  // a compute thread
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BQ = 64, BKV = 128;
constexpr int kThreads = 512, kComputeThreads = 256, kDrainThreads = 128;
constexpr int kDrainWarp0 = 4, kComputeWarp0 = 8;
constexpr int kStagesQ = 3;            // ring of (Q | dO) blocks
constexpr int kHalfK = BKV * 64 * 2;   // [128 keys x 64] 16-bit tile = 16 KB
constexpr int kHalfQ = BQ * 64 * 2;    // [64 queries x 64] 16-bit tile = 8 KB
constexpr int kTmemCols = 512;

template <int HD>
struct Cfg {
  static constexpr int NH = HD / 64;                 // 64-wide head_dim groups (one TMA box / swizzle span each)
  static constexpr int kTileK = NH * kHalfK;         // K or V tile
  static constexpr int kStageQdO = 2 * NH * kHalfQ;  // Q block + dO block
  static constexpr int kOffK = 0, kOffV = kTileK, kOffQdO = 2 * kTileK;
  static constexpr int kOffdS = kOffQdO + kStagesQ * kStageQdO;
  static constexpr int kOffStage = kOffdS + kHalfK;            // fp32 [64 queries x HD]
  static constexpr int kOffBars = kOffStage + BQ * HD * 4;
  static constexpr int kOffLD = kOffBars + 256;                // float [2 parities][2 (-L log2e, -D scale)][64]
  static constexpr int kSmem = kOffLD + 2 * 2 * 64 * 4 + 1024;
  static constexpr int kColS = 0 /* + 64 * (visit & 1) */, kColdP = 128, kColdV = 192, kColdK = kColdV + HD, kColdQ = kColdK + HD;
  static_assert(kColdQ + 64 <= kTmemCols, "TMEM budget");
  static_assert(kStagesQ * kStageQdO >= 2 * kTileK, "the (Q | dO) ring doubles as the dV / dK staging area");
};

struct BParams {
  int B, H, KVH, T, n_q_blocks, group;
  float scale, scale_log2;
  const float* lse;
  const float* delta;
  uint32_t idesc_s, idesc_dkv, idesc_dq;
  int* status;
  // A cluster of `split` CTAs shares one key tile: each takes a part of its visits, and they add up their dK and dV at the end.
  int split;
  void* out[2];          // split > 1: dV, dK, written directly
  long long out_s[2][3];  // element strides {batch, t, head}
};

template <int HD, bool F16, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_t_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmdQacc, const __grid_constant__ CUtensorMap tmdK,
                   const __grid_constant__ CUtensorMap tmdV, const BParams p) {
  using C = Cfg<HD>;
  constexpr int NH = C::NH, S = kStagesQ;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBars);
  // barriers: kv, q_full[3], q_empty[3], s_full[2], p_written[2], ld_full[2], ld_empty[2], dp_full, ds_written, dq_full, dq_read, all_done
  const uint32_t bar_kv = smem_u32(bars), bar_qf = bar_kv + 8, bar_qe = bar_qf + 8 * S, bar_s = bar_qe + 8 * S, bar_p = bar_s + 16;
  const uint32_t bar_lf = bar_p + 16, bar_le = bar_lf + 16, bar_dp = bar_le + 16, bar_ds = bar_dp + 8, bar_dq = bar_ds + 8;
  const uint32_t bar_dqr = bar_dq + 8, bar_fin = bar_dqr + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1 + 2 * S + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_ld = reinterpret_cast<float*>(smem + C::kOffLD);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = SPLIT ? p.split : 1, part = blockIdx.x % split;  // (part = rank in the cluster)
  const int kt = blockIdx.z, kvh = blockIdx.x / split, b = blockIdx.y;  // key tile slowest: the heavy CTAs (early keys) are scheduled first
  const int first_qb = (kt * BKV) / BQ;
  const int n_qb = p.n_q_blocks - first_qb;
  // visits are numbered head by head; this CTA's are [visit0, visit0 + iters)
  const int visit0 = n_qb * p.group * part / split, iters = n_qb * p.group * (part + 1) / split - visit0;
  const int head0 = kvh * p.group + visit0 / n_qb, qb0 = first_qb + visit0 % n_qb;

  if (threadIdx.x == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_qf + 8 * s, 1);
      mbar_init(bar_qe + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_s + 8 * i, 1);
      mbar_init(bar_p + 8 * i, kComputeThreads);
      mbar_init(bar_lf + 8 * i, 32);
      mbar_init(bar_le + 8 * i, kComputeThreads);
    }
    mbar_init(bar_dp, 1);
    mbar_init(bar_ds, kComputeThreads);
    mbar_init(bar_dq, 1);
    mbar_init(bar_dqr, kDrainThreads);
    mbar_init(bar_fin, 1);
    *abort_flag = 0;
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
  const float *g_lse = p.lse, *g_delta = p.delta;
  nnb_after_previous(g_lse, g_delta);
  int fail_role = 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_expect_tx(bar_kv, 2 * C::kTileK);
#pragma unroll
      for (int g = 0; g < NH; ++g) {
        tma_load_4d(s_base + C::kOffK + g * kHalfK, &tmK, bar_kv, g * 64, kvh, kt * BKV, b);
        tma_load_4d(s_base + C::kOffV + g * kHalfK, &tmV, bar_kv, g * 64, kvh, kt * BKV, b);
      }
      for (int n = 0; n < iters; ++n) {
        const int hq = kvh * p.group + (visit0 + n) / n_qb, qb = first_qb + (visit0 + n) % n_qb;
        const uint32_t s = n % S, ph = (n / S) & 1;
        if (!mbar_wait(bar_qe + 8 * s, ph ^ 1, abort_flag)) { fail_role = 1; break; }
        const uint32_t dst = s_base + C::kOffQdO + s * C::kStageQdO;
        mbar_expect_tx(bar_qf + 8 * s, C::kStageQdO);
#pragma unroll
        for (int g = 0; g < NH; ++g) {
          tma_load_4d(dst + g * kHalfQ, &tmQ, bar_qf + 8 * s, g * 64, hq, qb * BQ, b);
          tma_load_4d(dst + (NH + g) * kHalfQ, &tmdO, bar_qf + 8 * s, g * 64, hq, qb * BQ, b);
        }
      }
      nnb_release_next();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (every lane runs the loop, one lane's instructions count)
    const bool el = elect_one();
    bool ok = mbar_wait(bar_kv, 0, abort_flag);
    const uint32_t sK = s_base + C::kOffK, sV = s_base + C::kOffV, sdS = s_base + C::kOffdS;
    uint32_t cur = 0, nxt = 0, nxt_ph = 0;  // ring positions of visits n and n + 1, and the phase of the latter
    auto stage_at = [&](uint32_t s) { return s_base + C::kOffQdO + s * C::kStageQdO; };
    // S^T = K Q^T of visit n into score buffer n & 1, dP^T = V dO^T: K-major operands, k-steps of 16 over head_dim
    auto issue_s = [&](int n, uint32_t s) {
      const uint32_t sQ = stage_at(s);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_f16_elect(el, tmem_base + C::kColS + 64 * (n & 1), make_smem_desc(sK + (k / 4) * kHalfK + (k % 4) * 32, 16, 1024),
                       make_smem_desc(sQ + (k / 4) * kHalfQ + (k % 4) * 32, 16, 1024), p.idesc_s, k > 0);
      umma_commit_elect(el, bar_s + 8 * (n & 1));
    };
    auto issue_dp = [&](uint32_t s) {
      const uint32_t sdO = stage_at(s) + NH * kHalfQ;
#pragma unroll
      for (int k = 0; k < HD / 16; ++k)
        umma_f16_elect(el, tmem_base + C::kColdP, make_smem_desc(sV + (k / 4) * kHalfK + (k % 4) * 32, 16, 1024),
                       make_smem_desc(sdO + (k / 4) * kHalfQ + (k % 4) * 32, 16, 1024), p.idesc_s, k > 0);
      umma_commit_elect(el, bar_dp);
    };
    if (ok && iters > 0) {
      ok = mbar_wait(bar_qf, 0, abort_flag);
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        issue_dp(0);
      }
    }
    for (int n = 0; n < iters && ok; ++n) {
      const uint32_t sQ = stage_at(cur), sdO = sQ + NH * kHalfQ;
      if (++nxt == S) { nxt = 0; nxt_ph ^= 1; }
      if (n + 1 < iters) {
        // the other score buffer: its scores were read before bar_p of visit n - 1, and dV(n - 1), which read P^T there, is ahead in order
        if (!mbar_wait(bar_qf + 8 * nxt, nxt_ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        issue_s(n + 1, nxt);
      }
      if (!mbar_wait(bar_p + 8 * (n & 1), (n >> 1) & 1, abort_flag)) { ok = false; break; }  // P^T(n) is in tensor memory
      tc_fence_after();
      // dV += P^T dO: A = P^T in tensor memory (16 queries = 8 columns per k-step; the two halves of the queries sit 32 columns apart,
      // each over the scores its own threads have read), B = [query][head_dim] block read MN-major (64-wide head_dim groups
      // kHalfQ apart; 16 query rows = 2048 bytes per step)
      const uint32_t tP = tmem_base + C::kColS + 64 * (n & 1), tdS = tmem_base + C::kColdP;
#pragma unroll
      for (int k = 0; k < BQ / 16; ++k)
        umma_f16_ts_elect(el, tmem_base + C::kColdV, tP + (k / 2) * 32 + (k % 2) * 8, make_smem_desc(sdO + k * 2048, kHalfQ, 1024),
                          p.idesc_dkv, (n > 0 || k > 0) ? 1u : 0u);
      if (!mbar_wait(bar_ds, n & 1, abort_flag)) { ok = false; break; }                     // dS^T(n) written, dP^T(n) read
      if (n > 0 && !mbar_wait(bar_dqr, (n - 1) & 1, abort_flag)) { ok = false; break; }     // dQ^T(n - 1) drained
      tc_fence_after();
      // dQ^T = K^T dS^T: A = K tile read MN-major (M = head_dim in 64-wide groups kHalfK apart), B = dS^T tile read MN-major
      // (N = 64 queries: one group); 8 k-steps of 16 key rows = 2048 bytes. First, so that its drain runs beside the others.
#pragma unroll
      for (int k = 0; k < BKV / 16; ++k)
        umma_f16_elect(el, tmem_base + C::kColdQ, make_smem_desc(sK + k * 2048, kHalfK, 1024), make_smem_desc(sdS + k * 2048, kHalfK, 1024),
                       p.idesc_dq, k > 0);
      umma_commit_elect(el, bar_dq);
      // dK += dS^T Q, operands as for dV
#pragma unroll
      for (int k = 0; k < BQ / 16; ++k)
        umma_f16_ts_elect(el, tmem_base + C::kColdK, tdS + (k / 2) * 32 + (k % 2) * 8, make_smem_desc(sQ + k * 2048, kHalfQ, 1024),
                          p.idesc_dkv, (n > 0 || k > 0) ? 1u : 0u);
      umma_commit_elect(el, bar_qe + 8 * cur);
      if (n + 1 < iters) issue_dp(nxt);  // over dS^T(n), which dK(n), ahead in order, reads
      else umma_commit_elect(el, bar_fin);  // one-shot: every product has been accumulated
      cur = nxt;
    }
    if (!ok && lane == 0) fail_role = 2;
  } else if (warp == 2) {
    // ------------------------------------------------------------------ L and D of a visit's 64 queries, up to two visits ahead:
    // -L log2(e) and -D scale, the addends of the packed multiply-adds
    constexpr float kLog2e = 1.4426950408889634f;
    const float* gL = g_lse + ((size_t)b * p.H + head0) * p.T;
    const float* gD = g_delta + ((size_t)b * p.H + head0) * p.T;
    int qb = qb0;
    for (int n = 0; n < iters; ++n) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int qi = qb * BQ + i * 32 + lane;
        v[i] = qi < p.T ? -gL[qi] * kLog2e : 0.f;
        v[2 + i] = qi < p.T ? -gD[qi] * p.scale : 0.f;
      }
      if (++qb == p.n_q_blocks) { qb = first_qb; gL += p.T; gD += p.T; }
      if (n >= 2 && !mbar_wait(bar_le + 8 * (n & 1), ((n >> 1) - 1) & 1, abort_flag)) { fail_role = 5; break; }
      float* dst = s_ld + (n & 1) * 128 + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i) dst[i * 32] = v[i];
      mbar_arrive(bar_lf + 8 * (n & 1));
    }
  } else if (warp >= kDrainWarp0 && warp < kComputeWarp0) {
    // ------------------------------------------------------------------ drain warps: dQ^T of every visit, TMEM (lane = head_dim index,
    // columns = queries) -> fp32 staging [query][head_dim] -> TMA reduce-add
    const int q4 = warp & 3;
    const bool leader = warp == kDrainWarp0 && lane == 0;
    const uint32_t t_row = tmem_base + ((uint32_t)(q4 * 32) << 16) + C::kColdQ;
    float* stage = reinterpret_cast<float*>(smem + C::kOffStage);
    int hq = head0, qb = qb0;
    for (int m = 0; m < iters; ++m) {
      const bool ok = mbar_wait(bar_dq, m & 1, abort_flag);
      tc_fence_after();
      if (leader) tma_wait_group_read<0>();      // the previous reduce has finished reading the staging tile
      if (named_barrier_or(1, kDrainThreads, !ok)) { fail_role = 4; break; }  // all leave together
      uint32_t r0[32], r1[32];
      tmem_ld_32x32b_x32(t_row, r0);
      tmem_ld_32x32b_x32(t_row + 32, r1);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(bar_dqr);
      if (HD == 128 || lane < 16) {              // HD 64: M = 64 accumulator, row 16 q4 + lane lives in lane `lane` of this quarter
        float* col = stage + (HD == 128 ? q4 * 32 + lane : q4 * 16 + lane);
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          col[c * HD] = __uint_as_float(r0[c]);
          col[(c + 32) * HD] = __uint_as_float(r1[c]);
        }
      }
      fence_proxy_async_smem();
      named_barrier_sync(1, kDrainThreads);
      if (leader) {
        tma_reduce_add_4d(&tmdQacc, s_base + C::kOffStage, 0, hq, qb * BQ, b);
        tma_commit_group();
      }
      if (++qb == p.n_q_blocks) { qb = first_qb; ++hq; }
    }
    if (leader) tma_wait_group<0>();
  } else if (warp >= kComputeWarp0) {
    // ------------------------------------------------------------------ compute warps: (key row) x (half of the 64 queries)
    const int half = (warp - kComputeWarp0) >> 2;
    const int q4 = warp & 3, row = q4 * 32 + lane, sw = row & 7;
    const bool leader = half == 0 && row == 0;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q4 * 32) << 16);
    const int key = kt * BKV + row;
    uint8_t* my_ds = smem + C::kOffdS + row * 128;
    const uint64_t scale2 = pack_f32x2(p.scale, p.scale), scale_log2_2 = pack_f32x2(p.scale_log2, p.scale_log2);
    bool ok = true;
    NNB_PROF_DECL;
    int qb = qb0;
    for (int n = 0; n < iters; ++n) {
      NNB_PROF_T0;
      const int q0 = qb * BQ;
      if (++qb == p.n_q_blocks) qb = first_qb;
      const int buf = n & 1;
      const ulonglong2* sL = reinterpret_cast<const ulonglong2*>(s_ld + buf * 128 + half * 32);
      const ulonglong2* sD = sL + 16;
      const uint32_t t_s = t_lane + C::kColS + 64 * buf + half * 32, t_dp = t_lane + C::kColdP + half * 32;
      // per-element mask only on the diagonal blocks, at the end of the sequence or for padded key rows
      const bool need_mask = q0 < kt * BKV + BKV - 1 || q0 + BQ > p.T || kt * BKV + BKV > p.T;
      float prob[32];  // P^T of this thread's 32 queries, kept in fp32 from phase A to phase B
      // ---- phase A: P^T = exp2(S^T scale log2e - L log2e)
      if (!mbar_wait(bar_lf + 8 * buf, (n >> 1) & 1, abort_flag)) { ok = false; break; }
      if (!mbar_wait(bar_s + 8 * buf, (n >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      NNB_PROF_ADD(0);
      auto phase_a = [&](auto masked) {
        constexpr bool kMask = decltype(masked)::value;
        uint32_t rs[2][16], pk[16];
        tmem_ld_32x32b_x16(t_s, rs[0]);
        tmem_ld_32x32b_x16(t_s + 16, rs[1]);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld_wait(rs[c]);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const ulonglong2 l = sL[c * 4 + i / 4];
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const uint64_t s2 = pack_f32x2(__uint_as_float(rs[c][i + e]), __uint_as_float(rs[c][i + e + 1]));
              const float2 x = unpack_f32x2(fma_f32x2(s2, scale_log2_2, e == 0 ? l.x : l.y));
              float p0 = exp2f(x.x), p1 = exp2f(x.y);
              if (kMask) {
                const int qi = q0 + half * 32 + c * 16 + i + e;
                p0 = (key <= qi && qi < p.T && key < p.T) ? p0 : 0.f;
                p1 = (key <= qi + 1 && qi + 1 < p.T && key < p.T) ? p1 : 0.f;
              }
              prob[c * 16 + i + e] = p0;
              prob[c * 16 + i + e + 1] = p1;
              pk[(c * 16 + i + e) >> 1] = pack2_16<F16>(p0, p1);
            }
          }
        }
        tmem_st_32x32b_x16(t_s, pk);
      };
      if (need_mask) phase_a(std::true_type{});
      else phase_a(std::false_type{});
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_p + 8 * buf);
      NNB_PROF_ADD(1);
      // ---- phase B: dS^T = P^T (dP^T scale - D scale)
      // (dP^T(n) was issued after dQ^T(n - 1) and dK(n - 1): once it is complete they have read dS^T)
      if (!mbar_wait(bar_dp, n & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      NNB_PROF_ADD(2);
      {
        uint32_t rp[2][16], dk[16];
        tmem_ld_32x32b_x16(t_dp, rp[0]);
        tmem_ld_32x32b_x16(t_dp + 16, rp[1]);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld_wait(rp[c]);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const ulonglong2 d = sD[c * 4 + i / 4];
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const uint64_t t = fma_f32x2(pack_f32x2(__uint_as_float(rp[c][i + e]), __uint_as_float(rp[c][i + e + 1])), scale2, e == 0 ? d.x : d.y);
              const float2 g = unpack_f32x2(mul_f32x2(pack_f32x2(prob[c * 16 + i + e], prob[c * 16 + i + e + 1]), t));
              dk[(c * 16 + i + e) >> 1] = pack2_16<F16>(g.x, g.y);
            }
          }
        }
        tmem_st_32x32b_x16(t_dp, dk);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          *reinterpret_cast<uint4*>(my_ds + (((half * 4 + jj) ^ sw) << 4)) = make_uint4(dk[4 * jj], dk[4 * jj + 1], dk[4 * jj + 2], dk[4 * jj + 3]);
      }
      mbar_arrive(bar_le + 8 * buf);
      fence_proxy_async_smem();
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_ds);
      NNB_PROF_ADD(3);
    }
    if (ok && iters > 0 && !mbar_wait(bar_fin, 0, abort_flag)) ok = false;
    tc_fence_after();
    if (named_barrier_or(2, kComputeThreads, !ok)) {  // all leave together
      ok = false;
      fail_role = 3;
    }
    NNB_PROF_FLUSH_N(iters);
    // dV then dK of this key tile: TMEM -> bf16 staging (the (Q | dO) ring: every load has been consumed) -> TMA store
    if constexpr (SPLIT) {
      // In a cluster: dV, then dK, as fp32 [128 x HD] in the ring (16-byte units swizzled by the row), from where every CTA reads the
      // units that it adds up, in the order of the parts, and stores. All threads of the cluster meet four times.
      const uint32_t tile = s_base + C::kOffQdO;
      for (int which = 0; which < 2; ++which) {
        if (ok) {
          uint8_t* mine = smem + C::kOffQdO + row * (HD * 4);
#pragma unroll
          for (int g = 0; g < NH; ++g) {  // this thread's half of every 64-wide head_dim group
            uint32_t r[32];
            if (iters > 0) {
              tmem_ld_32x32b_x32(t_lane + (which == 0 ? C::kColdV : C::kColdK) + g * 64 + half * 32, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
              *reinterpret_cast<uint4*>(mine + g * 256 + half * 128 + ((u ^ sw) << 4)) = make_uint4(r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
          }
        }
        cluster_sync();  // every CTA's tile is written
        if (ok) {
          for (int u = part * kComputeThreads + (int)threadIdx.x - kComputeWarp0 * 32; u < BKV * (HD / 4); u += kComputeThreads * split) {
            const int r = u / (HD / 4), c = u % (HD / 4), t = kt * BKV + r;
            const uint32_t at = tile + r * (HD * 4) + (c >> 3) * 128 + (((c & 7) ^ (r & 7)) << 4);
            float4 v = load_cluster(at, 0);
            for (int k = 1; k < split; ++k) {
              const float4 w = load_cluster(at, k);
              v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            }
            if (t < p.T) {
              uint16_t* out = static_cast<uint16_t*>(p.out[which]) + b * p.out_s[which][0] + t * p.out_s[which][1] + kvh * p.out_s[which][2];
              *reinterpret_cast<uint2*>(out + c * 4) = make_uint2(pack2_16<F16>(v.x, v.y), pack2_16<F16>(v.z, v.w));
            }
          }
        }
        cluster_sync();  // ... and read
      }
    } else if (ok && iters > 0) {
#pragma unroll
      for (int u = half; u < 2 * NH; u += 2) {
        const int which = u / NH, g = u % NH;  // 0 = dV, 1 = dK; 64-wide head_dim group
        uint8_t* dst = smem + C::kOffQdO + which * C::kTileK + g * kHalfK + row * 128;
        const uint32_t col = (which == 0 ? C::kColdV : C::kColdK) + g * 64;
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(t_lane + col, r0);
        tmem_ld_32x32b_x32(t_lane + col + 32, r1);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = (jj & 3) * 8 + 2 * e;
            w[e] = pack2_16<F16>(__uint_as_float(jj < 4 ? r0[i] : r1[i]), __uint_as_float(jj < 4 ? r0[i + 1] : r1[i + 1]));
          }
          *reinterpret_cast<uint4*>(dst + ((jj ^ sw) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async_smem();
      named_barrier_sync(2, kComputeThreads);
      if (leader) {
#pragma unroll
        for (int g = 0; g < NH; ++g) {
          tma_store_4d(&tmdV, s_base + C::kOffQdO + g * kHalfK, g * 64, kvh, kt * BKV, b);
          tma_store_4d(&tmdK, s_base + C::kOffQdO + C::kTileK + g * kHalfK, g * 64, kvh, kt * BKV, b);
        }
        tma_commit_group();
      }
    }
    if (leader) tma_wait_group<0>();
  }
  if (SPLIT && warp < kComputeWarp0) {  // (the compute warps met the others above)
    for (int i = 0; i < 4; ++i) cluster_sync();
  }

  if (fail_role != 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, 3) == 0) {
      p.status[1] = fail_role;
      p.status[2] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
      p.status[3] = HD;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// delta[b, h, t] = sum_d dO[b, t, h, d] * O[b, t, h, d]; HD / 8 lanes per row, 16 bytes per lane per tensor. The same pass
// clears the fp32 dQ accumulator (its rows are visited in the same order).
template <int HD, typename T16>
__global__ void flash_delta_t_kernel(const T16* __restrict__ o, const T16* __restrict__ d_o,
                                     float* __restrict__ delta, float* __restrict__ dq_acc, int B, int T, int H, long long o_sb, long long o_st,
                                     long long o_sh, long long do_sb, long long do_st, long long do_sh) {
  nnb_after_previous(o, d_o, delta, dq_acc);
  nnb_release_next();
  constexpr int L = HD / 8;
  const long long gid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long w = gid / L;
  const int sub = threadIdx.x % L;
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
#pragma unroll
  for (int o2 = L / 2; o2 > 0; o2 >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o2);
  if (w < rows && sub == 0) delta[((size_t)b * H + h) * T + t] = s;
}

// dq[b, t, h, :] (bf16, strided) = dq_acc[b, t, h, :] (fp32, contiguous)
template <int HD, typename T16>
__global__ void flash_dq_convert_t_kernel(const float* __restrict__ acc, T16* __restrict__ dq, long long rows, int H,
                                          int T, long long sb, long long st, long long sh) {
  nnb_after_previous(acc, dq);
  nnb_release_next();
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;  // one thread per 8 elements
  const long long total = rows * (HD / 8);
  if (idx >= total) return;
  const long long r = idx / (HD / 8);
  const int j = (int)(idx % (HD / 8)) * 8;
  const int h = (int)(r % H);
  const long long bt = r / H;
  const int t = (int)(bt % T);
  const long long b = bt / T;
  float v[8];
  Chunk8<float>::load(acc + r * HD + j, v);
  Chunk8<T16>::store(dq + b * sb + t * st + h * sh + j, v);
}

template <int HD, bool F16>
int launch_bwd_t(const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse, void* delta,
                 void* dq_acc, void* dq, void* dk, void* dv, int B, int T, int H, int KVH, const long long* qs, const long long* ks,
                 const long long* vs, const long long* os, const long long* dos, const long long* dqs, const long long* dks,
                 const long long* dvs, float scale, int in_order, void* status, cudaStream_t st) {
  using C = Cfg<HD>;
  using T16 = typename sm100::Operand16<F16>::type;
  const CUtensorMapDataType dt = F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv;
  if (!nnb_make_tmap_4d(&tq, dt, 2, q, HD, H, T, B, qs[2] * 2, qs[1] * 2, qs[0] * 2, 64, 1, BQ, "flash_bwd Q")) return -4;
  if (!nnb_make_tmap_4d(&tk, dt, 2, k, HD, KVH, T, B, ks[2] * 2, ks[1] * 2, ks[0] * 2, 64, 1, BKV, "flash_bwd K")) return -4;
  if (!nnb_make_tmap_4d(&tv, dt, 2, v, HD, KVH, T, B, vs[2] * 2, vs[1] * 2, vs[0] * 2, 64, 1, BKV, "flash_bwd V")) return -4;
  if (!nnb_make_tmap_4d(&tdo, dt, 2, d_o, HD, H, T, B, dos[2] * 2, dos[1] * 2, dos[0] * 2, 64, 1, BQ, "flash_bwd dO")) return -4;
  if (!nnb_make_tmap_4d(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dq_acc, HD, H, T, B, (uint64_t)HD * 4, (uint64_t)H * HD * 4,
                        (uint64_t)T * H * HD * 4, HD, 1, BQ, "flash_bwd dQ acc")) return -4;
  if (!nnb_make_tmap_4d(&tdk, dt, 2, dk, HD, KVH, T, B, dks[2] * 2, dks[1] * 2, dks[0] * 2, 64, 1, BKV, "flash_bwd dK")) return -4;
  if (!nnb_make_tmap_4d(&tdv, dt, 2, dv, HD, KVH, T, B, dvs[2] * 2, dvs[1] * 2, dvs[0] * 2, 64, 1, BKV, "flash_bwd dV")) return -4;

  const long long rows = (long long)B * T * H;
  nnb_launch_pre_pass(rows * HD, flash_delta_t_kernel<HD, T16>, (unsigned)((rows * (HD / 8) + 255) / 256), 256, st, (const T16*)o, (const T16*)d_o, (float*)delta, (float*)dq_acc, B, T, H, os[0], os[1], os[2], dos[0], dos[1], dos[2]);
  NNB_LAUNCH_OK("flash_delta");
  BParams p{};
  p.B = B; p.H = H; p.KVH = KVH; p.T = T;
  p.n_q_blocks = (T + BQ - 1) / BQ;
  p.group = H / KVH;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = static_cast<const float*>(lse);
  p.delta = static_cast<const float*>(delta);
  constexpr int fmt = F16 ? 0 : 1;
  p.idesc_s = sm100::make_idesc_f16(fmt, 0, 0, BKV, BQ);
  p.idesc_dkv = sm100::make_idesc_f16(fmt, 0, 1, BKV, HD);
  p.idesc_dq = sm100::make_idesc_f16(fmt, 1, 1, HD, BQ);
  p.status = static_cast<int*>(status);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_bwd_t_kernel<HD, F16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem) != cudaSuccess ||
        cudaFuncSetAttribute(flash_bwd_t_kernel<HD, F16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem) != cudaSuccess) {
      nnb_set_error("flash_bwd: cannot reserve %d bytes of shared memory", C::kSmem);
      return -3;
    }
    configured = true;
  }
  p.split = in_order ? 1 : nnb_visits_split(T, BQ, (long long)KVH * B, p.group, nnb_num_sms());
  p.out[0] = dv;
  p.out[1] = dk;
  for (int i = 0; i < 3; ++i) {
    p.out_s[0][i] = dvs[i];
    p.out_s[1][i] = dks[i];
  }
  dim3 grid(KVH * p.split, B, (T + BKV - 1) / BKV);
  nnb_launch_clusters(p.split > 1 ? flash_bwd_t_kernel<HD, F16, true> : flash_bwd_t_kernel<HD, F16, false>, p.split, grid, kThreads, C::kSmem, st, tq, tk, tv, tdo, tdq, tdk, tdv, p);
  NNB_LAUNCH_OK("flash_bwd_t");
  nnb_launch(flash_dq_convert_t_kernel<HD, T16>, (unsigned)((rows * (HD / 8) + 255) / 256), 256, 0, st, (const float*)dq_acc, (T16*)dq, rows, H, T,
                                                                                                dqs[0], dqs[1], dqs[2]);
  NNB_LAUNCH_OK("flash_dq_convert");
  return 0;
}

}  // namespace

#ifdef NNB_PROFILE
extern "C" int nnb_flash_bwd_t_prof_read(unsigned long long* out) { return (int)cudaMemcpyFromSymbol(out, g_flash_prof, sizeof(g_flash_prof)); }
#endif

// Same contract as nnb_flash_bwd (flash_bwd.cu), which forwards here. All tensors are [B, T, heads, hd] views given by
// element strides {batch, t, head}; dq_acc: fp32 [B, T, H, hd] contiguous scratch (cleared by the delta pre-pass).
int nnb_flash_bwd_t_impl(int hd, const void* q, const void* k, const void* v, const void* o, const void* d_o, const void* lse,
                         void* delta, void* dq_acc, void* dq, void* dk, void* dv, int B, int T, int H, int KVH, const long long* qs,
                         const long long* ks, const long long* vs, const long long* os, const long long* dos, const long long* dqs,
                         const long long* dks, const long long* dvs, float scale, int dtype, int in_order, void* status, cudaStream_t st) {
#define NNB_BWD_T(HD_, F16_) \
  launch_bwd_t<HD_, F16_>(q, k, v, o, d_o, lse, delta, dq_acc, dq, dk, dv, B, T, H, KVH, qs, ks, vs, os, dos, dqs, dks, dvs, scale, in_order, status, st)
  const bool f16 = dtype == NNB_F16;
  if (hd == 64) return f16 ? NNB_BWD_T(64, true) : NNB_BWD_T(64, false);
  return f16 ? NNB_BWD_T(128, true) : NNB_BWD_T(128, false);
#undef NNB_BWD_T
}

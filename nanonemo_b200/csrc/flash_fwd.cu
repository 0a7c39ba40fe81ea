// Causal grouped-query FlashAttention forward on tcgen05 / TMEM / TMA for sm_100a.
//
// An item is one 128-row query tile of one (batch, query head); a CTA walks the key/value tiles (64 keys each) of one item after
// the other up to the diagonal; two CTAs are resident per SM. 192 threads per CTA:
//   warp 0        TMA producer: an item's Q, then K_j / V_j into a ring of stages (4-D tensor maps over
//                 (head_dim, head, t, batch), so any (B,T,H,hd) / (B,H,T,hd) / packed-QKV strides work and
//                 query head h reads KV head h / group directly — nothing is repeated or copied); takes the next item;
//   warp 1        MMA issuer: S_j = Q K_j^T and O_j = P_j V_j with tcgen05.mma, accumulators in TMEM;
//   warps 2..5    softmax, one thread per query row (= TMEM lane): tcgen05.ld the scores, online max and
//                 sum with exp2, 16-bit P_j back into tensor memory over the scores it came from (the A operand of
//                 the second MMA: no shared-memory round trip). O accumulates IN TENSOR MEMORY over the key tiles; the row maximum used for the
//                 exponentials is only raised when a tile exceeds it by more than 2^8 (probabilities then
//                 stay below 256, exact in fp32 / safe in bf16), so the accumulator has to be rescaled —
//                 tcgen05.ld, multiply, tcgen05.st by the softmax threads — on a few tiles only.
// The score tile (and the P tile in it) is DOUBLE BUFFERED and the MMA warp runs two tiles ahead: S_{j+2} is
// issued as soon as the softmax threads have read S_j, and P_j V_j runs while they work on tile j+1, so
// neither side waits for a hand-off in steady state.
// Items follow one another without a seam: the grid has one block per item, heaviest first, and a block that is running takes over
// blocks that have not started (cluster launch control: the hardware's own order and balance, no counter in memory). The producer asks
// when it has requested its item's last keys, loads the next item's Q and first keys while the softmax works on the last ones, and the
// MMA warp starts the next item's first scores right behind the last product, while the softmax stores, at head_dim 64 into an O accumulator of its own. With a
// launch per item a CTA spent 4.7 us on set-up, first loads, first and last products and its store, as long as six key tiles. (First scores ahead of
// the last products, where a test found the next item there already: B32 T1024 99.2 us, now 94.4, B8 T4096 307 and 299, B64 T512 64.1 and 60.6, head_dim
// 128 B64 T256 41.3 and 40.5; and each lane of the MMA warp made that test for itself.)
// Forward alone, in a row, us, a CTA per item / items in sequence: 12/4 heads of 64, B200 T64 30.5 / 17.8, B64 T300 49.1 / 36.2, B64 T512 81.3 / 60.8,
// B32 T1024 112.7 / 94.2, B8 T4096 305 / 296; 16/4 heads of 128, B64 T256 56.0 / 40.9, B16 T1024 90 / 82.5, B8 T2048 142 / 137 to 143 (power).
// Outputs: O (16 bits) through a swizzled staging tile + TMA store, and L = m * scale + ln(l) per row (fp32)
// for the backward pass. Every mbarrier wait is bounded; on expiry the kernel records a status word
// and leaves cleanly.
//
// Replaces the reference's WMMA kernel for sm_75 (nanonemo/kernels/cuda/flash_attn.cu:52-174) and
// the mem-efficient SDPA path it benchmarks against; same math contract (causal, GQA-direct, saves
// the log-sum-exp per row).
#include <type_traits>

#include "sm100.cuh"

#ifdef NNB_PROFILE
extern "C" int nnb_flash_prof_read(unsigned long long* out) { return (int)cudaMemcpyFromSymbol(out, g_flash_prof, sizeof(g_flash_prof)); }
#endif

namespace {

using namespace sm100;

constexpr int BQ = 128;  // query rows per tile (= TMEM lanes)
constexpr int kThreads = 192;
constexpr int kSoftmaxThreads = 128;

// TAKE: a CTA goes on to blocks that have not started (nnb_flash_fwd has the rule).
template <int HD, bool TAKE>
struct FCfg {
  static constexpr int BN = 64;                             // keys per KV tile
  // K and V have rings of their own: K_j is free once S_j has been computed, V_j only after P_j V_j. Two CTAs per SM at both head
  // sizes (256 of the 512 tensor-memory columns each): while one's softmax runs on the special-function unit the other's
  // products run. At head_dim 128 that takes two stages instead of three (100 KB a CTA): 228 -> 142 us at B8 H16/4 T2048.
  static constexpr int kStages = HD == 64 ? 3 : 2;
  static constexpr int kQBytes = BQ * HD * 2;               // HD/64 swizzled K-blocks of 16 KB
  static constexpr int kKBytes = BN * HD * 2;
  static constexpr int kVBytes = BN * HD * 2;
  // Q tiles, and O accumulators in tensor memory: two where they fit twice beside the rest, so that the next item starts early
  static constexpr int kItems = TAKE && HD == 64 ? 2 : 1;
  static constexpr int kOBytes = TAKE ? BQ * 128 : 0;       // staging of 64 columns of O; a CTA with one item stages all of O where its Q was
  static constexpr int kBarBytes = 512;
  // 113 KB a CTA is what two per SM leave: nothing to spare for aligning the base at head_dim 128 with the staging tile. There the kernel checks it,
  // which costs a CTA 0.1 us.
  static constexpr int kSpare = TAKE && HD == 128 ? 0 : 1024;
  static constexpr int kSmem = kItems * kQBytes + kStages * (kKBytes + kVBytes) + kOBytes + kBarBytes + kSpare;
  static_assert(2 * (kSmem + 1024) <= 228 * 1024, "two CTAs per SM");
  static constexpr int kColS = 0;                           // S buffers at columns 0 and 64; P_j takes the first 32 of S_j's
  static constexpr int kColO = 128;                         // O accumulators from column 128
  static constexpr int kTmemCols = 256;
};

struct FParams {
  int B, H, KVH, T;
  int n_q_tiles;
  float scale_log2;   // softmax scale * log2(e)
  float scale;        // softmax scale
  float* lse;         // [B, H, T]
  uint32_t idesc_qk, idesc_pv;
  int* status;
};

template <int HD, bool F16, bool TAKE>
__global__ void __launch_bounds__(kThreads, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FParams p) {
  using C = FCfg<HD, TAKE>;
  constexpr int BN = C::BN;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sQ = C::kSpare == 0 ? smem_raw : reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sKV = sQ + C::kItems * C::kQBytes;                  // [stages][K | V]
  uint8_t* sO = TAKE ? sKV + C::kStages * (C::kKBytes + C::kVBytes) : sQ;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + C::kStages * (C::kKBytes + C::kVBytes) + C::kOBytes);
  // k_full[S], v_full[S], k_empty[S], v_empty[S], s_full[2], p_full[2], o_tile, o_all, q_full[2], q_empty[2], o_empty[2], next_full[2], next_empty[2]
  const uint32_t bar_k = smem_u32(bars), bar_v = bar_k + 8 * C::kStages;
  const uint32_t bar_ke = bar_v + 8 * C::kStages, bar_ve = bar_ke + 8 * C::kStages;
  const uint32_t bar_s = bar_ve + 8 * C::kStages, bar_p = bar_s + 16, bar_o = bar_p + 16, bar_of = bar_o + 8;
  const uint32_t bar_q = bar_of + 8, bar_qe = bar_q + 16, bar_oe = bar_qe + 16, bar_nf = bar_oe + 16, bar_ne = bar_nf + 16;
  constexpr int kBars = 4 * C::kStages + 16;
  static_assert(kBars % 2 == 0 && kBars * 8 + 32 + 12 <= C::kBarBytes, "the answers are 16-byte aligned behind the barriers");
  const uint32_t answers = bar_k + 8 * kBars;  // [2] of 16 bytes: which block is taken over
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* never_set = abort_flag + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (C::kSpare == 0 && (smem_u32(sQ) & 1023)) {  // (swizzled tiles)
    if (threadIdx.x == 0 && p.status != nullptr && atomicCAS(p.status, 0, 2) == 0) p.status[1] = 6;
    return;
  }
  // Longest-job-first over the WHOLE grid: the query tile is the slowest-varying block index, so every
  // (heaviest) latest query tile is begun before any of the next one and the kernel ends on the short ones.
  const int kv_total = (p.T + BN - 1) / BN;
  auto query_tile = [&](int z) { return p.n_q_tiles - 1 - z; };
  auto kv_tiles = [&](int qt) { return min(((qt + 1) * BQ + BN - 1) / BN, kv_total); };  // KV tiles holding keys <= the tile's last row
  const int group = p.H / p.KVH, first_kvh = blockIdx.x / group;  // (divisions: not on the way to the first load)
  // Item i + 1 is the answer in slot i & 1, read by the MMA warp, the four softmax warps and the producer.
  constexpr int kNextReaders = 32 + 4;  // lanes of the MMA warp, each for itself, and softmax warps (not the producer, who writes the slot again)
  auto next_item = [&](int i, int& x, int& y, int& z) { return taken_block(answers + 16 * (i & 1), x, y, z); };

  if (warp == 0) {  // a barrier a lane
    static_assert(kBars <= 32, "");
    const uint32_t bar = bar_k + 8 * lane;
    const bool softmax = (bar >= bar_p && bar < bar_o) || (bar >= bar_oe && bar < bar_nf);
    if (lane < kBars) mbar_init(bar, softmax ? kSoftmaxThreads : (bar >= bar_ne ? kNextReaders : 1));
    if (lane == 0) *abort_flag = *never_set = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmO);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  nnb_after_previous();  // (all its reads of global memory are TMA loads)
  int fail_role = 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int h = blockIdx.x, b = blockIdx.y, z = blockIdx.z, kvh = first_kvh;
      uint32_t s = 0, ph = 0;  // ring position and phase of the next K and V tile, counted along over all items
      bool ok = true;
      for (int i = 0;; ++i) {
        const int qt = query_tile(z), n_kv = kv_tiles(qt);
        const int qs = i % C::kItems;
        if (TAKE) ok = mbar_wait(bar_qe + 8 * qs, ((i / C::kItems) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar_q + 8 * qs, C::kQBytes);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) tma_load_4d(smem_u32(sQ) + qs * C::kQBytes + c * (BQ * 128), &tmQ, bar_q + 8 * qs, c * 64, h, qt * BQ, b);
        for (int j = 0; j < n_kv && ok; ++j) {
          const uint32_t sk = smem_u32(sKV) + s * (C::kKBytes + C::kVBytes), sv = sk + C::kKBytes;
          ok = mbar_wait(bar_ke + 8 * s, ph ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_k + 8 * s, C::kKBytes);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c) tma_load_4d(sk + c * (BN * 128), &tmK, bar_k + 8 * s, c * 64, kvh, j * BN, b);
          ok = mbar_wait(bar_ve + 8 * s, ph ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_v + 8 * s, C::kVBytes);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c) tma_load_4d(sv + c * (BN * 128), &tmV, bar_v + 8 * s, c * 64, kvh, j * BN, b);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
        if (!TAKE || !ok) break;
        // not earlier: a block that is asked for at the beginning of a long item would go to the busiest CTA
        ok = mbar_wait(bar_ne + 8 * (i & 1), ((i >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        take_block(answers + 16 * (i & 1), bar_nf + 8 * (i & 1));
        // (the answer has to arrive before the shared memory is given up, whatever the others do)
        ok = mbar_wait(bar_nf + 8 * (i & 1), (i >> 1) & 1, never_set);
        if (!ok) *abort_flag = 1;
        if (!ok || !next_item(i, h, b, z)) break;
        kvh = h / group;
      }
      if (!ok) fail_role = 1;
      nnb_release_next();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform: see umma_f16_elect)
    // Two cursors over the CTA's key tiles, numbered on over all items: S (scores) runs up to two tiles ahead of PV (second products). Every lane keeps
    // both, and nothing that a lane does next depends on when it asks: the order of the products is that of the tiles.
    const bool el = elect_one();
    bool ok = true, s_end = false;
    uint32_t sg = 0, s_stage = 0, s_ph = 0;             // S: tile, its stage and phase
    int s_item = 0, s_j = 0, s_n = kv_tiles(query_tile(blockIdx.z));
    uint32_t first_tile = 0, last_tile = 0, o_of = 0, o_ph = 0;  // per score buffer (bit): what PV has to know of its tile
    // S_j = Q K_j^T into score buffer sg & 1.
    auto issue_s = [&]() -> bool {
      if (s_j == s_n) {
        if (!TAKE) { s_end = true; return false; }
        const uint32_t bar = bar_nf + 8 * (s_item & 1), ph = (s_item >> 1) & 1;
        if (!mbar_wait(bar, ph, abort_flag)) { ok = false; return false; }
        int x, y, z;
        const bool more = next_item(s_item, x, y, z);
        fence_proxy_async_smem();
        mbar_arrive(bar_ne + 8 * (s_item & 1));  // (each lane for itself)
        if (!more) { s_end = true; return false; }
        ++s_item;
        s_j = 0;
        s_n = kv_tiles(query_tile(z));
      }
      const uint32_t qs = s_item % C::kItems;
      if (s_j == 0) {
        const uint32_t ph = (s_item / C::kItems) & 1;
        if (!mbar_wait(bar_q + 8 * qs, ph, abort_flag)) { ok = false; return false; }
      }
      if (!mbar_wait(bar_k + 8 * s_stage, s_ph, abort_flag)) { ok = false; return false; }
      tc_fence_after();
      const uint32_t sk = smem_u32(sKV) + s_stage * (C::kKBytes + C::kVBytes), sq = smem_u32(sQ) + qs * C::kQBytes;
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
        const uint32_t off_q = (k / 4) * (BQ * 128) + (k % 4) * 32, off_k = (k / 4) * (BN * 128) + (k % 4) * 32;
        umma_f16_elect(el, tmem_base + C::kColS + (sg & 1) * BN, make_smem_desc(sq + off_q, 16, 1024), make_smem_desc(sk + off_k, 16, 1024), p.idesc_qk,
                       k > 0 ? 1u : 0u);
      }
      umma_commit_elect(el, bar_s + 8 * (sg & 1));
      umma_commit_elect(el, bar_ke + 8 * s_stage);
      if (s_j == s_n - 1) umma_commit_elect(el, bar_qe + 8 * qs);  // Q has been read
      const uint32_t bit = 1u << (sg & 1);
      auto note = [&](uint32_t& word, bool on) { word = on ? word | bit : word & ~bit; };
      note(first_tile, s_j == 0);
      note(last_tile, s_j == s_n - 1);
      note(o_of, qs != 0);
      note(o_ph, (s_item / C::kItems) & 1);
      ++s_j;
      ++sg;
      if (++s_stage == C::kStages) { s_stage = 0; s_ph ^= 1; }
      return true;
    };
    uint32_t s = 0, ph = 0;
    for (uint32_t g = 0;; ++g) {  // PV: tile
      // (score buffer sg & 1 was released by the bar_p of tile sg - 2 below; the next item's first scores follow this item's last second product)
      while (ok && !s_end && sg < g + 2 && (s_j < s_n || sg == g)) {
        if (!issue_s()) break;
      }
      if (!ok || sg == g) break;
      const uint32_t pb = g & 1;
      if (!mbar_wait(bar_v + 8 * s, ph, abort_flag)) { ok = false; break; }
      const bool first = TAKE ? (first_tile >> pb) & 1 : g == 0, last = TAKE ? (last_tile >> pb) & 1 : (int)g == s_n - 1;
      const uint32_t ob = TAKE ? (o_of >> pb) & 1 : 0;
      if (TAKE && first && !mbar_wait(bar_oe + 8 * ob, ((o_ph >> pb) & 1) ^ 1, abort_flag)) { ok = false; break; }  // the item before has taken its O
      if (!mbar_wait(bar_p + 8 * pb, (g >> 1) & 1, abort_flag)) { ok = false; break; }   // P_j written, S_j consumed, O rescaled if needed
      tc_fence_after();
      const uint32_t sv = smem_u32(sKV) + s * (C::kKBytes + C::kVBytes) + C::kKBytes;
      const uint32_t tp = tmem_base + C::kColS + pb * BN;
#pragma unroll
      for (int k = 0; k < BN / 16; ++k)  // P from tensor memory: 16 keys = 8 columns per step; V is MN-major: 16 key rows (2048 B)
        umma_f16_ts_elect(el, tmem_base + C::kColO + ob * HD, tp + k * 8, make_smem_desc(sv + k * (16 * 128), BN * 128, 1024), p.idesc_pv,
                          (!first || k > 0) ? 1u : 0u);
      umma_commit_elect(el, bar_o);              // one completion per tile: O holds the item's sum up to it
      if (last) umma_commit_elect(el, bar_of);   // "all products of the item done" for the epilogue (no phase aliasing)
      umma_commit_elect(el, bar_ve + 8 * s);     // V_j is free
      if (++s == C::kStages) { s = 0; ph ^= 1; }
    }
    if (!ok && lane == 0) fail_role = 2;
  } else {
#include "flash_fwd_softmax.inc"
  }

  if (fail_role != 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, 2) == 0) {
      p.status[1] = fail_role;
      p.status[2] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
      p.status[3] = 0;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int HD, bool F16, bool TAKE>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const FParams& p, cudaStream_t st) {
  auto kern = flash_fwd_kernel<HD, F16, TAKE>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FCfg<HD, TAKE>::kSmem) != cudaSuccess) {
      nnb_set_error("flash_fwd: cannot reserve %d bytes of shared memory", FCfg<HD, TAKE>::kSmem);
      return -3;
    }
    configured = true;
  }
  nnb_launch(kern, dim3(p.H, p.B, p.n_q_tiles), kThreads, FCfg<HD, TAKE>::kSmem, st, tq, tk, tv, to, p);
  return 0;
}

}  // namespace

// q: [B, T, H, hd] addressed by element strides (q_sb, q_st, q_sh) with a contiguous last dim; k, v:
// [B, T, KVH, hd] likewise; o: [B, T, H, hd] likewise; lse: fp32 [B, H, T] contiguous.
extern "C" int nnb_flash_fwd(const void* q, const void* k, const void* v, void* o, void* lse, int B, int T, int H, int KVH,
                             int hd, long long q_sb, long long q_st, long long q_sh, long long k_sb, long long k_st,
                             long long k_sh, long long v_sb, long long v_st, long long v_sh, long long o_sb, long long o_st,
                             long long o_sh, float scale, int dtype, void* status, cudaStream_t st) {
  NNB_REQUIRE(hd == 64 || hd == 128, "flash_fwd: head_dim %d not supported (64 or 128)", hd);
  NNB_REQUIRE(dtype == NNB_BF16 || dtype == NNB_F16, "flash_fwd: bf16 or fp16 only (dtype code %d)", dtype);
  const bool f16 = dtype == NNB_F16;
  NNB_REQUIRE(H % KVH == 0 && B > 0 && T > 0, "flash_fwd: bad shape B=%d T=%d H=%d KVH=%d", B, T, H, KVH);
  const CUtensorMapDataType dt = f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int BN = 64;
  CUtensorMap tq, tk, tv, to;
  if (!nnb_make_tmap_4d(&tq, dt, 2, q, hd, H, T, B, q_sh * 2, q_st * 2, q_sb * 2, 64, 1, BQ, "flash Q")) return -4;
  if (!nnb_make_tmap_4d(&tk, dt, 2, k, hd, KVH, T, B, k_sh * 2, k_st * 2, k_sb * 2, 64, 1, BN, "flash K")) return -4;
  if (!nnb_make_tmap_4d(&tv, dt, 2, v, hd, KVH, T, B, v_sh * 2, v_st * 2, v_sb * 2, 64, 1, BN, "flash V")) return -4;
  if (!nnb_make_tmap_4d(&to, dt, 2, o, hd, H, T, B, o_sh * 2, o_st * 2, o_sb * 2, 64, 1, BQ, "flash O")) return -4;
  FParams p{};
  p.B = B; p.H = H; p.KVH = KVH; p.T = T;
  p.n_q_tiles = (T + BQ - 1) / BQ;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = static_cast<float*>(lse);
  p.idesc_qk = sm100::make_idesc_f16(f16 ? 0 : 1, 0, 0, BQ, BN);
  p.idesc_pv = sm100::make_idesc_f16(f16 ? 0 : 1, 0, 1, BQ, hd);
  p.status = static_cast<int*>(status);
  // A grid that runs at once has nothing to take over, and an instance without what that takes. us, in a row, that instance / the other one, with
  // a switch at run time: 12/4 heads of 64, B2 T333 6.7 / 7.3, B1 T201 5.4 / 5.85, B1 T1024 13.2 / 14.5, 16/4 heads of 128, B1 T200 6.2 / 6.6, B1 T1000
  // 14.5 / 15.8. Asking costs 0.8 more.
  const bool take = (long long)H * B * p.n_q_tiles > 2 * nnb_num_sms();
#define NNB_FWD(HD, F16) (take ? launch_fwd<HD, F16, true>(tq, tk, tv, to, p, st) : launch_fwd<HD, F16, false>(tq, tk, tv, to, p, st))
  const int rc = hd == 64 ? (f16 ? NNB_FWD(64, true) : NNB_FWD(64, false)) : (f16 ? NNB_FWD(128, true) : NNB_FWD(128, false));
#undef NNB_FWD
  if (rc != 0) return rc;
  NNB_LAUNCH_OK("flash_fwd");
  return 0;
}

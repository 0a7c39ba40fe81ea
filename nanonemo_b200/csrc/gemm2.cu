// bf16/fp16 GEMM with CTA PAIRS on the 5th-generation tensor cores: D[M,N] (+)= A[M,K] * B[N,K]^T, fp32 accumulate.
//
// Two CTAs of a cluster (two SMs) own one 256 x 256 output tile. Each CTA loads its own 128 rows of A and its own
// 128 of the 256 rows of B; ONE thread of the even ("leader") CTA issues tcgen05.mma.cta_group::2 (M = 256), which
// reads A and B from the shared memory of both CTAs and accumulates each CTA's 128 rows into that CTA's own tensor
// memory. Per 128 x 256 of output a CTA therefore stages 32 KB per k-block instead of the 48 KB of the single-CTA
// kernel (gemm.cu): the L2 -> shared-memory fill, which bounds these GEMMs at K = 768..2048, drops by a third.
// No multicast is used: every CTA fetches its own tiles; the pair is coupled only through
//   * TMA loads of both CTAs completing on the leader's "full" barrier (cta_group::2 form of the load),
//   * tcgen05.commit.cta_group::2 arriving on the "empty" / "accumulator full" barriers of BOTH CTAs (one commit per CTA),
//   * the peer's epilogue warps arriving remotely on the leader's "accumulator empty" barrier.
// Roles per CTA as in gemm.cu: warp 0 TMA producer, warp 1 MMA issuer (leader only; both allocate TMEM), warps 2.. (4 or 8)
// epilogue (tcgen05.ld -> swizzled staging -> TMA store / reduce-add). All waits are bounded.
// Replaces the cuBLAS calls behind nn.Linear in the reference (nanonemo/model/layers.py:80-83, 128-130).
//
// Fused epilogues (template parameter EPI), each replacing a separate pass over HBM of the reference's elementwise kernels:
//   EPI_SWIGLU    gate||up projection: the leader stages 128 GATE rows of the weight, its peer the matching 128 UP rows, so
//                 one accumulator holds gate (columns 0..127) and up (128..255) of the same 128 features; the epilogue
//                 writes both halves of the projection (kept for backward) AND act = silu(gate) * up
//                 (nanonemo/kernels/triton/swiglu.py:19-38).
//   EPI_ROPE      QKV projection: rotate-half RoPE applied to the query / key heads while the tile leaves tensor memory
//                 (one cos / sin row per token; a 64-column chunk is one head, two chunks at head_dim 128)
//                 (nanonemo/kernels/triton/rope.py:18-47).
//   EPI_CE_STATS  LM head: besides the 16-bit logits, every (row, 256-column tile) gets its (max, sum of exp(x - max)), so
//                 the cross-entropy kernel needs one sweep over the logits instead of two
//                 (nanonemo/kernels/triton/linear_ce.py:21-41).
//   EPI_SWIGLU_ACT  the same for a forward pass without gradients: nobody reads the projection, so only act leaves the tile, a
//                 third of the bytes. One staging tile per 64 features instead of three: two epilogue groups and a sixth
//                 operand stage fit. 32768 x 4096 x 768: 133 us, EPI_SWIGLU 168.
//   EPI_CE_LOSS   LM head of a loss without gradients (validation): the statistics and the target's logit of every row, and no
//                 logits at all. Against EPI_CE_STATS + the one-sweep kernel this drops the 16-bit logits' write, read and
//                 rewrite; the accumulator goes straight from tensor memory to the statistics, so the staging tiles' shared
//                 memory holds a seventh operand stage instead.
//   EPI_CHAINED   no fusion, fp32 output of a long K loop that is not cut into splits: the accumulator is handed over every p.chain
//                 k-blocks and added to sums in registers (128 columns a thread, two epilogue groups) while the tensor core fills
//                 the other one. The tensor core's own additions lose more than an fp32 addition does, and what they lose grows
//                 with the length of the chain: normal bf16 operands, K = 8192, one chain is 9.1e-6 off 64 bits (2-norm), chains
//                 of 16 k-blocks 1.0e-6, of 8 4.8e-7 (torch.matmul in fp32: 9.5e-7). Reduce-adding that many splits to memory
//                 instead costs the output's bytes each time: see nnb_plan_k.
// All of them compute on the values ROUNDED to the 16-bit output type, so they match the unfused kernels bit for bit.
#include "gemm2.cuh"

#include "common.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128;   // rows per CTA (256 per pair)
constexpr int BN = 256;   // columns per pair tile; each CTA stages BN / 2 rows of B
constexpr int BK = 64;
constexpr int kEpilogueThreads = 128;  // one epilogue GROUP: four warps, one per tensor-memory lane quadrant
constexpr int kStageBytesA = BM * BK * 2, kStageBytesB = (BN / 2) * BK * 2, kStageBytes = kStageBytesA + kStageBytesB;
constexpr int kTmemCols = 512;
// The SwiGLU epilogue fills three staging tiles per 64-feature round (gate, up, act); its backward has a ring of two (gate, up)
// tile pairs (three and a stage less: 139 us instead of 141 at K = 768, 182 instead of 176 at K = 2048, M 8192, F 5632), the chained
// fp32 output two tiles per group: they pay for the staging with one stage of the operand ring
// (chained, 2048 x 5632 x 4096: 93 us, with two tiles and six stages 112; 11264 x 2048 x 2048 87 / 89, 3072 x 2048 x 8192 84 / 81).
template <int EPI> struct Cfg {
  static constexpr int kStages = (EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_BWD || EPI == EPI_CHAINED) ? 5 : (EPI == EPI_CE_LOSS ? 7 : 6);
  static constexpr int kStagingTiles = EPI == EPI_SWIGLU ? 3 : ((EPI == EPI_SWIGLU_BWD || EPI == EPI_CHAINED) ? 4 : (EPI == EPI_CE_LOSS ? 0 : 2));
  static constexpr int kStagingBytes = kStagingTiles * BM * 128;
  // Epilogue warps. A group shares staging tiles, a named barrier and a thread that issues its TMA traffic.
  //   one group of four warps  the plain epilogue: a thread per accumulator row.
  //   two groups of four       each has staging tiles of its own and takes alternate 64-column chunks: softmax statistics (an exponential
  //                            per logit), activation only, and EPI_CHAINED, where a thread holds the sums of 128 columns.
  //   one group of eight       two threads a row, half the columns of a round each, in the SAME staging tiles: the arithmetic of a
  //                            round is spread over twice the warps without a second set of tiles, which would cost an operand
  //                            stage, and is done before the tiles are waited for, so it overlaps the stores of the round before.
  //                            SwiGLU forward 176 -> 168 us (32768 x 4096 x 768), RoPE 65 -> 61 (32768 x 1280 x 768) and at
  //                            head_dim 128 91 -> 80 (8192 x 3072 x 2048), SwiGLU backward 162 -> 141 (32768 x 2048 x 768).
  static constexpr int kEpiGroups = (EPI == EPI_NONE || EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_BWD || EPI == EPI_ROPE) ? 1 : 2;
  static constexpr int kGroupThreads = EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_BWD || EPI == EPI_ROPE ? 2 * kEpilogueThreads : kEpilogueThreads;
  static constexpr int kEpiThreads = kEpiGroups * kGroupThreads;
  static constexpr int kThreads = 64 + kEpiThreads + (EPI == EPI_SWIGLU_BWD ? 32 : 0);  // (SwiGLU backward: a warp for the epilogue's loads and stores)
  static constexpr int kPairs = kStagingTiles / 2;  // SwiGLU backward: ring of (gate, up) tile pairs
  static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + 1024 + 256;
};

struct Params2 {
  int M, N, K;
  int m_pairs, n_blocks, k_splits, kblocks_total, kblocks_per_split;
  int chain;    // EPI_CHAINED: k-blocks per accumulator
  int group_m;  // tile order: groups of group_m 256-row blocks are swept n-block by n-block
  int a_mn, b_mn, out_f32, reduce_add, out_bf16;
  uint32_t idesc;
  int* status;
  // fused epilogues
  int epi_cols;        // EPI_SWIGLU: F (the up rows of the weight start at row F); EPI_ROPE: columns that are rotated
  int t_len, half_dim; // EPI_ROPE: sequence length (row m uses table row m % t_len), head_dim / 2
  const float* cos_t;  // EPI_ROPE: [t_len, half_dim] fp32
  const float* sin_t;
  float* stats;        // EPI_CE_STATS: [M, 2 n_blocks, 2] fp32 (max, sum of exp(x - max)): two entries per 256-column tile (64-column
                       // chunks 0, 2 and 1, 3 of the tile: one entry per epilogue warp group; (-inf, 0) when the group had no chunk)
  const long long* targets;  // EPI_CE_LOSS: [M]
  float* target_logit;       // EPI_CE_LOSS: [M]
};

__device__ __forceinline__ uint32_t pack16(float lo, float hi, bool bf) {
  if (bf) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack16(uint32_t w, bool bf) {
  if (bf) return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
  return __half22float2(*reinterpret_cast<__half2*>(&w));
}
__device__ __forceinline__ float round16(float x, bool bf) {
  return bf ? __bfloat162float(__float2bfloat16_rn(x)) : __half2float(__float2half_rn(x));
}
// 32 consecutive columns (16 packed words) of this thread's row into 16-byte units [u0, u0 + 4) of a swizzled staging row.
__device__ __forceinline__ void stage32(uint8_t* my_row, int sw, int u0, const uint32_t (&w)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    *reinterpret_cast<uint4*>(my_row + (((u0 + j) ^ sw) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
}
// Rotate-half on 16 (lo, hi) column pairs of one token: lo' = lo c - hi s, hi' = lo s + hi c, computed on the rounded values.
__device__ __forceinline__ void rope16(uint32_t (&lo)[16], uint32_t (&hi)[16], const float (&cc)[16], const float (&ss)[16], bool bf) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float a = round16(__uint_as_float(lo[i]), bf), b = round16(__uint_as_float(hi[i]), bf);
    lo[i] = __float_as_uint(a * cc[i] - b * ss[i]);
    hi[i] = __float_as_uint(a * ss[i] + b * cc[i]);
  }
}
// 16 consecutive fp32 table entries of one token (16-byte aligned: the tables have 32 or 64 entries per row).
__device__ __forceinline__ void load_table16(const float* __restrict__ src, float (&dst)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(src + i));
    dst[i] = v.x; dst[i + 1] = v.y; dst[i + 2] = v.z; dst[i + 3] = v.w;
  }
}
// 16 consecutive columns of this thread's row into 16-byte units [u0, u0 + 2) of a swizzled staging row.
__device__ __forceinline__ void stage16(uint8_t* my_row, int sw, int u0, const uint32_t (&r)[16], bool bf) {
  uint32_t w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = pack16(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]), bf);
  *reinterpret_cast<uint4*>(my_row + ((u0 ^ sw) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(my_row + (((u0 + 1) ^ sw) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
}
__device__ __forceinline__ void pack32(const uint32_t (&r)[32], uint32_t (&w)[16], bool bf) {
#pragma unroll
  for (int e = 0; e < 16; ++e) w[e] = pack16(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]), bf);
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// TMA tile load issued by either CTA of the pair; the bytes are counted on the LEADER's mbarrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, uint32_t leader_bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(bool elected, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"((uint32_t)elected) : "memory");
}
// Arrive on ONE mbarrier (a shared::cluster address, own or the peer's) once the pair MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(bool elected, uint32_t cluster_bar) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %1, 0;\n@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}"
               ::"r"(cluster_bar), "r"((uint32_t)elected) : "memory");
}

// BF16: the 16-bit format of operands and output (false = fp16). A template parameter rather than a launch argument so that the
// epilogues' conversions are straight-line code: with a run-time flag every pack / unpack is a branch, the unrolled per-element
// arithmetic is cut into hundreds of basic blocks and the epilogue warps (two per scheduler at most) lose the overlap between
// independent elements that hides the special-function and conversion latencies.
template <int EPI, bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Cfg<EPI>::kThreads, 1)
gemm2_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmE, const Params2 p) {
  constexpr int kStages = Cfg<EPI>::kStages, kStagingBytes = Cfg<EPI>::kStagingBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  uint8_t* staging = smem + kStages * kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + kStagingBytes);
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kStages;
  const uint32_t bar_tfull = bar_empty + 8 * kStages, bar_tempty = bar_tfull + 16;
  const uint32_t bar_in = bar_tempty + 16, bar_out = bar_in + 24;  // EPI_SWIGLU_BWD: a (gate, up) pair has landed / has been worked off
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_abort_base = abort_flag + 1;  // one word per epilogue group

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);    // leader: its producer's expect-tx arrival (bytes of both CTAs)
      mbar_init(bar_empty + 8 * s, 1);   // one commit per CTA
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);
      mbar_init(bar_tempty + 8 * a, 2 * Cfg<EPI>::kEpiThreads / 32);  // leader: epilogue warps of both CTAs
    }
    for (int a = 0; a < 3; ++a) {
      mbar_init(bar_in + 8 * a, 1);
      mbar_init(bar_out + 8 * a, Cfg<EPI>::kEpiThreads / 32);
    }
    *abort_flag = 0;
    epi_abort_base[0] = 0;
    epi_abort_base[1] = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish2();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmD);
    if (EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_BWD) tma_prefetch_desc(&tmE);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anybody signals the peer
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const float *cos_t = p.cos_t, *sin_t = p.sin_t;
  const long long* targets = p.targets;
  nnb_after_previous(cos_t, sin_t, targets);

  const int items = p.m_pairs * p.n_blocks * p.k_splits;
  const int pair0 = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
  int fail_role = 0, fail_item = -1;
  // consecutive tiles (the ones the persistent pairs work on at the same time) cover group_m x (pairs / group_m) blocks
  auto tile_coords = [&](int tile, int& m_pair, int& n_blk) {
    const int per_group = p.group_m * p.n_blocks, g = tile / per_group, r = tile - g * per_group;
    const int gm = min(p.group_m, p.m_pairs - g * p.group_m);
    m_pair = g * p.group_m + r % gm;
    n_blk = r / gm;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      const uint32_t leader_full0 = map_to_cta(bar_full, 0);  // the same barrier slot in the even CTA of the pair
      for (int item = pair0; item < items && ok; item += npairs) {
        const int ks = item % p.k_splits, tile = item / p.k_splits;
        int m_pair, n_blk;
        tile_coords(tile, m_pair, n_blk);
        const int m_row0 = (m_pair * 2 + (int)rank) * BM;
        // SwiGLU: the leader stages gate rows, the peer the up rows (F further down) of the same 128 features
        const int n_row0 = EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_ACT ? n_blk * (BN / 2) + (int)rank * p.epi_cols : n_blk * BN + (int)rank * (BN / 2);
        const int kb0 = ks * p.kblocks_per_split, kb1 = min(kb0 + p.kblocks_per_split, p.kblocks_total);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % kStages, ph = (it / kStages) & 1;
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag)) { ok = false; fail_role = 1; fail_item = item; break; }
          const uint32_t full = bar_full + 8 * s, leader_full = leader_full0 + 8 * s;
          if (rank == 0) mbar_expect_tx(full, 2 * kStageBytes);
          const uint32_t sa = smem_u32(stage_base + s * kStageBytes), sb = sa + kStageBytesA;
          if (!p.a_mn) {
            tma_load_2d_pair(sa, &tmA, leader_full, kb * BK, m_row0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * (BK * 128), &tmA, leader_full, m_row0 + j * 64, kb * BK);
          }
          if (!p.b_mn) {
            tma_load_2d_pair(sb, &tmB, leader_full, kb * BK, n_row0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(sb + j * (BK * 128), &tmB, leader_full, n_row0 + j * 64, kb * BK);
          }
        }
      }
      nnb_release_next();  // the last operands are on their way
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only; warp-uniform, see umma_f16_elect)
    if (rank == 0) {
      const bool el = elect_one();
      uint32_t s = 0, ph = 0, tile_iter = 0;  // ring position and phase, counted along
      bool ok = true;
      const uint32_t a_step = p.a_mn ? (16 * 128) >> 4 : 32 >> 4, b_step = p.b_mn ? (16 * 128) >> 4 : 32 >> 4;
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, b_lbo = p.b_mn ? BK * 128 : 16;
      const uint32_t peer_empty = map_to_cta(bar_empty, 1), peer_tfull = map_to_cta(bar_tfull, 1);
      const int chain = EPI == EPI_CHAINED ? p.chain : p.kblocks_per_split;  // k-blocks per accumulator
      for (int item = pair0; item < items && ok; item += npairs) {
        const int ks = item % p.k_splits;
        const int kb0 = ks * p.kblocks_per_split, kb1 = min(kb0 + p.kblocks_per_split, p.kblocks_total);
        for (int c0 = kb0; c0 < kb1 && ok; c0 += chain, ++tile_iter) {
          const int c1 = min(c0 + chain, kb1);
          const uint32_t acc = tile_iter & 1, acc_ph = (tile_iter >> 1) & 1;
          if (!mbar_wait(bar_tempty + 8 * acc, acc_ph ^ 1, abort_flag)) { ok = false; fail_role = 2; fail_item = lane == 0 ? item : -1; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          for (int kb = c0; kb < c1; ++kb) {
            if (!mbar_wait(bar_full + 8 * s, ph, abort_flag)) { ok = false; fail_role = 2; fail_item = lane == 0 ? item : -1; break; }
            tc_fence_after();
            const uint32_t sa = smem_u32(stage_base + s * kStageBytes), sb = sa + kStageBytesA;
            const uint64_t da = make_smem_desc(sa, a_lbo, 1024), db = make_smem_desc(sb, b_lbo, 1024);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_f16_pair(el, d_tmem, da + (uint64_t)(k * a_step), db + (uint64_t)(k * b_step), p.idesc, (kb > c0 || k > 0) ? 1u : 0u);
            umma_commit_pair(el, bar_empty + 8 * s);    // this CTA's stage is free once the MMAs have read it
            umma_commit_pair(el, peer_empty + 8 * s);   // ... and so is the peer's
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
          if (ok) {
            umma_commit_pair(el, bar_tfull + 8 * acc);
            umma_commit_pair(el, peer_tfull + 8 * acc);
          }
        }
      }
    }
  } else if (EPI == EPI_SWIGLU_BWD && warp == 2 + Cfg<EPI>::kEpiThreads / 32) {
    // ------------------------------------------------------------------ I/O warp of the SwiGLU backward (both CTAs)
    // Fetches the (gate, up) tiles of every 64-column chunk into a ring of pairs and stores what the epilogue warps leave in them, so
    // that neither a load's latency nor a store's drain stops a warp that computes (when the warps did both themselves, a third of an
    // epilogue's 16,000 cycles a tile were such waits). The chunks of the NEXT tile are pulled into L2 a whole tile ahead of their use.
    // (The values straight into registers, 32 bytes of its own row a thread: 195 us, 32 cache lines an access are too many.)
    if (lane == 0) {
      constexpr uint32_t kPairs = Cfg<EPI>::kPairs;
      struct Cursor { int item, c, chunks, col, row; };
      auto enter = [&](Cursor& u, int item) {  // the first chunk at or after `item`
        for (u.c = u.chunks = 0; item < items; item += npairs) {
          int m_pair, n_blk;
          tile_coords(item / p.k_splits, m_pair, n_blk);
          u.row = (m_pair * 2 + (int)rank) * BM;
          u.col = n_blk * BN;
          u.chunks = u.row < p.M ? min(BN / 64, (p.N - u.col) / 64) : 0;
          if (u.chunks > 0) break;
        }
        u.item = item;
      };
      auto step = [&](Cursor& u) { if (++u.c == u.chunks) enter(u, u.item + npairs); };
      Cursor load{}, store{}, ahead{};
      auto fetch = [&](uint32_t pair) {
        const uint32_t bar = bar_in + 8 * pair, dst = smem_u32(staging + pair * 2 * BM * 128);
        mbar_expect_tx(bar, 2 * BM * 128);
        tma_load_2d(dst, &tmE, bar, load.col + load.c * 64, load.row);
        tma_load_2d(dst + BM * 128, &tmE, bar, p.N + load.col + load.c * 64, load.row);
        if (load.c == 0) {
          enter(ahead, load.item + npairs);
          for (; ahead.c < ahead.chunks; ++ahead.c) {
            tma_prefetch_l2_2d(&tmE, ahead.col + ahead.c * 64, ahead.row);
            tma_prefetch_l2_2d(&tmE, p.N + ahead.col + ahead.c * 64, ahead.row);
          }
        }
        step(load);
      };
      enter(load, pair0);
      store = load;
      uint32_t loaded = 0, stored = 0;
      for (; loaded < kPairs && load.item < items; ++loaded) fetch(loaded);
      for (; store.item < items; ++stored) {
        const uint32_t pair = stored % kPairs;
        if (!mbar_wait(bar_out + 8 * pair, (stored / kPairs) & 1, abort_flag)) { fail_role = 3; fail_item = store.item; break; }
        const uint32_t src = smem_u32(staging + pair * 2 * BM * 128);
        tma_store_2d(&tmD, src, store.col + store.c * 64, store.row);
        tma_store_2d(&tmD, src + BM * 128, p.N + store.col + store.c * 64, store.row);
        tma_commit_group();
        step(store);
        if (load.item < items) {
          tma_wait_group_read<0>();  // the pair is free again
          fetch(pair);
          ++loaded;
        }
      }
      // whatever was requested has to have landed before the shared memory is given up (after a wait that ran out, too)
      volatile int unset = 0;
      for (uint32_t k = stored; k < loaded; ++k) mbar_wait(bar_in + 8 * (k % kPairs), (k / kPairs) & 1, const_cast<int*>(&unset));
      tma_wait_group<0>();
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2.., both CTAs)
    const int q = warp & 3;
    const int row = q * 32 + lane;
    constexpr int kGroup = Cfg<EPI>::kGroupThreads;
    const int grp = Cfg<EPI>::kEpiGroups == 1 ? 0 : (threadIdx.x - 64) / kGroup;  // epilogue group
    const int et = (threadIdx.x - 64) % kGroup;                     // thread within the group; et == 0 issues its TMA traffic
    const int half = et / kEpilogueThreads;                         // groups of eight warps: which of the row's two threads this is
    const int epi_bar = 1 + grp;                                    // the group's named barrier
    volatile int* epi_abort = epi_abort_base + grp;
    uint32_t tile_iter = 0, gchunk = 0;
    int pending_stores = 0;
    const uint32_t leader_tempty = map_to_cta(bar_tempty, 0);
    for (int item = pair0; item < items; item += npairs, ++tile_iter) {
      const int tile = item / p.k_splits;
      int m_pair, n_blk;
      tile_coords(tile, m_pair, n_blk);
      const int d_row = (m_pair * 2 + (int)rank) * BM;
      if constexpr (EPI == EPI_CHAINED) {
        // group g holds the sums of 32-column chunks g, g + 2, g + 4, g + 6 of this thread's row, chain after chain, then stores them
        const bool live = d_row < p.M;
        const int kb0 = item % p.k_splits * p.kblocks_per_split, kbs = min(p.kblocks_per_split, p.kblocks_total - kb0);
        const int chains = (kbs + p.chain - 1) / p.chain;
        float sum[4][32];
#pragma unroll
        for (int e = 0; e < 128; ++e) sum[e >> 5][e & 31] = 0.f;
        bool left = false;
        for (int i = 0; i < chains; ++i, ++tile_iter) {
          const uint32_t acc = tile_iter & 1, acc_ph = (tile_iter >> 1) & 1;
          const bool ok = mbar_wait(bar_tfull + 8 * acc, acc_ph, abort_flag);
          if (!ok) { fail_role = 3; fail_item = item; }
          if (named_barrier_or(epi_bar, kGroup, !ok)) { left = true; break; }  // the group leaves together
          tc_fence_after();
          if (live) {
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN + grp * 32;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t r[16];
              tmem_ld_32x32b_x16(t_row + (j >> 1) * 64 + (j & 1) * 16, r);
              tmem_ld_wait(r);
#pragma unroll
              for (int e = 0; e < 16; ++e) sum[j >> 1][(j & 1) * 16 + e] += __uint_as_float(r[e]);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (rank == 0) mbar_arrive(bar_tempty + 8 * acc);
            else mbar_arrive_cluster(leader_tempty + 8 * acc);
          }
        }
        if (left) break;
        --tile_iter;  // (the loop's own step)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = n_blk * BN + grp * 32 + j * 64;
          if (live && col < p.N) {
            uint8_t* buf = staging + (grp * 2 + (int)(gchunk & 1)) * (BM * 128);  // (counted by stores: a tile may have fewer than four)
            ++gchunk;
            if (et == 0 && pending_stores >= 2) tma_wait_group_read<1>();  // the store that last read `buf` is done
            named_barrier_sync(epi_bar, kGroup);
#pragma unroll
            for (int u = 0; u < 8; ++u)
              *reinterpret_cast<float4*>(buf + row * 128 + ((u ^ (row & 7)) << 4)) =
                  make_float4(sum[j][4 * u], sum[j][4 * u + 1], sum[j][4 * u + 2], sum[j][4 * u + 3]);
            fence_proxy_async_smem();
            named_barrier_sync(epi_bar, kGroup);
            if (et == 0) {
              if (p.reduce_add) tma_reduce_add_2d(&tmD, smem_u32(buf), col, d_row);
              else tma_store_2d(&tmD, smem_u32(buf), col, d_row);
              tma_commit_group();
            }
            if (pending_stores < 2) ++pending_stores;
          }
        }
        continue;
      }
      const uint32_t acc = tile_iter & 1, acc_ph = (tile_iter >> 1) & 1;
      if constexpr (EPI == EPI_SWIGLU_BWD) {
        // accumulator = d(act). The saved gate and up values arrive in pairs of 64-column tiles (see the I/O warp); a row's two
        // threads turn 32 columns each into d(gate) | d(up) in place:
        //   s = sigmoid(g), d(gate) = d(act) u s (1 + g (1 - s)), d(up) = d(act) g s
        // Every warp goes its own way: it hands over to the I/O warp and to the MMA warp through mbarriers only.
        const int chunks = d_row < p.M ? min(BN / 64, (p.N - n_blk * BN) / 64) : 0, sw = row & 7;
        if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * acc, acc_ph, abort_flag))) { fail_role = 3; fail_item = item; break; }
        tc_fence_after();
        bool ok = true;
        for (int c = 0; c < chunks; ++c, ++gchunk) {
          const uint32_t pair = gchunk % Cfg<EPI>::kPairs, ph = (gchunk / Cfg<EPI>::kPairs) & 1;
          uint32_t d[32];
          tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN + c * 64 + half * 32, d);
          tmem_ld_wait();
          ok = __all_sync(0xffffffffu, mbar_wait(bar_in + 8 * pair, ph, abort_flag));
          if (!ok) { fail_role = 3; fail_item = item; break; }
          uint8_t* row_g = staging + (pair * 2 * BM + row) * 128;
          uint8_t* row_u = row_g + BM * 128;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4* pg = reinterpret_cast<uint4*>(row_g + (((half * 4 + j) ^ sw) << 4));
            uint4* pu = reinterpret_cast<uint4*>(row_u + (((half * 4 + j) ^ sw) << 4));
            const uint4 gw = *pg, uw = *pu;
            const uint32_t gin[4] = {gw.x, gw.y, gw.z, gw.w}, uin[4] = {uw.x, uw.y, uw.z, uw.w};
            uint32_t og[4], ou[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float d0 = __uint_as_float(d[j * 8 + 2 * e]), d1 = __uint_as_float(d[j * 8 + 2 * e + 1]);
              const float2 g2 = unpack16(gin[e], BF16), u2 = unpack16(uin[e], BF16);
              const float s0 = 1.f / (1.f + __expf(-g2.x)), s1 = 1.f / (1.f + __expf(-g2.y));
              og[e] = pack16(d0 * u2.x * s0 * (1.f + g2.x * (1.f - s0)), d1 * u2.y * s1 * (1.f + g2.y * (1.f - s1)), BF16);
              ou[e] = pack16(d0 * g2.x * s0, d1 * g2.y * s1, BF16);
            }
            *pg = make_uint4(og[0], og[1], og[2], og[3]);
            *pu = make_uint4(ou[0], ou[1], ou[2], ou[3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_out + 8 * pair);
        }
        if (!ok) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(bar_tempty + 8 * acc);
          else mbar_arrive_cluster(leader_tempty + 8 * acc);
        }
        continue;
      }
      long long tgt_col = -1;  // EPI_CE_LOSS: this row's target relative to the tile's first column
      if constexpr (EPI == EPI_CE_LOSS) {
        if (d_row + row < p.M) tgt_col = targets[d_row + row] - (long long)n_blk * BN;
      }
      // EPI_ROPE: the table entries of this thread's token, fetched while the tile is still being multiplied: 16 at head_dim 64, 32 at 128
      float rope_c[2][16], rope_s[2][16];
      if constexpr (EPI == EPI_ROPE) {
        if (n_blk * BN < p.epi_cols) {
          const size_t at = (size_t)((d_row + row) % p.t_len) * p.half_dim;
          load_table16(cos_t + at + half * 16, rope_c[0]);
          load_table16(sin_t + at + half * 16, rope_s[0]);
          if (p.half_dim == 64) {
            load_table16(cos_t + at + 32 + half * 16, rope_c[1]);
            load_table16(sin_t + at + 32 + half * 16, rope_s[1]);
          }
        }
      }
      const bool ok = mbar_wait(bar_tfull + 8 * acc, acc_ph, abort_flag);
      if (!ok) { fail_role = 3; fail_item = item; }
      if (et == 0) *epi_abort = *abort_flag;
      named_barrier_sync(epi_bar, kGroup);
      if (*epi_abort) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      const bool rows_live = d_row < p.M;  // an odd number of 128-row blocks leaves the peer's last block outside the matrix
      constexpr bool bf = BF16;
      const int sw = row & 7;
      if constexpr (EPI == EPI_SWIGLU) {
        // accumulator columns [0, 128) = gate, [128, 256) = up of features n_blk * 128 ...; 64 features per round, a row's two
        // threads take 32 of them each into the three staging tiles (gate | up | act), then three TMA stores. The arithmetic of a
        // round is done before the tiles are waited for, so that it overlaps the stores of the round before.
        const int F = p.epi_cols;
        for (int c = 0; c < 2 && rows_live; ++c) {
          const int fcol = n_blk * (BN / 2) + c * 64;
          if (fcol >= F) break;
          uint32_t g[32], u[32], wg[16], wu[16], wa[16];
          tmem_ld_32x32b_x32(t_row + c * 64 + half * 32, g);
          tmem_ld_32x32b_x32(t_row + BN / 2 + c * 64 + half * 32, u);
          tmem_ld_wait();
          pack32(g, wg, bf);
          pack32(u, wu, bf);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 gg = unpack16(wg[e], bf), uu = unpack16(wu[e], bf);
            wa[e] = pack16(gg.x / (1.f + __expf(-gg.x)) * uu.x, gg.y / (1.f + __expf(-gg.y)) * uu.y, bf);
          }
          if (et == 0 && pending_stores > 0) tma_wait_group_read<0>();  // the previous round has left the tiles
          named_barrier_sync(epi_bar, kGroup);
          stage32(staging + row * 128, sw, half * 4, wg);
          stage32(staging + (BM + row) * 128, sw, half * 4, wu);
          stage32(staging + (2 * BM + row) * 128, sw, half * 4, wa);
          fence_proxy_async_smem();
          named_barrier_sync(epi_bar, kGroup);
          if (et == 0) {
            tma_store_2d(&tmD, smem_u32(staging), fcol, d_row);
            tma_store_2d(&tmD, smem_u32(staging + BM * 128), F + fcol, d_row);
            tma_store_2d(&tmE, smem_u32(staging + 2 * BM * 128), fcol, d_row);
            tma_commit_group();
          }
          pending_stores = 1;
        }
      } else if constexpr (EPI == EPI_SWIGLU_ACT) {
        // group g takes the 64 features of chunk g through its own staging tile; the arithmetic is EPI_SWIGLU's, on the rounded values
        const int fcol = n_blk * (BN / 2) + grp * 64;
        if (rows_live && fcol < p.epi_cols) {
          uint8_t* tile_a = staging + grp * (BM * 128);
          if (et == 0 && pending_stores > 0) tma_wait_group_read<0>();
          named_barrier_sync(epi_bar, kGroup);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t g[32], u[32], wa[16];
            tmem_ld_32x32b_x32(t_row + grp * 64 + h * 32, g);
            tmem_ld_32x32b_x32(t_row + BN / 2 + grp * 64 + h * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float2 gg = unpack16(pack16(__uint_as_float(g[2 * e]), __uint_as_float(g[2 * e + 1]), bf), bf);
              const float2 uu = unpack16(pack16(__uint_as_float(u[2 * e]), __uint_as_float(u[2 * e + 1]), bf), bf);
              wa[e] = pack16(gg.x / (1.f + __expf(-gg.x)) * uu.x, gg.y / (1.f + __expf(-gg.y)) * uu.y, bf);
            }
            stage32(tile_a + row * 128, sw, h * 4, wa);
          }
          fence_proxy_async_smem();
          named_barrier_sync(epi_bar, kGroup);
          if (et == 0) {
            tma_store_2d(&tmD, smem_u32(tile_a), fcol, d_row);
            tma_commit_group();
          }
          pending_stores = 1;
        }
      } else if constexpr (EPI == EPI_ROPE) {
        // 128 columns a round, in two staging tiles; of every 32 column pairs a row's two threads rotate 16 each. head_dim 64: two
        // heads, the partners are the 32-column halves of one tile; head_dim 128: one head, column i of the first tile rotates
        // with column i of the second.
        const bool wide = p.half_dim == 64;
        const int lo1 = wide ? 32 : 64, to_hi = wide ? 64 : 32;  // first column of the second 32 pairs; distance of the partners
        for (int g = 0; g < BN / 128 && rows_live; ++g) {
          const int gcol = n_blk * BN + g * 128;  // (at head_dim 64 the second head may lie outside the matrix)
          if (gcol >= p.N) break;
          uint32_t lo[2][16], hi[2][16];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            tmem_ld_32x32b_x16(t_row + g * 128 + h * lo1 + half * 16, lo[h]);
            tmem_ld_32x32b_x16(t_row + g * 128 + h * lo1 + to_hi + half * 16, hi[h]);
          }
          tmem_ld_wait();
          if (gcol < p.epi_cols) rope16(lo[0], hi[0], rope_c[0], rope_s[0], bf);
          if (wide) {
            if (gcol < p.epi_cols) rope16(lo[1], hi[1], rope_c[1], rope_s[1], bf);
          } else if (gcol + 64 < p.epi_cols) {
            rope16(lo[1], hi[1], rope_c[0], rope_s[0], bf);
          }
          if (et == 0 && pending_stores > 0) tma_wait_group_read<0>();
          named_barrier_sync(epi_bar, kGroup);
          uint8_t *row0 = staging + row * 128, *row1 = row0 + BM * 128;
          stage16(row0, sw, half * 2, lo[0], bf);
          stage16(wide ? row0 : row1, sw, (wide ? 4 : 0) + half * 2, lo[1], bf);
          stage16(wide ? row1 : row0, sw, (wide ? 0 : 4) + half * 2, hi[0], bf);
          stage16(row1, sw, 4 + half * 2, hi[1], bf);
          fence_proxy_async_smem();
          named_barrier_sync(epi_bar, kGroup);
          if (et == 0) {
            tma_store_2d(&tmD, smem_u32(staging), gcol, d_row);
            if (gcol + 64 < p.N) tma_store_2d(&tmD, smem_u32(staging + BM * 128), gcol + 64, d_row);
            tma_commit_group();
          }
          pending_stores = 1;
        }
      } else {
        const int cols_per_chunk = p.out_f32 ? 32 : 64;
        const int chunks = BN / cols_per_chunk;
        constexpr int G = Cfg<EPI>::kEpiGroups;  // with two groups: group g takes chunks g, g + 2 through staging tile g
        constexpr bool kStats = EPI == EPI_CE_STATS || EPI == EPI_CE_LOSS, kStore = EPI != EPI_CE_LOSS;
        float st_m = -INFINITY, st_s = 0.f;  // kStats: this row's running (max, sum of exp) over the group's chunks of the tile
        for (int c = (G == 2 ? grp : 0); c < chunks && rows_live; c += G) {
          const int col0 = c * cols_per_chunk;
          if (n_blk * BN + col0 >= p.N) break;
          uint8_t* buf = staging + (G == 2 ? grp : (int)(gchunk & 1)) * (BM * 128);
          ++gchunk;
          if (!kStore) {
          } else if (G == 2) {
            if (et == 0 && pending_stores >= 1) tma_wait_group_read<0>();
          } else if (et == 0 && pending_stores >= 2) {
            tma_wait_group_read<1>();
          }
          if (kStore) named_barrier_sync(epi_bar, kGroup);
          uint8_t* my_row = buf + row * 128;
          if (p.out_f32) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_row + col0, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(my_row + ((j ^ sw) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          } else {
            uint32_t r0[32], r1[32], w0[16], w1[16];
            tmem_ld_32x32b_x32(t_row + col0, r0);
            tmem_ld_32x32b_x32(t_row + col0 + 32, r1);
            tmem_ld_wait();
            pack32(r0, w0, bf);
            pack32(r1, w1, bf);
            if constexpr (kStats) {
              constexpr float kLog2e = 1.4426950408889634f;
              float x[64];
              float cm = -INFINITY;
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const float2 a = unpack16(w0[e], bf), b = unpack16(w1[e], bf);
                x[2 * e] = a.x; x[2 * e + 1] = a.y; x[32 + 2 * e] = b.x; x[32 + 2 * e + 1] = b.y;
                cm = fmaxf(cm, fmaxf(fmaxf(a.x, a.y), fmaxf(b.x, b.y)));
              }
              if (cm > st_m) {
                st_s *= exp2f((st_m - cm) * kLog2e);
                st_m = cm;
              }
              const float mb = st_m * kLog2e;
#pragma unroll
              for (int i = 0; i < 64; ++i) st_s += exp2f(x[i] * kLog2e - mb);
              if constexpr (EPI == EPI_CE_LOSS) {
                const long long off = tgt_col - col0;  // one chunk of the whole row holds the target: the branch is rarely taken
                if (off >= 0 && off < 64) {
                  float xt = 0.f;
#pragma unroll
                  for (int i = 0; i < 64; ++i) xt = i == (int)off ? x[i] : xt;
                  p.target_logit[d_row + row] = xt;
                }
              }
            }
            if constexpr (kStore) {
              stage32(my_row, sw, 0, w0);
              stage32(my_row, sw, 4, w1);
            }
          }
          if constexpr (!kStore) continue;
          fence_proxy_async_smem();
          named_barrier_sync(epi_bar, kGroup);
          if (et == 0) {
            if (p.reduce_add) tma_reduce_add_2d(&tmD, smem_u32(buf), n_blk * BN + col0, d_row);
            else tma_store_2d(&tmD, smem_u32(buf), n_blk * BN + col0, d_row);
            tma_commit_group();
          }
          if (pending_stores < 2) ++pending_stores;
        }
        if constexpr (kStats) {
          if (rows_live && d_row + row < p.M)
            *reinterpret_cast<float2*>(p.stats + (((size_t)(d_row + row) * p.n_blocks + n_blk) * G + grp) * 2) = make_float2(st_m, st_s);
        }
      }
      // this CTA's half of the accumulator has been read: tell the leader's MMA thread
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (rank == 0) mbar_arrive(bar_tempty + 8 * acc);
        else mbar_arrive_cluster(leader_tempty + 8 * acc);
      }
    }
    if (et == 0) tma_wait_group<0>();
  }

  if (fail_item >= 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, 1) == 0) {
      p.status[1] = fail_role;
      p.status[2] = blockIdx.x;
      p.status[3] = fail_item;
    }
  }
  // The peer's shared memory and barriers are in use until the leader's last MMA and commit have completed, and the pair
  // frees its tensor memory together: meet before leaving.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, kTmemCols);
  }
}

}  // namespace

namespace {

template <int EPI, bool BF16>
int max_resident_pairs() {
  static int max_clusters = -1;
  if (max_clusters < 0) {
    auto kern = gemm2_tcgen05_kernel<EPI, BF16>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<EPI>::kSmemBytes) != cudaSuccess) {
      nnb_set_error("gemm2: cannot reserve %d bytes of shared memory", Cfg<EPI>::kSmemBytes);
      cudaGetLastError();
      return -3;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * (nnb_num_sms() / 2));
    cfg.blockDim = dim3(Cfg<EPI>::kThreads);
    cfg.dynamicSmemBytes = Cfg<EPI>::kSmemBytes;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = 0; }
    max_clusters = n;
  }
  return max_clusters;
}

template <int EPI, bool BF16>
int launch2(const NnbGemm2Args& a, cudaStream_t st) {
  const int sms = a.max_ctas > 0 ? min(a.max_ctas, nnb_num_sms()) : nnb_num_sms();
  const int resident = max_resident_pairs<EPI, BF16>();
  if (resident < 0) return resident;
  const int pairs = min(sms / 2, resident);  // persistent pairs must all be resident at once
  if (pairs < 1 || a.M < 2 * BM || a.N < BN / 2) return 1;
  Params2 p{};
  p.M = a.M; p.N = a.N; p.K = a.K;
  p.m_pairs = (a.M + 2 * BM - 1) / (2 * BM);
  p.n_blocks = (a.N + BN - 1) / BN;
  p.kblocks_total = (a.K + BK - 1) / BK;
  if (EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_ACT) {
    // a.N = 2 F (rows of the gate||up weight); one tile = 128 features = gate and up columns of the same features
    NNB_REQUIRE(!a.out_f32 && !a.a_mn && !a.b_mn && !a.accumulate && a.E != nullptr, "gemm_swiglu: plain K-major 16-bit problem expected");
    NNB_REQUIRE(a.N % 256 == 0, "gemm_swiglu: F = %d must be a multiple of 128", a.N / 2);
    p.epi_cols = a.N / 2;
    p.n_blocks = p.epi_cols / (BN / 2);
  } else if (EPI == EPI_ROPE) {
    NNB_REQUIRE(!a.out_f32 && !a.accumulate, "gemm_rope: 16-bit output expected");
    NNB_REQUIRE((a.head_dim == 64 || a.head_dim == 128) && a.rope_cols % a.head_dim == 0 && a.N % a.head_dim == 0 && a.t_len > 0 &&
                    a.cos_t != nullptr && a.sin_t != nullptr && nnb_aligned16(a.cos_t) && nnb_aligned16(a.sin_t),
                "gemm_rope: head_dim must be 64 or 128, columns whole heads, tables 16-byte aligned");
    p.epi_cols = a.rope_cols; p.t_len = a.t_len; p.half_dim = a.head_dim / 2;
    p.cos_t = static_cast<const float*>(a.cos_t); p.sin_t = static_cast<const float*>(a.sin_t);
  } else if (EPI == EPI_CE_LOSS) {
    NNB_REQUIRE(!a.out_f32 && !a.accumulate && a.N % 64 == 0 && a.stats != nullptr && a.targets != nullptr && a.target_logit != nullptr,
                "gemm_ce_loss: N a multiple of 64, targets and both outputs expected");
    p.stats = static_cast<float*>(a.stats);
    p.targets = static_cast<const long long*>(a.targets);
    p.target_logit = static_cast<float*>(a.target_logit);
  } else if (EPI == EPI_CE_STATS) {
    NNB_REQUIRE(!a.out_f32 && !a.accumulate && a.N % 64 == 0 && a.stats != nullptr, "gemm_ce_stats: 16-bit output with N a multiple of 64 expected");
    p.stats = static_cast<float*>(a.stats);
  } else if (EPI == EPI_SWIGLU_BWD) {
    NNB_REQUIRE(!a.out_f32 && !a.accumulate && a.N % 64 == 0 && a.E != nullptr && nnb_aligned16(a.E) && a.lde % 8 == 0,
                "gemm_swiglu_bwd: 16-bit output, F a multiple of 64 and an aligned saved projection expected");
    p.epi_cols = a.N;
  }
  const int splits = a.out_f32 ? max(1, min(a.k_splits, p.kblocks_total)) : 1;
  p.chain = a.chain;
  p.kblocks_per_split = (p.kblocks_total + splits - 1) / splits;
  p.k_splits = (p.kblocks_total + p.kblocks_per_split - 1) / p.kblocks_per_split;
  p.group_m = 1;
  {
    int g = 1;
    while ((g + 1) * (g + 1) * 2 * BM <= pairs * BN) ++g;  // least wave footprint: group_m = sqrt(pairs BN / (2 BM))
    if (p.n_blocks * g > pairs) p.group_m = min(g, p.m_pairs);
  }
  p.a_mn = a.a_mn ? 1 : 0;
  p.b_mn = a.b_mn ? 1 : 0;
  p.out_f32 = a.out_f32 ? 1 : 0;
  p.reduce_add = (a.accumulate || p.k_splits > 1) ? 1 : 0;
  p.out_bf16 = a.dtype == NNB_BF16 ? 1 : 0;
  p.idesc = sm100::make_idesc_f16(a.dtype == NNB_BF16 ? 1 : 0, p.a_mn, p.b_mn, 2 * BM, BN);
  p.status = static_cast<int*>(a.status);
  const CUtensorMapDataType in_dt = a.dtype == NNB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tmA, tmB, tmD, tmE;
  if (!p.a_mn) { if (!nnb_make_tmap_2d(&tmA, in_dt, 2, a.A, a.M, a.K, a.lda * 2, BM, BK, "gemm2 A")) return -4; }
  else         { if (!nnb_make_tmap_2d(&tmA, in_dt, 2, a.A, a.K, a.M, a.lda * 2, BK, 64, "gemm2 A^T")) return -4; }
  if (!p.b_mn) { if (!nnb_make_tmap_2d(&tmB, in_dt, 2, a.B, a.N, a.K, a.ldb * 2, BN / 2, BK, "gemm2 B")) return -4; }
  else         { if (!nnb_make_tmap_2d(&tmB, in_dt, 2, a.B, a.K, a.N, a.ldb * 2, BK, 64, "gemm2 B^T")) return -4; }
  const CUtensorMapDataType d_dt = a.out_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : in_dt;
  const int d_bytes = a.out_f32 ? 4 : 2, d_box = a.out_f32 ? 32 : 64;
  // (EPI_SWIGLU_BWD writes d(gate) | d(up): its output, like the projection it reads through tmE, is 2 N columns wide)
  const int d_cols = EPI == EPI_SWIGLU_BWD ? 2 * a.N : a.N;
  if (EPI == EPI_CE_LOSS) tmD = tmA;  // nothing is stored
  else if (EPI == EPI_SWIGLU_ACT) { if (!nnb_make_tmap_2d(&tmD, in_dt, 2, a.E, a.M, a.N / 2, a.lde * 2, BM, 64, "gemm2 act")) return -4; }
  else if (!nnb_make_tmap_2d(&tmD, d_dt, d_bytes, a.D, a.M, d_cols, a.ldd * d_bytes, BM, d_box, "gemm2 D")) return -4;
  tmE = tmD;
  if (EPI == EPI_SWIGLU_BWD && !nnb_make_tmap_2d(&tmE, in_dt, 2, a.E, a.M, 2 * a.N, a.lde * 2, BM, 64, "gemm2 gate|up")) return -4;
  if (EPI == EPI_SWIGLU && !nnb_make_tmap_2d(&tmE, in_dt, 2, a.E, a.M, a.N / 2, a.lde * 2, BM, 64, "gemm2 act")) return -4;
  if (a.out_f32 && !a.accumulate && p.k_splits > 1) {
    if (a.ldd == a.N) cudaMemsetAsync(a.D, 0, (size_t)a.M * a.N * 4, st);
    else cudaMemset2DAsync(a.D, a.ldd * 4, 0, (size_t)a.N * 4, a.M, st);
  }
  const int items = p.m_pairs * p.n_blocks * p.k_splits;
  const int grid = 2 * min(items, pairs);
  nnb_launch(gemm2_tcgen05_kernel<EPI, BF16>, grid, Cfg<EPI>::kThreads, Cfg<EPI>::kSmemBytes, st, tmA, tmB, tmD, tmE, p);
  NNB_LAUNCH_OK("gemm2_tcgen05");
  return 0;
}

}  // namespace

int nnb_gemm2_launch(const NnbGemm2Args& a, cudaStream_t st) {
#define NNB_LAUNCH2(E) (a.dtype == NNB_BF16 ? launch2<E, true>(a, st) : launch2<E, false>(a, st))
  if (a.epilogue == EPI_NONE && a.out_f32 && a.k_splits <= 0) {
    const int sms = a.max_ctas > 0 ? min(a.max_ctas, nnb_num_sms()) : nnb_num_sms();
    const int resident = a.dtype == NNB_BF16 ? max_resident_pairs<EPI_NONE, true>() : max_resident_pairs<EPI_NONE, false>();
    const long long tiles = (long long)((a.M + 2 * BM - 1) / (2 * BM)) * ((a.N + BN - 1) / BN);
    NnbGemm2Args f = a;
    nnb_plan_k(tiles, max(1, min(sms / 2, resident)), (a.K + BK - 1) / BK, 0.5, (double)a.M * a.N * 4, a.accumulate != 0, f.k_splits, f.chain);
    if (f.chain > 0) return a.dtype == NNB_BF16 ? launch2<EPI_CHAINED, true>(f, st) : launch2<EPI_CHAINED, false>(f, st);
    return a.dtype == NNB_BF16 ? launch2<EPI_NONE, true>(f, st) : launch2<EPI_NONE, false>(f, st);
  }
  switch (a.epilogue) {
    case EPI_NONE: return NNB_LAUNCH2(EPI_NONE);
    case EPI_SWIGLU: return NNB_LAUNCH2(EPI_SWIGLU);
    case EPI_ROPE: return NNB_LAUNCH2(EPI_ROPE);
    case EPI_CE_STATS: return NNB_LAUNCH2(EPI_CE_STATS);
    case EPI_SWIGLU_BWD: return NNB_LAUNCH2(EPI_SWIGLU_BWD);
    case EPI_CE_LOSS: return NNB_LAUNCH2(EPI_CE_LOSS);
    case EPI_SWIGLU_ACT: return NNB_LAUNCH2(EPI_SWIGLU_ACT);
    default: nnb_set_error("gemm2: unknown epilogue %d", a.epilogue); return -1;
  }
#undef NNB_LAUNCH2
}

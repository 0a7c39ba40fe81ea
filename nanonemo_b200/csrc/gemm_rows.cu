// Products of a few hundred rows with a weight: D[M, N] = A[M, K] * W[N, K]^T, 16-bit A, W in fp32 or 16 bits, fp32 accumulation, on tcgen05 / TMA.
//
// Scoring or decoding a short text is 4 such products a layer with M = 16 ... 512. What bounds them is not arithmetic: the weights
// come out of HBM once, every SM can take in only so many bytes of its tile, and the latencies of one tile (first loads, last products,
// store) are as long as its loop. The tiles of gemm.cu (128 x 128 and wider, for thousands of rows) leave most SMs without work there, and
// a weight that exists in fp32 only (a model that no training engine keeps a 16-bit copy of) cost a launch and three passes over it
// for the cast. Hence:
//   * tiles of 128 rows x 32, 64 or 128 columns, each one K loop (the sums, and so the bits, are those of gemm.cu);
//   * W arrives as it is, fp32 by TMA into a ring, and eight warps round it into the swizzled 16-bit operand tile (round to nearest even, the
//     bits that the cast would give);
//   * the columns of a tile are two groups of weight rows that may lie apart, so that rotate-half partners (RoPE) or gate and up (SwiGLU)
//     of the same features meet in one thread of the epilogue, whose arithmetic on the rounded values is that of the stand-alone kernels;
//   * a block that waits for the previous kernel (programmatic launch) meanwhile asks for its weight tiles in L2.
// Roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 convert the weight, then run the epilogue (with four of them 201 x 768 x
// 768 from 16 bits took 4.5 us, now 4.2). All waits are bounded.
// In a row with 24 weights (as a model has them), us, before / now: 201 rows of 768, cast + product of 768 x 768 9.7 / 5.1, + RoPE of 1280 x 768
// 10.3 + 4.3 / 6.3, + SwiGLU of 4096 x 768 11.0 + 2.2 / 7.3, 768 x 2048 15.7 / 9.2; 16-bit weights: see nnb_rows_tile.
// Replaces the cuBLAS calls behind nn.Linear in the reference's evaluation (nanonemo/model/layers.py:80-83, 128-130).
#include "common.cuh"
#include "gemm2.cuh"
#include "sm100.cuh"

namespace {

using namespace sm100;

constexpr int BM = 128;
constexpr int kBlock = 64;  // K columns of a swizzled operand block
constexpr int kThreads = 320, kWorkThreads = 256;
enum RowsEpilogue : int { ROWS_NONE = 0, ROWS_ROPE = 1, ROWS_SWIGLU = 2 };

// G: weight rows per group; a tile has 2 G columns. SUB: 64-column blocks of K in a stage (a pass of the MMA warp over its barriers takes as
// long as eight products of the narrow tiles: two blocks a stage there). The ring is as deep as one CTA per SM allows, or two where there
// are more tiles than SMs.
template <int G, bool F32W>
struct RCfg {
  static constexpr int BN = 2 * G, SUB = G == 64 || (F32W && G == 32) ? 1 : 2 /* (two stages of 80 KB in fp32: 29 us for 777 x 768 x 4096, five of 40 27) */, BK = SUB * kBlock;
  static constexpr int kBytesA = BM * BK * 2, kBytesW = BN * BK * 2, kBytesF = F32W ? BN * BK * 4 : 0;
  static constexpr int kStageBytes = kBytesA + kBytesF + kBytesW;
  static constexpr int kMaxStages = 225 * 1024 / kStageBytes < 8 ? 225 * 1024 / kStageBytes : 8;
  static constexpr int kTwoPerSm = 112 * 1024 / kStageBytes;
  static constexpr int kTxBytes = kBytesA + (F32W ? kBytesF : kBytesW);
  static constexpr int kRowFloats = BN + 4;  // a row of the fp32 sums in shared memory (padded: no bank conflicts)
  static constexpr int smem(int stages) { return stages * kStageBytes + 256; }
  static_assert(BM * kRowFloats * 4 <= kTwoPerSm * kStageBytes && kTwoPerSm >= 2, "the sums take the ring's place");
  static constexpr int kTmemCols = BN;
};

struct RParams {
  int M, N, K;          // N: columns of D (the weight has N rows, 2 N for SwiGLU)
  int kblocks, stages;
  int tiles_per_half;   // RoPE: tiles that share a half head
  int head_dim, rope_cols, t_len;
  uint32_t idesc;
  void* D;
  long long ldd;
  const float *cos_t, *sin_t;
  int* status;
};

template <bool BF16>
__device__ __forceinline__ uint32_t pack_rn(float a, float b) { return pack2_16<!BF16>(a, b); }
template <bool BF16>
__device__ __forceinline__ float round16(float x) {
  if constexpr (BF16) return __bfloat162float(__float2bfloat16_rn(x));
  else return __half2float(__float2half_rn(x));
}

// BMN: W is stored [K, N] (an input gradient's weight). In fp32 its boxes, [64 K rows][32 columns], are as many and as large as those of 64 weight rows.
template <int G, bool BF16, bool F32W, bool BMN, int EPI>
__global__ void __launch_bounds__(kThreads) gemm_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const RParams p) {
  using C = RCfg<G, F32W>;
  constexpr int BN = C::BN, BK = C::BK;
  static_assert(!BMN || (G >= 32 && EPI == ROWS_NONE && (!F32W || G == 32)), "");
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t stages = p.stages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * C::kStageBytes);
  constexpr int kMax = C::kMaxStages;
  const uint32_t bar_full = smem_u32(bars), bar_conv = bar_full + 8 * kMax, bar_empty = bar_conv + 8 * kMax, bar_acc = bar_empty + 8 * kMax;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kMax + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* never_set = abort_flag + 1;
  static_assert((3 * kMax + 1) * 8 + 12 <= 256, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool aligned = (smem_u32(smem) & 1023) == 0;  // (swizzled tiles; nothing is issued otherwise)
  const int tile = blockIdx.x, m0 = blockIdx.y * BM;
  // first weight row of either group; D's columns of the groups are the same numbers, except for SwiGLU (gate row = feature = column)
  int r0, r1;
  if (EPI == ROWS_ROPE) {
    r0 = tile / p.tiles_per_half * p.head_dim + tile % p.tiles_per_half * G;
    r1 = r0 + p.head_dim / 2;
  } else if (EPI == ROWS_SWIGLU) {
    r0 = tile * G;
    r1 = p.N + r0;
  } else {
    r0 = tile * BN;
    r1 = r0 + G;
  }
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < kMax; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_conv + 8 * s, kWorkThreads);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_acc, 1);
    *abort_flag = *never_set = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmW);
    // Weight tiles into L2 while the previous kernel ends. (L2 is where every write ends up: a weight that the previous kernel still
    // writes is not seen too early, this only brings the line closer.)
    for (int kb = 0; kb < p.kblocks; ++kb) {
#pragma unroll
      for (int x = 0; x < BK; x += F32W ? 32 : 64) {
        if (kb * BK + x >= p.K) break;
        if (BMN) {
          if (x % kBlock) continue;
          tma_prefetch_l2_2d(&tmW, r0, kb * BK + x);
          if ((G > 32 || F32W) && r1 < p.N) tma_prefetch_l2_2d(&tmW, r1, kb * BK + x);
        } else {
          tma_prefetch_l2_2d(&tmW, kb * BK + x, r0);
          if (EPI != ROWS_NONE || r1 < p.N) tma_prefetch_l2_2d(&tmW, kb * BK + x, r1);
        }
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const float *cos_t = p.cos_t, *sin_t = p.sin_t;
  nnb_after_previous(cos_t, sin_t);
  int fail_role = aligned ? 0 : 6;
  bool ok = aligned;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t s = 0, ph = 0;
      int kb = 0;
      for (; kb < p.kblocks && ok; ++kb) {
        ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag);
        if (!ok) { if (aligned) fail_role = 1; break; }
        const uint32_t full = bar_full + 8 * s, sa = smem_u32(smem) + s * C::kStageBytes, sw = sa + C::kBytesA;
        mbar_expect_tx(full, C::kTxBytes);
        constexpr int kWCols = F32W ? 32 : 64;  // columns of a 128-byte box row; boxes are [2 G rows][128 bytes]
#pragma unroll
        for (int x = 0; x < BK / 64; ++x) tma_load_2d(sa + x * BM * 128, &tmA, full, kb * BK + x * 64, m0);
#pragma unroll
        for (int x = 0; x < BK / kWCols; ++x) {
          if (BMN && F32W) {  // [64 K rows][32 columns] boxes: r0 and r1 are 32 columns apart
            tma_load_2d(sw + x * BN * 128, &tmW, full, x % 2 ? r1 : r0, kb * BK + x / 2 * kBlock);
          } else if (BMN) {  // [64 K rows][64 columns] boxes, one after the other along the tile's columns
            tma_load_2d(sw + x * BN * 128, &tmW, full, r0, kb * BK + x * kBlock);
            if (G > 32) tma_load_2d(sw + x * BN * 128 + kBlock * 128, &tmW, full, r1, kb * BK + x * kBlock);
          } else {
            tma_load_2d(sw + x * BN * 128, &tmW, full, kb * BK + x * kWCols, r0);
            tma_load_2d(sw + x * BN * 128 + G * 128, &tmW, full, kb * BK + x * kWCols, r1);
          }
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      nnb_release_next();
      if (!ok)  // what was requested has to land before the shared memory is given up
        for (int i = max(0, kb - (int)stages); i < kb; ++i) mbar_wait(bar_full + 8 * (i % stages), (i / stages) & 1, never_set);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform: see umma_f16_elect)
    const bool el = elect_one();
    uint32_t s = 0, ph = 0;
    for (int kb = 0; kb < p.kblocks && ok; ++kb) {
      ok = mbar_wait(bar_full + 8 * s, ph, abort_flag) && (!F32W || mbar_wait(bar_conv + 8 * s, ph, abort_flag));
      if (!ok) { fail_role = lane == 0 ? 2 : 0; break; }
      tc_fence_after();
      const uint32_t sa = smem_u32(smem) + s * C::kStageBytes, sw = sa + C::kBytesA + C::kBytesF;
#pragma unroll
      for (int k = 0; k < BK / 16; ++k)
        umma_f16_elect(el, tmem_base, make_smem_desc(sa + k / 4 * (BM * 128) + k % 4 * 32, 16, 1024),
                       make_smem_desc(sw + k / 4 * (BN * 128) + k % 4 * (BMN ? 16 * 128 : 32), BMN ? kBlock * 128 : 16, 1024), p.idesc, (kb > 0 || k > 0) ? 1u : 0u);
      umma_commit_elect(el, bar_empty + 8 * s);
      if (++s == stages) { s = 0; ph ^= 1; }
    }
    if (ok) umma_commit_elect(el, bar_acc);
  } else {
    const int t = threadIdx.x - 64;
    if (F32W) {
      // ---------------------------------------------------------------- conversion: 8 weights a step, 32 bytes in, 16 out
      uint32_t s = 0, ph = 0;
      for (int kb = 0; kb < p.kblocks && ok; ++kb) {
        ok = mbar_wait(bar_full + 8 * s, ph, abort_flag);
        if (!ok) { fail_role = 4; break; }
        const uint8_t* src = smem + s * C::kStageBytes + C::kBytesA;
        uint8_t* dst = smem + s * C::kStageBytes + C::kBytesA + C::kBytesF;
        constexpr int kUnits = BN * BK / 8 / kWorkThreads;  // all loads before the first store: which the compiler, for all it knows, may overwrite what is to be loaded
        float4 v[kUnits][2];
#pragma unroll
        for (int i = 0; i < kUnits; ++i) {
          const int u = t + i * kWorkThreads, r = (u >> 3) % BN, c = u & 7, x = u / (8 * BN);  // 16-byte unit c of the 16-bit row of block x = units 2 (c % 4), + 1 of its half c / 4
          const uint8_t* row = src + (2 * x + (c >> 2)) * BN * 128 + r * 128;
          const int odd = c >> 2;  // (the lanes of the second half take their units in the other order: eight different bank groups)
          v[i][0] = *reinterpret_cast<const float4*>(row + (((2 * (c & 3) + odd) ^ (r & 7)) << 4));
          v[i][1] = *reinterpret_cast<const float4*>(row + (((2 * (c & 3) + 1 - odd) ^ (r & 7)) << 4));
        }
#pragma unroll
        for (int i = 0; i < kUnits; ++i) {
          const int u = t + i * kWorkThreads, r = (u >> 3) % BN, c = u & 7, x = u / (8 * BN);
          const bool odd = c >> 2;
          const float4 a = odd ? v[i][1] : v[i][0], b = odd ? v[i][0] : v[i][1];
          *reinterpret_cast<uint4*>(dst + x * BN * 128 + r * 128 + ((c ^ (r & 7)) << 4)) =
              make_uint4(pack_rn<BF16>(a.x, a.y), pack_rn<BF16>(a.z, a.w), pack_rn<BF16>(b.x, b.y), pack_rn<BF16>(b.z, b.w));
        }
        fence_proxy_async_smem();
        mbar_arrive(bar_conv + 8 * s);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    }
    // ------------------------------------------------------------------ the fp32 sums -> shared memory (every load and product is complete)
    if (ok && !mbar_wait(bar_acc, 0, abort_flag)) { ok = false; fail_role = 3; }
    ok = !named_barrier_or(1, kWorkThreads, !ok);  // all leave together
    if (ok) {
      tc_fence_after();
      const int q = warp & 3;
      float* mine = reinterpret_cast<float*>(smem) + (q * 32 + lane) * C::kRowFloats;
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        if (BN > 32 && (c & 1) != (t >> 7)) continue;  // (two warps a lane quadrant)
        if (BN == 32 && t >= 128) break;
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) *reinterpret_cast<uint4*>(mine + c * 32 + e * 4) = make_uint4(r[4 * e], r[4 * e + 1], r[4 * e + 2], r[4 * e + 3]);
      }
      tc_fence_before();
    }
  }
  if (warp >= 2 && ok) {
    named_barrier_sync(1, kWorkThreads);
    // 8 + 8 columns of a row a step
    for (int u = (int)threadIdx.x - 64; u < BM * (G / 8); u += kWorkThreads) {
      const int row = u / (G / 8), c = u % (G / 8) * 8, m = m0 + row;
      if (m >= p.M) break;  // (rows grow with u)
      const float* sums = reinterpret_cast<const float*>(smem) + row * C::kRowFloats + c;
      float lo[8], hi[8];
      Chunk8<float>::load(sums, lo);
      Chunk8<float>::load(sums + G, hi);
      if (EPI == ROWS_ROPE && r0 < p.rope_cols) {
        const size_t at = (size_t)(m % p.t_len) * (p.head_dim / 2) + r0 % p.head_dim + c;
        float cs[8], sn[8];
        Chunk8<float>::load(cos_t + at, cs);
        Chunk8<float>::load(sin_t + at, sn);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float a = round16<BF16>(lo[i]), b = round16<BF16>(hi[i]);
          lo[i] = a * cs[i] - b * sn[i];
          hi[i] = a * sn[i] + b * cs[i];
        }
      }
      if (EPI == ROWS_SWIGLU) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float g = round16<BF16>(lo[i]), up = round16<BF16>(hi[i]);
          lo[i] = g / (1.f + __expf(-g)) * up;
        }
      }
      uint16_t* out = static_cast<uint16_t*>(p.D) + (size_t)m * p.ldd;
      auto store = [&](int col, const float (&v)[8]) {
        if (col < p.N)  // (N is a multiple of 8)
          *reinterpret_cast<uint4*>(out + col) = make_uint4(pack_rn<BF16>(v[0], v[1]), pack_rn<BF16>(v[2], v[3]), pack_rn<BF16>(v[4], v[5]), pack_rn<BF16>(v[6], v[7]));
      };
      store(r0 + c, lo);
      if (EPI != ROWS_SWIGLU) store(r1 + c, hi);
    }
  }
  if (fail_role != 0 && p.status != nullptr) {
    if (atomicCAS(p.status, 0, 4) == 0) {
      p.status[1] = fail_role;
      p.status[2] = blockIdx.x + gridDim.x * blockIdx.y;
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

template <int G, bool BF16, bool F32W, bool BMN, int EPI>
int launch_rows(const CUtensorMap& ta, const CUtensorMap& tw, RParams p, int tiles, int m_blocks, cudaStream_t st) {
  using C = RCfg<G, F32W>;
  p.kblocks = (p.K + C::BK - 1) / C::BK;
  p.stages = tiles * m_blocks > nnb_num_sms() ? C::kTwoPerSm : C::kMaxStages;
  auto kern = gemm_rows_kernel<G, BF16, F32W, BMN, EPI>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(C::kMaxStages)) != cudaSuccess) {
      nnb_set_error("gemm_rows: cannot reserve %d bytes of shared memory", C::smem(C::kMaxStages));
      return -3;
    }
    configured = true;
  }
  nnb_launch(kern, dim3(tiles, m_blocks), kThreads, C::smem(p.stages), st, ta, tw, p);
  NNB_LAUNCH_OK("gemm_rows");
  return 0;
}

}  // namespace

// Whether a product of M rows with an fp32 weight of N rows (kind 0; kind 1, SwiGLU: 2 N) and K columns is taken straight from it, and not from its cast.
// GPU time, us in a row, straight from fp32 / cast + product: 256 x 128 weights 2.7 / 4.5, 201 x 768 x 2048 9.2 / 11.6, 512 x 768 x 2048 10.2 / 11.7; more tiles than
// SMs 201 x 4096 x 768 8.4 / 9.3, 512 x 2048 x 768 8.3 / 8.4, 512 x 1280 x 768 8.1 / 7.7, 777 x 768 x 1024 9.7 / 8.0, 512 x 2048 x 2048 17.4 / 13.9 (not served). Up to K = 1024 the second
// wave is taken all the same: a cast costs the host of an eager call 5.5 us (10.0 / 15.5 us a forward call, whichever of these sizes) and few rows of a block
// their one workspace (binding.cpp): scoring 512 tokens 964 us, 1002 with a line at one wave, 800 tokens 1021 and 1125. SwiGLU gains at every size that it
// serves (201 x 2048 x 768 7.4 / 11.6). Fewest rows (nnb_rows_tile says why): 13 x 8304 x 856 17.9 / 14.8, 2 x 3040 x 4016 33.1 / 28.7; 1 x 4096 x 768 7.2 / 9.6.
// Input gradients (kind 2: the weight has K rows and N columns), us in a row, from fp32 / cast + 64-wide tiles: 201 x 768 x 768 6.3 / 6.9, 201 x 2048
// x 768 6.7 / 8.4, 777 x 768 x 768 6.7 / 7.0, 777 x 768 x 1280 9.5 / 9.1, 777 x 768 x 4096 26.7 / 20.1 (a stage waits for its 32 KB of weights to be
// rounded).
extern "C" int nnb_gemm_rows_f32w_serves(int M, int N, int K, int kind) {
  const long long sms = nnb_num_sms(), cols = kind == 2 ? 64 : kind == 1 ? 16 : 32, t = (long long)((M + BM - 1) / BM) * ((N + cols - 1) / cols);
  if (kind == 0 && (long long)M * K < 1 << 16 && ((long long)N * K > 1 << 22 || t > sms)) return 0;
  return kind == 2 ? t <= sms && K <= 1024 : t <= sms || (t <= 2 * sms && K <= 1024);
}

namespace {

template <bool F32W, bool BMN, int EPI>
int rows_impl(const void* A, const void* W, void* D, int M, int N, int K, long long lda, long long ldw, long long ldd, int dtype, RParams& p, int g, void* status, cudaStream_t st) {
  const int w_bytes = F32W ? 4 : 2;
  if (N % 8 || ldd % 8 || lda % 8 || ldw * w_bytes % 16 || !nnb_aligned16(A) || !nnb_aligned16(W) || !nnb_aligned16(D)) return 1;
  p.M = M; p.N = N; p.K = K;
  p.D = D; p.ldd = ldd;
  p.status = static_cast<int*>(status);
  const int m_blocks = (M + BM - 1) / BM, tiles = EPI == ROWS_SWIGLU ? (N + g - 1) / g : (N + 2 * g - 1) / (2 * g);
  if (EPI == ROWS_SWIGLU && N % g) return 1;
  if (EPI == ROWS_ROPE) {
    if (p.head_dim / 2 % g) return 1;
    p.tiles_per_half = p.head_dim / 2 / g;
  }
  p.idesc = make_idesc_f16(dtype == NNB_BF16 ? 1 : 0, 0, BMN ? 1 : 0, BM, 2 * g);
  const CUtensorMapDataType in_dt = dtype == NNB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap ta, tw;
  if (!nnb_make_tmap_2d(&ta, in_dt, 2, A, M, K, lda * 2, BM, kBlock, "gemm_rows A")) return -4;
  if (BMN) {
    if (!nnb_make_tmap_2d(&tw, F32W ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : in_dt, w_bytes, W, K, N, ldw * w_bytes, kBlock, F32W ? 32 : kBlock, "gemm_rows W^T")) return -4;
  } else if (!nnb_make_tmap_2d(&tw, F32W ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : in_dt, w_bytes, W, EPI == ROWS_SWIGLU ? 2 * N : N, K, ldw * w_bytes, g, F32W ? 32 : kBlock, "gemm_rows W")) {
    return -4;
  }
#define NNB_ROWS(GG) (dtype == NNB_BF16 ? launch_rows<GG, true, F32W, BMN, EPI>(ta, tw, p, tiles, m_blocks, st) : launch_rows<GG, false, F32W, BMN, EPI>(ta, tw, p, tiles, m_blocks, st))
  if constexpr (F32W) {
    NNB_REQUIRE(g == (BMN ? 32 : 16) || (EPI == ROWS_SWIGLU && g == 32), "gemm_rows: no tile of %d", g);
    if constexpr (BMN) {
      if (!nnb_gemm_rows_f32w_serves(M, N, K, 2)) return 1;
      return NNB_ROWS(32);
    } else {
      if (!nnb_gemm_rows_f32w_serves(M, N, K, EPI == ROWS_SWIGLU ? 1 : 0)) return 1;
      if constexpr (EPI == ROWS_SWIGLU) {
        if (g == 32) return NNB_ROWS(32);
      }
      return NNB_ROWS(16);
    }
  } else {
    NNB_REQUIRE(g == 32 || g == 64, "gemm_rows: no tile of %d", g);
    return g == 32 ? NNB_ROWS(32) : NNB_ROWS(64);
  }
#undef NNB_ROWS
}

bool operands_ok(int M, int N, int K, int dtype) {
  if (M > 0 && N > 0 && K > 0 && (dtype == NNB_BF16 || dtype == NNB_F16)) return true;
  nnb_set_error("gemm_rows: bad problem %dx%dx%d or dtype code %d", M, N, K, dtype);
  return false;
}

}  // namespace

// D[M, N] = A[M, K] W[N, K]^T (w_mn: W is stored [K, N]), W in the dtype of A. Strides in elements. g: columns of a tile / 2, 32 or 64. Answers 1, with
// nothing launched, where operands are not aligned for it.
extern "C" int nnb_gemm_rows(const void* A, const void* W, void* D, int M, int N, int K, long long lda, long long ldw, long long ldd, int w_mn, int dtype, int g, void* status,
                             cudaStream_t st) {
  if (!operands_ok(M, N, K, dtype)) return -1;
  RParams p{};
  return w_mn ? rows_impl<false, true, ROWS_NONE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, g, status, st)
              : rows_impl<false, false, ROWS_NONE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, g, status, st);
}

// The same with rotate-half RoPE on columns [0, rope_cols) in heads of head_dim (64 or 128), row m at position m % t_len; tables fp32 [t_len, head_dim / 2].
// f32w: W in fp32 (g is 16 then).
extern "C" int nnb_gemm_rows_rope(const void* A, const void* W, void* D, const void* cos_t, const void* sin_t, int M, int N, int K, long long lda, long long ldw, long long ldd,
                                  int t_len, int rope_cols, int head_dim, int dtype, int f32w, int g, void* status, cudaStream_t st) {
  if (!operands_ok(M, N, K, dtype)) return -1;
  NNB_REQUIRE((head_dim == 64 || head_dim == 128) && N % head_dim == 0 && rope_cols % head_dim == 0 && t_len > 0 && cos_t != nullptr && sin_t != nullptr,
              "gemm_rows_rope: head_dim must be 64 or 128 and columns whole heads");
  if (!nnb_aligned16(cos_t) || !nnb_aligned16(sin_t)) return 1;
  RParams p{};
  p.head_dim = head_dim; p.rope_cols = rope_cols; p.t_len = t_len;
  p.cos_t = static_cast<const float*>(cos_t); p.sin_t = static_cast<const float*>(sin_t);
  return f32w ? rows_impl<true, false, ROWS_ROPE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, 16, status, st)
              : rows_impl<false, false, ROWS_ROPE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, g, status, st);
}

// D[M, N] = A[M, K] W[N, K]^T (w_mn: W is stored [K, N]) with W in fp32, rounded to the dtype of A on the way.
extern "C" int nnb_gemm_rows_f32w(const void* A, const void* W, void* D, int M, int N, int K, long long lda, long long ldw, long long ldd, int w_mn, int dtype, void* status,
                                  cudaStream_t st) {
  if (!operands_ok(M, N, K, dtype)) return -1;
  RParams p{};
  if (w_mn) return rows_impl<true, true, ROWS_NONE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, 32, status, st);
  return rows_impl<true, false, ROWS_NONE>(A, W, D, M, N, K, lda, ldw, ldd, dtype, p, 16, status, st);
}

// act[M, F] = silu(A W[0:F]^T) * (A W[F:2F]^T) with W in fp32, both products rounded to the 16-bit type first.
extern "C" int nnb_gemm_rows_f32w_swiglu(const void* A, const void* W, void* act, int M, int F, int K, long long lda, long long ldw, long long ldact, int dtype, void* status,
                                         cudaStream_t st) {
  if (!operands_ok(M, F, K, dtype)) return -1;
  RParams p{};
  const int g = F % 32 == 0 && (long long)((M + BM - 1) / BM) * (F / 16) > nnb_num_sms() ? 32 : 16;
  return rows_impl<true, false, ROWS_SWIGLU>(A, W, act, M, F, K, lda, ldw, ldact, dtype, p, g, status, st);
}

// MXFP8 (OCP microscaling: 1 x 32 blocks along the contraction dimension, e4m3 elements, e8m0 scales)
// quantisation kernels.
//   nnb_mxfp8_quantize     x [M, K] (bf16)  ->  q [M, K] (e4m3 bytes) + scales [M, K/32] (e8m0 bytes)
//   nnb_mxfp8_fake_quant   x -> dequant(quant(x)) in bf16: the exact values an MXFP8 GEMM would multiply
// One warp per 32-element block row segment group: a lane owns 8 consecutive elements, four lanes share a
// block; amax by shuffles; scale = 2^(floor(log2(amax)) - 8) so the block maximum lands in [256, 448],
// the top binade of e4m3 (max 448). This is the quantiser the reference delegates to Transformer
// Engine's recipes (nanonemo/te/__init__.py:28-39, per-tensor scaling there; block scaling here).
#include <cuda_fp8.h>

#include "common.cuh"

namespace {

__device__ __forceinline__ float block_scale_e8m0(float amax, uint8_t* biased) {
  // e8m0: value 2^(b - 127); pick b so that amax / 2^(b-127) <= 448 with the exponent of amax mapped to 8
  int e = amax > 0.f ? ((__float_as_int(amax) >> 23) & 0xff) - 127 : -127;  // floor(log2(amax)) for normals
  int b = e - 8 + 127;
  b = b < 0 ? 0 : (b > 254 ? 254 : b);
  *biased = (uint8_t)b;
  return __int_as_float(b << 23);  // 2^(b-127) (b = 0 gives 0 -> treated as the smallest scale below)
}

template <bool kFake>
__global__ void mxfp8_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ scales,
                             __nv_bfloat16* __restrict__ y, long long M, int K, long long ldx, long long ldo) {
  const int vec_per_row = K >> 3;
  const long long total = M * vec_per_row;
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool live = idx < total;
  const long long m = live ? idx / vec_per_row : 0;
  const int j = live ? (int)(idx - m * vec_per_row) * 8 : 0;
  float v[8];
  if (live) Chunk8<__nv_bfloat16>::load(x + m * ldx + j, v);
  else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
  }
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));  // 4 lanes x 8 elements = one 32-element block
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  uint8_t sb;
  float scale = block_scale_e8m0(amax, &sb);
  if (scale == 0.f) scale = __int_as_float(1 << 23);
  const float inv = 1.f / scale;
  if (!live) return;
  uint8_t bytes[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) bytes[i] = (uint8_t)__nv_cvt_float_to_fp8(v[i] * inv, __NV_SATFINITE, __NV_E4M3);
  if (kFake) {
    float o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half_raw h = __nv_cvt_fp8_to_halfraw(bytes[i], __NV_E4M3);
      o[i] = __half2float(*reinterpret_cast<const __half*>(&h)) * scale;
    }
    Chunk8<__nv_bfloat16>::store(y + m * ldo + j, o);
  } else {
    *reinterpret_cast<uint2*>(q + m * ldo + j) = *reinterpret_cast<uint2*>(bytes);
    if ((j & 31) == 0) scales[m * (K >> 5) + (j >> 5)] = sb;
  }
}

// Tile quantiser for the tensor-core path. A block owns a 128 x 128 tile of x [R, C] (bf16) held in shared memory and writes
//   ROW: q  [R, C] e4m3, blocks of 32 along C, scales chunked for a GEMM that contracts over C;
//   COL: qt [C, R] e4m3 (the transpose), blocks of 32 along R, scales chunked for a GEMM that contracts over R
// from ONE read of x. Scale layout ("chunked"): for a matrix of `rows` x `k`, chunk [row / 128][k / 128] of 512 bytes, the four
// scales of (row, 128-wide k chunk) form one 32-bit word at byte (row % 32) * 16 + ((row % 128) / 32) * 4 — the order in which
// tcgen05.cp (32x128b, warpx4) expects to find them in shared memory.
constexpr int kTile = 128, kTilePad = 8, kBlockSkew = 16;  // (the same columns of four blocks of 32 rows are in different banks)

__device__ __forceinline__ uint32_t quant4(const float* v, float inv) {
  const uint16_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[0] * inv, v[1] * inv), __NV_SATFINITE, __NV_E4M3);
  const uint16_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[2] * inv, v[3] * inv), __NV_SATFINITE, __NV_E4M3);
  return (uint32_t)lo | ((uint32_t)hi << 16);
}

// 32 bytes, in one store where the address allows it
__device__ __forceinline__ void store_sector(uint8_t* out, const uint32_t (&w)[8]) {
  if (reinterpret_cast<uintptr_t>(out) % 32 == 0) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
  } else {
    reinterpret_cast<uint4*>(out)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(out)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// N elements of one scale block, given its largest magnitude: the biased exponent goes to *biased, the bytes to w.
template <int N>
__device__ __forceinline__ void quant_block(const float (&v)[N], float amax, uint8_t* biased, uint32_t (&w)[N / 4]) {
  float scale = block_scale_e8m0(amax, biased);
  if (scale == 0.f) scale = __int_as_float(1 << 23);
  const float inv = 1.f / scale;
#pragma unroll
  for (int k = 0; k < N / 4; ++k) w[k] = quant4(v + 4 * k, inv);
}

// Both directions work on the tile with all 256 threads. Rows: eight lanes hold a row's 128 columns as they come from memory, 16 each
// (two lanes share a scale), and store them as one 128-byte line. Columns: a thread takes 32 rows of two neighbouring columns out of
// shared memory (four-byte accesses, no bank conflicts) and writes each as one 32-byte store; the four lanes that have the same columns
// fill a 128-byte line. When a warp wrote 64 different lines in halves of sectors, and two blocks were on an SM instead of three, bf16 8192 x 4096
// took 32.6 us, now 29.1 (the bytes alone 21); 2048 x 4096 9.1 and 8.5, 1024 x 4096 6.5 and 5.95, 1024 x 2048 3.1 and 2.95.
//
// SRC: what the tile's values are. MX_PLAIN: x. MX_SWIGLU: silu(gate) * up of the projection gu = gate | up [R, 2 C]. MX_SWIGLU_BWD: the gradient
// d(gate) | d(up) [R, C] of that projection (gu [R, C]) where x [R, C / 2] is the activation's; a tile is 64 columns of either half, which share the
// loads and the sigmoid. Values are rounded to bf16 first: the bytes are those of the stand-alone activation kernels (elementwise.cu)
// and then this one, whose 16-bit result, written and read back, was half of the traffic. us, two kernels / one: 8192 rows, F = 2048 30.2 / 22.3,
// backward 54.2 / 39.2; F = 5632 82 / 54, 143 / 98; 1024 rows, F = 2048 8.8 / 4.0, 9.3 / 8.7.
enum MxSource : int { MX_PLAIN = 0, MX_SWIGLU = 1, MX_SWIGLU_BWD = 2 };

__device__ __forceinline__ uint4 pack_bf16(const float (&v)[8]) {
  uint4 out;
  Chunk8<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(&out), v);
  return out;
}

template <bool ROW, bool COL, int SRC>
__global__ void __launch_bounds__(256, 3) mxfp8_tile_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ gu,
                                                                                 long long ldgu, uint8_t* __restrict__ q, long long ldq, uint8_t* __restrict__ sf,
                                                                                 uint8_t* __restrict__ qt, long long ldqt, uint8_t* __restrict__ sft, int R, int C) {
  nnb_after_previous(x, gu, q, sf, qt, sft);
  nnb_release_next();
  __shared__ __align__(16) __nv_bfloat16 tile[kTile * (kTile + kTilePad) + 3 * kBlockSkew];
  auto at = [](int r, int c) { return r * (kTile + kTilePad) + r / 32 * kBlockSkew + c; };
  constexpr bool kBwd = SRC == MX_SWIGLU_BWD;
  const int c0 = blockIdx.x * (kBwd ? kTile / 2 : kTile), r0 = blockIdx.y * kTile, F = kBwd ? C / 2 : C;
  const int seg = threadIdx.x & 7;
  uint4 raw[4][2];  // sixteen neighbouring columns, or eight of either half
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long m = r0 + k * 32 + (threadIdx.x >> 3);
    if constexpr (SRC == MX_PLAIN) {
      const uint4* src = reinterpret_cast<const uint4*>(x + m * ldx + c0 + seg * 16);
      raw[k][0] = src[0];
      raw[k][1] = src[1];
    } else if constexpr (SRC == MX_SWIGLU) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __nv_bfloat16* g = gu + m * ldgu + c0 + seg * 16 + h * 8;
        float a[8], b[8];
        Chunk8<__nv_bfloat16>::load(g, a);
        Chunk8<__nv_bfloat16>::load(g + F, b);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = a[i] / (1.f + __expf(-a[i])) * b[i];
        raw[k][h] = pack_bf16(a);
      }
    } else {
      const __nv_bfloat16* g = gu + m * ldgu + c0 + seg * 8;
      float d[8], a[8], b[8];
      Chunk8<__nv_bfloat16>::load(x + m * ldx + c0 + seg * 8, d);
      Chunk8<__nv_bfloat16>::load(g, a);
      Chunk8<__nv_bfloat16>::load(g + F, b);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float s = 1.f / (1.f + __expf(-a[i]));
        b[i] = d[i] * b[i] * s * (1.f + a[i] * (1.f - s));
        d[i] = d[i] * a[i] * s;
      }
      raw[k][0] = pack_bf16(b);
      raw[k][1] = pack_bf16(d);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = k * 32 + (threadIdx.x >> 3);
    if (COL) {
      *reinterpret_cast<uint4*>(&tile[at(r, kBwd ? seg * 8 : seg * 16)]) = raw[k][0];
      *reinterpret_cast<uint4*>(&tile[at(r, kBwd ? kTile / 2 + seg * 8 : seg * 16 + 8)]) = raw[k][1];
    }
    if (ROW) {
      float v[16], amax[2] = {0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 f = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(raw[k])[e]);
        v[2 * e] = f.x; v[2 * e + 1] = f.y;
        amax[e / 4] = fmaxf(amax[e / 4], fmaxf(fabsf(f.x), fabsf(f.y)));
      }
      uint8_t* row = q + (long long)(r0 + r) * ldq;
      const int word = (r & 31) * 16 + (r >> 5) * 4;
      if constexpr (kBwd) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          amax[h] = fmaxf(amax[h], __shfl_xor_sync(0xffffffffu, amax[h], 1));
          amax[h] = fmaxf(amax[h], __shfl_xor_sync(0xffffffffu, amax[h], 2));
          float half[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) half[e] = v[8 * h + e];
          uint32_t w[2];
          uint8_t sb;
          quant_block(half, amax[h], &sb, w);
          const int c = h * F + c0 + seg * 8;
          *reinterpret_cast<uint2*>(row + c) = make_uint2(w[0], w[1]);
          if ((seg & 3) == 0) sf[((long long)blockIdx.y * (C / kTile) + c / kTile) * 512 + word + (c % kTile) / 32] = sb;
        }
      } else {
        float m = fmaxf(amax[0], amax[1]);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        uint32_t w[4];
        uint8_t sb;
        quant_block(v, m, &sb, w);
        *reinterpret_cast<uint4*>(row + c0 + seg * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        if ((seg & 1) == 0) sf[((long long)blockIdx.y * (C / kTile) + blockIdx.x) * 512 + word + (seg >> 1)] = sb;
      }
    }
  }
  if (COL) {
    __syncthreads();
    // columns c and c + 1 of the tile = rows row and row + 1 of the transpose, block b of 32 rows
    const int c = (threadIdx.x >> 5) * 16 + (threadIdx.x & 7) * 2, b = threadIdx.x >> 3 & 3;
    const int row = kBwd && c >= kTile / 2 ? F + c0 + c - kTile / 2 : c0 + c;
    float v[2][32], amax[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&tile[at(b * 32 + i, c)]));
      v[0][i] = f.x; v[1][i] = f.y;
      amax[0] = fmaxf(amax[0], fabsf(f.x));
      amax[1] = fmaxf(amax[1], fabsf(f.y));
    }
    const long long chunk = (long long)(row / kTile) * (R / kTile) + blockIdx.y;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t w[8];
      uint8_t sb;
      quant_block(v[u], amax[u], &sb, w);
      store_sector(qt + (long long)(row + u) * ldqt + r0 + b * 32, w);
      sft[chunk * 512 + ((row + u) & 31) * 16 + ((row + u) % kTile >> 5) * 4 + b] = sb;
    }
  }
}

}  // namespace

namespace {

template <int SRC>
int quantize_tiles(const void* x, long long ldx, const void* gu, long long ldgu, void* q, long long ldq, void* sf, void* qt, long long ldqt, void* sft, int R, int C, cudaStream_t st) {
  NNB_REQUIRE(R > 0 && C > 0 && R % 128 == 0 && C % 128 == 0, "mxfp8_quantize_sw: R=%d and C=%d must be positive multiples of 128", R, C);
  NNB_REQUIRE(SRC != MX_SWIGLU_BWD || C % 256 == 0, "mxfp8_swiglu_bwd: both halves of C=%d must be multiples of 128", C);
  NNB_REQUIRE(ldx % 8 == 0 && nnb_aligned16(x) && ldgu % 8 == 0 && nnb_aligned16(gu),
              "mxfp8_quantize_sw: x must be 16-byte aligned with a row stride that is a multiple of 8");
  const bool row = q != nullptr, col = qt != nullptr;
  NNB_REQUIRE(row || col, "mxfp8_quantize_sw: nothing to do");
  NNB_REQUIRE(!row || (sf != nullptr && ldq % 16 == 0 && nnb_aligned16(q)), "mxfp8_quantize_sw: bad row-wise output");
  NNB_REQUIRE(!col || (sft != nullptr && ldqt % 16 == 0 && nnb_aligned16(qt)), "mxfp8_quantize_sw: bad transposed output");
  const dim3 grid(C / 128, R / 128);
#define NNB_MX_LAUNCH(ROW, COL) nnb_launch(mxfp8_tile_kernel<ROW, COL, SRC>, grid, 256, 0, st, (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)gu, ldgu, \
    (uint8_t*)q, ldq, (uint8_t*)sf, (uint8_t*)qt, ldqt, (uint8_t*)sft, R, C)
  if (row && col) NNB_MX_LAUNCH(true, true);
  else if (row) NNB_MX_LAUNCH(true, false);
  else NNB_MX_LAUNCH(false, true);
#undef NNB_MX_LAUNCH
  NNB_LAUNCH_OK("mxfp8_quantize_sw");
  return 0;
}

}  // namespace

// x [R, C] bf16 (row stride ldx elements) -> any of
//   q [R, C] e4m3 (row stride ldq bytes) + sf (chunked scales, R / 128 x C / 128 chunks of 512 bytes), blocks along C;
//   qt [C, R] e4m3 (row stride ldqt bytes) + sft (C / 128 x R / 128 chunks), blocks along R.
// Pass null for the pair that is not wanted. R and C must be multiples of 128.
extern "C" int nnb_mxfp8_quantize_sw(const void* x, long long ldx, void* q, long long ldq, void* sf, void* qt, long long ldqt,
                                     void* sft, int R, int C, cudaStream_t st) {
  return quantize_tiles<MX_PLAIN>(x, ldx, x, ldx, q, ldq, sf, qt, ldqt, sft, R, C, st);
}

// The same of silu(gate) * up, gu = gate | up [R, 2 F].
extern "C" int nnb_mxfp8_swiglu(const void* gu, long long ldgu, void* q, long long ldq, void* sf, void* qt, long long ldqt, void* sft, int R, int F, cudaStream_t st) {
  return quantize_tiles<MX_SWIGLU>(gu, ldgu, gu, ldgu, q, ldq, sf, qt, ldqt, sft, R, F, st);
}

// The same of the gradient of gu [R, 2 F] for the gradient dact [R, F] of that activation.
extern "C" int nnb_mxfp8_swiglu_bwd(const void* dact, long long ldd, const void* gu, long long ldgu, void* q, long long ldq, void* sf, void* qt, long long ldqt, void* sft,
                                    int R, int F, cudaStream_t st) {
  return quantize_tiles<MX_SWIGLU_BWD>(dact, ldd, gu, ldgu, q, ldq, sf, qt, ldqt, sft, R, 2 * F, st);
}

extern "C" int nnb_mxfp8_fake_quant(const void* x, void* y, long long M, int K, long long ldx, long long ldy, cudaStream_t st) {
  NNB_REQUIRE(K % 32 == 0 && ldx % 8 == 0 && ldy % 8 == 0, "mxfp8: K=%d must be a multiple of 32 and strides multiples of 8", K);
  if (M == 0) return 0;
  const long long total = M * (K / 8);
  mxfp8_kernel<true><<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)x, nullptr, nullptr, (__nv_bfloat16*)y, M, K, ldx, ldy);
  NNB_LAUNCH_OK("mxfp8_fake_quant");
  return 0;
}

extern "C" int nnb_mxfp8_quantize(const void* x, void* q, void* scales, long long M, int K, long long ldx, long long ldq, cudaStream_t st) {
  NNB_REQUIRE(K % 32 == 0 && ldx % 8 == 0 && ldq % 8 == 0, "mxfp8: K=%d must be a multiple of 32 and strides multiples of 8", K);
  if (M == 0) return 0;
  const long long total = M * (K / 8);
  mxfp8_kernel<false><<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)x, (uint8_t*)q, (uint8_t*)scales, nullptr, M, K, ldx, ldq);
  NNB_LAUNCH_OK("mxfp8_quantize");
  return 0;
}

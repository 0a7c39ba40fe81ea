// Host entry of the CTA-pair GEMM (gemm2.cu); called by the dispatcher in gemm.cu.
#pragma once
#include <cuda_runtime.h>

// Work fused into the epilogue while a tile leaves tensor memory (see gemm2.cu).
enum NnbGemm2Epilogue : int { EPI_NONE = 0, EPI_SWIGLU = 1, EPI_ROPE = 2, EPI_CE_STATS = 3, EPI_SWIGLU_BWD = 4, EPI_CE_LOSS = 5, EPI_SWIGLU_ACT = 6,
                              EPI_CHAINED = 7 /* never asked for: see nnb_plan_k */ };

struct NnbGemm2Args {
  const void *A, *B;
  void* D;
  int M, N, K;
  long long lda, ldb, ldd;  // row strides in elements of the stored matrices
  int a_mn, b_mn;           // operand majors (0 = K-major, 1 = MN-major)
  int dtype;                // NNB_BF16 / NNB_F16
  int out_f32, accumulate, k_splits, max_ctas;
  void* status;             // device int[4] or null
  int epilogue = EPI_NONE;
  // EPI_SWIGLU: B = gate||up weight [2 F, K] (N = 2 F), D = projection [M, 2 F], E = act [M, F] with row stride lde
  void* E = nullptr;
  long long lde = 0;
  // EPI_SWIGLU_ACT: the same without the projection (D is not written): act alone, for a forward pass without gradients
  // EPI_ROPE: rotate-half on columns [0, rope_cols) in heads of head_dim columns; row m uses table row m % t_len of the
  // fp32 tables [t_len, head_dim / 2]
  const void *cos_t = nullptr, *sin_t = nullptr;
  int t_len = 0, rope_cols = 0, head_dim = 0;
  // EPI_SWIGLU_BWD: the product [M, N = F] is the gradient of act = silu(gate) * up; E = the saved projection gate||up
  // [M, 2 F] (row stride lde), D = its gradient [M, 2 F] (row stride ldd); the product itself is never stored
  // EPI_CE_STATS: fp32 [M, 2 ceil(N / 256), 2] receiving (max, sum of exp(x - max)) of every row's logits in two parts per
  // 256-column tile (the tile's even and odd 64-column chunks); a part without columns holds (-inf, 0)
  void* stats = nullptr;
  // EPI_CE_LOSS: the same statistics without the logits (D is not written); target_logit[m] fp32 receives the logit of column
  // targets[m] (int64) and is left alone where that column does not exist
  const void* targets = nullptr;
  void* target_logit = nullptr;
  int chain = 0;  // EPI_CHAINED: k-blocks per accumulator
};

// Returns 0 on success, 1 when the shape is not served by the pair kernel (caller falls back), < 0 on error.
int nnb_gemm2_launch(const NnbGemm2Args& a, cudaStream_t st);

// The kernel for few rows (gemm_rows.cu): columns of its tile / 2 (32 or 64) for a product with a 16-bit output that it serves faster than the
// persistent kernels, 0 otherwise. Its tiles are narrow and short-lived: a set-up of 2.3 us against 4 to 5, and the SMs that a few wide tiles
// would leave idle; with more tiles than SMs it is bound by the bytes an SM takes in. us in a row of products with 24 weights, taken with four
// epilogue warps (the eight it has are 0.3 us faster; pair kernel,
// single-CTA kernel below 256 rows / 64-wide / 128-wide tiles): 201 x 768 x 768 6.5 / 4.5 / 6.2, 512 x 768 x 2048 13.9 / 8.0 / 10.9, 1024
// x 768 x 4096 23.0 / 14.4 / 20.1, 512 x 2048 x 11264 54.9 / 39.3 / 56.7, 777 x 1280 x 768 8.1 / 4.9 / 6.4; more 64-wide tiles than SMs:
// 1024 x 1280 x 768 8.2 / 6.7 / 6.6, 2048 x 768 x 2048 14.3 / 13.9 / 12.3, 512 x 4096 x 768 8.7 / 7.4 / 7.0, 2048 x 768 x 4096 23.2 / 26.1 /
// 22.3, 1024 x 2048 x 5632 30.7 / 39.8 / 33.0; more 128-wide ones: 777 x 3072 x 2048 15.6 / 26.3 / 17.2, 4096 x 768 x 2048 15.3 / 27.1 / 19.0.
inline int nnb_rows_tile(long long M, long long N, long long K, int sms) {
  const long long m = (M + 127) / 128;
  if (m * ((N + 63) / 64) <= sms) return 32;
  if (m * ((N + 127) / 128) <= sms && K <= 4096) return 64;
  return 0;
}
extern "C" int nnb_gemm_rows(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, void*, cudaStream_t);
extern "C" int nnb_gemm_rows_rope(const void*, const void*, void*, const void*, const void*, int, int, int, long long, long long, long long, int, int, int, int, int, int, void*, cudaStream_t);

// K splits that even out the last wave of `tiles` tiles on `workers` persistent CTAs (or pairs), whatever traffic they add. This is how
// long an accumulator's chain may get: with it as the limit a product is as exact as if it were cut into these splits.
inline int nnb_even_k_splits(long long tiles, int workers, int kblocks) {
  const int s_max = kblocks / 4 < 1 ? 1 : (kblocks / 4 > 32 ? 32 : kblocks / 4);
  int best_s = 1;
  double best = 1e30;
  for (int s = 1; s <= s_max; ++s) {
    const double cost = (double)((tiles * s + workers - 1) / workers) / s + 0.002 * s;
    if (cost < best - 1e-9) { best = cost; best_s = s; }
  }
  return best_s;
}

// How the K loop of an fp32-output product is cut: into `splits` that are reduce-added to memory, each of them into chains of `chain`
// k-blocks that are added up in registers (0: the whole split is one chain). For kernels that hold a thread's sums in registers.
// Splitting evens out the last wave (ceil(tiles s / workers) / s of a whole tile's K loop) but adds the output's bytes once more per
// split, and a cleared output where the product does not accumulate. Measured: a k-block of a tile takes `us_per_kblock`, a
// megabyte reduce-added about 0.1 us. Of counts within 1 % of the least cost the smallest is taken: they measured up to 13 % faster
// and never more than 1 % slower (2048 x 2048 x 16384: 1 split 100 us, 8 splits 114; 1280 x 768 x 32768: 9 splits 61, 14 64).
// Fewer splits alone would lengthen the accumulators' chains, and the error grows with them (see EPI_CHAINED): the chains stay
// as short as the even splits would make them. bf16, accumulating, us and error off 64 bits, even splits / fewer splits without
// chains / as here: 11264 x 2048 x 8192 386 us 6.0e-7 / 245 us 9.1e-6 / 259 us 6.0e-7; 2048 x 2048 x 8192 81 us 1.0e-6 / 63 us 9.1e-6 /
// 62 us 1.0e-6; 3072 x 2048 x 4096 77 us 4.1e-7 / 48 us 1.4e-6 / 55 us 4.0e-7; 50304 x 2048 x 1024 360 us 3.2e-7 / 204 us 9.9e-7 /
// 259 us 3.2e-7; MXFP8 11264 x 2048 x 8192 302 us 7.8e-8 / 222 us 4.7e-7 / 228 us 7.9e-8.
inline void nnb_plan_k(long long tiles, int workers, int kblocks, double us_per_kblock, double out_bytes, bool accumulate, int& splits,
                       int& chain) {
  const double us_tile = kblocks * us_per_kblock, us_out = out_bytes * 1e-7;
  const int s_max = kblocks / 4 < 1 ? 1 : (kblocks / 4 > 32 ? 32 : kblocks / 4);
  auto cost = [&](int s) {
    return (double)((tiles * s + workers - 1) / workers) / s * us_tile + s * us_out + (s > 1 && !accumulate ? us_out + 2.0 : 0.0);
  };
  double best = 1e30;
  for (int s = 1; s <= s_max; ++s) best = cost(s) < best ? cost(s) : best;
  splits = 1;
  while (cost(splits) > 1.01 * best) ++splits;
  const int even = nnb_even_k_splits(tiles, workers, kblocks);
  const int limit = (kblocks + even - 1) / even;
  chain = limit < (kblocks + splits - 1) / splits ? limit : 0;
}

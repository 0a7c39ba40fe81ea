// Host entry of the CTA-pair GEMM (gemm2.cu); called by the dispatcher in gemm.cu.
#pragma once
#include <stdint.h>

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
// would leave idle; with more tiles than SMs it is bound by the bytes an SM takes in. us in a row of products with 24 weights, pair kernel (single-CTA
// kernel below 256 rows) / 64-wide / 128-wide tiles: 201 x 768 x 768 6.4 / 4.25 / 5.65, 512 x 768 x 2048 13.9 / 7.8 / 10.5, 1024 x 768 x 4096 23.0 / 14.3 / 20.1,
// 512 x 2048 x 11264 54.5 / 37.7 / 56.7, 777 x 1280 x 768 8.2 / 4.8 / 5.9; more 64-wide tiles than SMs: 1024 x 1280 x 768 8.1 / 6.8 / 6.2, 2048 x 768 x 2048
// 14.4 / 13.7 / 11.9, 512 x 4096 x 768 8.75 / 7.6 / 6.6, 2048 x 768 x 4096 23.4 / 25.9 / 22.0, UNSERVED. Weights stored [K, N] (input gradients) within 0.3 us of these.
// Three limits to that. `lines`: rows of both operands start at multiples of 128 bytes; others cost every row of a box two lines, which tiles with a long K
// loop do not make good: 555 x 2896 x 2424 19.3 / 28.9 / 21.6 (512 x 2944 x 2432 16.3 / 16.2 / 13.7), 63 x 680 x 8920 46.8 / 49.9 / -; 2304 x 560 x 896 8.8 / 7.6 / 7.2.
// Very wide weights, where 128-wide tiles lose: 16384 x 2048 with 32 to 100 rows 14.9 / - / 14.2, 7488 x 3008 17.1 / - / 17.7, 11264 x 4096 22.0 / - / 22.5, 18944 x 4096 29.7 / - / 32.6.
// Fewest rows: an A of less than 128 KB is the same few lines of L2 for every CTA, and the more of them read it the longer that takes. 32 CTAs and more,
// 1 to 12 rows: 2048 x 4096 19.9 / 18.2 / 20.1, 2048 x 5632 25.3 / 26.9 / 26.5, 3072 x 5632 25.8 / 29.6 / 27.2; 64 and more, where 128-wide tiles are half as many:
// 4096 x 1024 7.8 / 6.4 / 6.1, 6144 x 1024 7.9 / 9.5 / 6.2, 9472 x 768 7.5 / 7.7 / 6.1, 4096 x 4096 20.1 / 24.8 / 20.4, 4096 x 5632 25.9 / 33.6 / 30.6,
// 8192 x 2048 (stored [K, N]) 13.3 / 17.6 / 14.6; not on lines, 1904 x 3152 16.0 / 17.1 / 18.0, 1536 x 3152 15.9 / 12.0 / 17.9, 5048 x 792 7.5 / 8.9 / -. The same with 16 or 32 rows, A of
// 128 KB or more: 4096 x 4096 20.2 / 14.7 / 20.4, 3072 x 5632 25.8 / 18.8 / 27.3.
inline int nnb_rows_tile(long long M, long long N, long long K, bool lines, int sms) {
  const long long m = (M + 127) / 128, weights = N * K;
  const bool narrow = m * ((N + 63) / 64) <= sms && (lines || K <= 4096), wide = m * ((N + 127) / 128) <= sms && K <= (lines ? 4096 : 1024);
  if (M * K < 1 << 16 && N >= 1600 && (weights > 1 << 22 || (N >= 4096 && !lines))) {
    if (N < 4096) return narrow && lines && weights <= 1 << 23 ? 32 : 0;
    return wide && K <= 1536 && weights < 1 << 24 ? 64 : 0;
  }
  return narrow ? 32 : wide && weights <= (K <= 2560 ? 1 << 25 : 1 << 24) ? 64 : 0;
}
// Row strides in elements of 16 bits
inline bool nnb_rows_on_lines(const void* a, const void* w, long long lda, long long ldw) {
  return lda % 64 == 0 && ldw % 64 == 0 && reinterpret_cast<uintptr_t>(a) % 128 == 0 && reinterpret_cast<uintptr_t>(w) % 128 == 0;
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

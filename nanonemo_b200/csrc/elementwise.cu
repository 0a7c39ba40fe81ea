// HBM-bandwidth-bound operators of the transformer block, written for B200:
//   fused residual-add + RMSNorm forward/backward, fused Q/K RoPE on the packed QKV projection,
//   SwiGLU forward/backward, embedding gather / scatter-add, the toolchain warm-up add.
// Every kernel moves 16 bytes per thread per access, keeps its row in registers (one warp per row
// for the norms) and reads each input exactly once; the roofline for all of them is the HBM3e copy
// bandwidth. Contracts follow the reference operators (nanonemo/kernels/cuda/rmsnorm.cu:64-167,
// nanonemo/kernels/triton/{rope,swiglu}.py) with bf16 added (the reference kernels reject it).
#include <initializer_list>

#include "common.cuh"

// ============================================================================ add + RMSNorm
// Sum over the WPR warps that share a row (WPR 1 or 2; `pair` numbers the row's warps in the block). `slot` alternates from row to
// row, so that one barrier per row is enough. Every lane gets the sum, added in the same order.
template <int WPR>
__device__ __forceinline__ float row_sum(float v, float (*s_part)[2][2], int pair, int slot) {
  v = warp_sum(v);
  if constexpr (WPR == 1) return v;
  if ((threadIdx.x & 31) == 0) s_part[pair][slot][(threadIdx.x >> 5) & 1] = v;
  asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
  return s_part[pair][slot][0] + s_part[pair][slot][1];
}

// y = rmsnorm(h) * w,  h = round_to_TX(x + delta);  rstd saved for backward. WPR warps per row (two for rows wider than 1024, so
// that a lane never holds more than four chunks); lane l of them owns 8-element chunks l, l + 32 WPR, ...; MAXC chunks per lane.
// HBM-bound. M = 32768, N = 2048, fp32 residual, bf16 delta and y, cold L2: 129 us with two warps a row, 158 with one
// (floor 123); 8192 rows 41 and 49 us. Whole sectors a lane (WIDE) count where the rows come out of L2: 4096 x 768 7.7 -> 6.3 us, 8192 x 768
// 13.2 -> 11.5, 32768 x 768 46.5 (the floor) both ways.
template <typename TX, typename TD, typename TY, int MAXC, int WPR, bool WIDE>
__global__ void __launch_bounds__(256) add_rmsnorm_fwd_kernel(const TX* __restrict__ x, const TD* __restrict__ delta,
                                                              const float* __restrict__ w, TY* __restrict__ y,
                                                              TX* __restrict__ h, float* __restrict__ rstd, int M,
                                                              int N, float eps) {
  nnb_after_previous(x, delta, w, y, h, rstd);
  nnb_release_next();
  __shared__ float s_part[8 / WPR][2][2];
  constexpr int kLanes = 32 * WPR;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes, lane = threadIdx.x % kLanes;
  if (row >= M) return;  // (all warps of a row together)
  const int nchunks = N >> 3;
  const size_t base = (size_t)row * N;
  float v[MAXC][8];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int ch = lane + kLanes * c;
    if (ch < nchunks) {
      GlobalChunk8<TX, WIDE>::load(x + base + ch * 8, v[c]);
      if (delta != nullptr) {
        float d[8];
        Chunk8<TD>::load(delta + base + ch * 8, d);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[c][i] = to_f32(from_f32<TX>(v[c][i] + d[i]));
        GlobalChunk8<TX, WIDE>::store(h + base + ch * 8, v[c]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[c][i] * v[c][i];
    }
  }
  ss = row_sum<WPR>(ss, s_part, threadIdx.x / kLanes, 0);
  const float r = rsqrtf(ss / (float)N + eps);
  if (lane == 0) rstd[row] = r;
#pragma unroll
  for (int c = 0; c < MAXC; ++c) {
    const int ch = lane + kLanes * c;
    if (ch < nchunks) {
      float g[8];
      Chunk8<float>::load(w + ch * 8, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) g[i] = v[c][i] * r * g[i];
      Chunk8<TY>::store(y + base + ch * 8, g);
    }
  }
}

// n = h*rstd, dn = dy*w, dh = rstd*(dn - n*mean(dn*n)) + dres; dx = ddelta = dh; dw = sum_rows dy*n.
// Persistent: each warp strides over rows; the norm weight and a per-warp dw accumulator live in shared memory (so the
// register file only holds one row), warps of a block are then summed and the block writes one partial row of dw, reduced in
// index order by dw_reduce_kernel. Every load of a row (h, dy AND the incoming residual gradient) is issued before the first
// use, so a warp has its whole ~8 KB in flight at once instead of paying the memory latency twice per row, and blocks are
// 128 threads with at most 128 registers so that four of them (16 warps) share an SM. Rows wider than 1024 take two warps: with one, a
// row's loads did not fit the registers, the residual gradient was fetched late and only half the warps fitted. With the reduction
// of dw, cold L2, fp32 residual, bf16 dy and ddelta: M = 32768, N = 2048 278 -> 198 us (floor 164), 8192 rows 99 -> 73 us. With
// whole sectors a lane (WIDE) 4096 x 768 14.3 -> 13.7 us, 32768 x 768 70.8 -> 69.6, 8192 x 2048 58.5 -> 56.8.
template <typename TX, typename TD, typename TY, int MAXC, int WPR, bool WIDE>
__global__ void __launch_bounds__(128, 4) add_rmsnorm_bwd_kernel(const TY* __restrict__ dy, const TX* __restrict__ h,
                                                                 const float* __restrict__ rstd,
                                                                 const float* __restrict__ w, const TX* __restrict__ dres,
                                                                 TX* __restrict__ dx, TD* __restrict__ ddelta,
                                                                 float* __restrict__ dw_partial, int M, int N) {
  extern __shared__ float s_mem[];  // [N] weight, then [rows in flight][N] accumulators
  __shared__ float s_part[4 / WPR][2][2];
  constexpr int kLanes = 32 * WPR;
  const int lane = threadIdx.x % kLanes, warp_in_block = threadIdx.x / kLanes, warps_per_block = blockDim.x / kLanes;  // (groups of WPR warps)
  int slot = 0;
  const int nchunks = N >> 3;
  float* s_w = s_mem;
  float* s_acc = s_mem + N + (size_t)warp_in_block * N;
  for (int i = threadIdx.x; i < N * warps_per_block; i += blockDim.x) s_mem[N + i] = 0.f;
  nnb_after_previous(dy, h, rstd, w, dres, dx, ddelta, dw_partial);
  for (int i = threadIdx.x; i < N; i += blockDim.x) s_w[i] = w[i];
  __syncthreads();
  const float inv_n = 1.f / (float)N;
  for (int row = blockIdx.x * warps_per_block + warp_in_block; row < M; row += gridDim.x * warps_per_block) {
    const size_t base = (size_t)row * N;
    float n_[MAXC][8], dn[MAXC][8], res[MAXC][8];
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
      const int ch = lane + kLanes * c;
      if (ch < nchunks) {
        GlobalChunk8<TX, WIDE>::load(h + base + ch * 8, n_[c]);
        Chunk8<TY>::load(dy + base + ch * 8, dn[c]);
        if (dres != nullptr) GlobalChunk8<TX, WIDE>::load(dres + base + ch * 8, res[c]);
      }
    }
    const float r = rstd[row];
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
      const int ch = lane + kLanes * c;
      if (ch < nchunks) {
        float g[8], a[8];
        Chunk8<float>::load(s_w + ch * 8, g);
        Chunk8<float>::load(s_acc + ch * 8, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          n_[c][i] *= r;
          a[i] += dn[c][i] * n_[c][i];
          dn[c][i] *= g[i];
          dot += dn[c][i] * n_[c][i];
        }
        Chunk8<float>::store(s_acc + ch * 8, a);
      }
    }
    dot = row_sum<WPR>(dot, s_part, warp_in_block, slot) * inv_n;
    slot ^= 1;
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
      const int ch = lane + kLanes * c;
      if (ch < nchunks) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = r * (dn[c][i] - n_[c][i] * dot) + (dres != nullptr ? res[c][i] : 0.f);
        GlobalChunk8<TX, WIDE>::store(dx + base + ch * 8, o);
        if (ddelta != nullptr) Chunk8<TD>::store(ddelta + base + ch * 8, o);
      }
    }
  }
  nnb_release_next();
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    float s = 0.f;
    for (int wv = 0; wv < warps_per_block; ++wv) s += s_mem[N + (size_t)wv * N + i];
    dw_partial[(size_t)blockIdx.x * N + i] = s;
  }
}

// dw[c] (+)= sum over partial rows; 32 columns per block, 128 rows at a time (a warp: 4 rows x 32 columns in 16-byte loads), in a fixed
// order within a thread and between them: the result does not depend on scheduling. Bound by latency (592 rows of 768 are 1.8 MB in L2,
// read by 24 blocks): with 8 rows at a time and 4-byte loads, 74 dependent rounds, it took 7.9 us after the kernel before it, now 5.2.
__global__ void __launch_bounds__(1024) dw_reduce_kernel(const float* __restrict__ partial, float* __restrict__ dw, int rows,
                                                         int N, int accumulate) {
  nnb_after_previous(partial, dw);
  nnb_release_next();
  __shared__ float s_red[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + (lane & 7) * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < N) {
#pragma unroll 5
    for (int r = warp * 4 + (lane >> 3); r < rows; r += 128) {
      const float4 v = *reinterpret_cast<const float4*>(partial + (size_t)r * N + col);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
    s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
  }
  if (lane < 8) {
    float* d = &s_red[warp][lane * 4];
    d[0] = s.x; d[1] = s.y; d[2] = s.z; d[3] = s.w;
  }
  __syncthreads();
  const float t = warp_sum(s_red[lane][warp]);  // a warp per column
  const int c = blockIdx.x * 32 + warp;
  if (lane == 0 && c < N) dw[c] = accumulate ? dw[c] + t : t;
}

// Supported dtype triples (residual TX, delta TD, output TY): the compute dtype C for delta and y,
// and the residual stream either fp32 or C.
#define NNB_RMS_COMBOS(X)                                   \
  X(NNB_F32, NNB_F32, NNB_F32, float, float, float)         \
  X(NNB_F32, NNB_BF16, NNB_BF16, float, __nv_bfloat16, __nv_bfloat16) \
  X(NNB_BF16, NNB_BF16, NNB_BF16, __nv_bfloat16, __nv_bfloat16, __nv_bfloat16) \
  X(NNB_F32, NNB_F16, NNB_F16, float, __half, __half)       \
  X(NNB_F16, NNB_F16, NNB_F16, __half, __half, __half)

// fp32 rows whose 8-element chunks start at multiples of 32 bytes (the length of a row is a multiple of eight)
static bool wide_rows(std::initializer_list<const void*> rows) {
  for (const void* p : rows)
    if (reinterpret_cast<uintptr_t>(p) % 32) return false;
  return true;
}

template <typename TX, typename TD, typename TY>
static void rmsnorm_fwd_t(const void* x, const void* delta, const float* w, void* y, void* h, float* rstd, int M, int N,
                          float eps, cudaStream_t st) {
#define NNB_RMS_FWD(MAXC, WPR, WIDE) \
  nnb_launch(add_rmsnorm_fwd_kernel<TX, TD, TY, MAXC, WPR, WIDE>, (M * WPR + 7) / 8, 256, 0, st, (const TX*)x, (const TD*)delta, w, (TY*)y, (TX*)h, rstd, M, N, eps)
  if constexpr (sizeof(TX) == 4) {
    if (wide_rows({x, delta != nullptr ? h : x})) {
      if (N <= 1024) NNB_RMS_FWD(4, 1, true);
      else NNB_RMS_FWD(4, 2, true);
      return;
    }
  }
  if (N <= 1024) NNB_RMS_FWD(4, 1, false);
  else NNB_RMS_FWD(4, 2, false);
#undef NNB_RMS_FWD
}

// x: [M,N] residual dtype; delta: [M,N] or null; w fp32 [N]; y: [M,N] y_dtype; h: [M,N] residual dtype
// (written only when delta != null); rstd fp32 [M].
extern "C" int nnb_add_rmsnorm_fwd(const void* x, const void* delta, const void* w, void* y, void* h, void* rstd,
                                   int M, int N, float eps, int x_dtype, int delta_dtype, int y_dtype,
                                   cudaStream_t st) {
  NNB_REQUIRE(N % 8 == 0 && N <= 2048 && N > 0, "add_rmsnorm: N=%d must be a multiple of 8 and <= 2048", N);
  NNB_REQUIRE(M > 0, "add_rmsnorm: empty input");
  NNB_REQUIRE(nnb_aligned16(x) && nnb_aligned16(y) && nnb_aligned16(w) && (!delta || (nnb_aligned16(delta) && nnb_aligned16(h))),
              "add_rmsnorm: pointers must be 16-byte aligned");
  bool done = false;
#define X(cx, cd, cy, TX, TD, TY)                                                              \
  if (!done && x_dtype == cx && delta_dtype == cd && y_dtype == cy) {                           \
    rmsnorm_fwd_t<TX, TD, TY>(x, delta, (const float*)w, y, h, (float*)rstd, M, N, eps, st);    \
    done = true;                                                                                \
  }
  NNB_RMS_COMBOS(X)
#undef X
  NNB_REQUIRE(done, "add_rmsnorm: unsupported dtype combination (x=%d, delta=%d, y=%d)", x_dtype, delta_dtype, y_dtype);
  NNB_LAUNCH_OK("add_rmsnorm_fwd");
  return 0;
}

extern "C" int nnb_rmsnorm_bwd_blocks() { return 4 * nnb_num_sms(); }  // four 128-thread blocks per SM, persistent

template <typename TX, typename TD, typename TY>
static int rmsnorm_bwd_t(const void* dy, const void* h, const float* rstd, const float* w, const void* dres, void* dx,
                         void* ddelta, float* partial, int blocks, int M, int N, cudaStream_t st) {
#define NNB_RMS_BWD(MAXC, WPR, WIDE)                                                                              \
  {                                                                                                               \
    const size_t smem = (size_t)N * (1 + 4 / WPR) * sizeof(float); /* the weight, and an accumulator per row in flight */ \
    auto k = add_rmsnorm_bwd_kernel<TX, TD, TY, MAXC, WPR, WIDE>;                                                 \
    if (smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -3; \
    nnb_launch(k, blocks, 128, smem, st, (const TY*)dy, (const TX*)h, rstd, w, (const TX*)dres, (TX*)dx, (TD*)ddelta, partial, M, N); \
  }
  if constexpr (sizeof(TX) == 4) {
    if (wide_rows({h, dx, dres})) {
      if (N <= 768) NNB_RMS_BWD(3, 1, true)   // one row fits 3 chunks per lane: fewer registers, more resident warps
      else if (N <= 1024) NNB_RMS_BWD(4, 1, true)
      else NNB_RMS_BWD(4, 2, true)
      return 0;
    }
  }
  if (N <= 768) NNB_RMS_BWD(3, 1, false)
  else if (N <= 1024) NNB_RMS_BWD(4, 1, false)
  else NNB_RMS_BWD(4, 2, false)
#undef NNB_RMS_BWD
  return 0;
}

// dw_partial: scratch fp32 [nnb_rmsnorm_bwd_blocks(), N]; dw fp32 [N] (+= when accumulate).
extern "C" int nnb_add_rmsnorm_bwd(const void* dy, const void* h, const void* rstd, const void* w, const void* dres,
                                   void* dx, void* ddelta, void* dw, void* dw_partial, int M, int N, int x_dtype,
                                   int delta_dtype, int y_dtype, int accumulate_dw, cudaStream_t st) {
  NNB_REQUIRE(N % 8 == 0 && N <= 2048 && N > 0, "add_rmsnorm_bwd: N=%d must be a multiple of 8 and <= 2048", N);
  const int rows_per_block = N > 1024 ? 2 : 4;
  const int blocks = min(nnb_rmsnorm_bwd_blocks(), (M + rows_per_block - 1) / rows_per_block);
  bool done = false;
  int rc = 0;
#define X(cx, cd, cy, TX, TD, TY)                                                                      \
  if (!done && x_dtype == cx && delta_dtype == cd && y_dtype == cy) {                                   \
    rc = rmsnorm_bwd_t<TX, TD, TY>(dy, h, (const float*)rstd, (const float*)w, dres, dx, ddelta,        \
                                   (float*)dw_partial, blocks, M, N, st);                               \
    done = true;                                                                                        \
  }
  NNB_RMS_COMBOS(X)
#undef X
  NNB_REQUIRE(done, "add_rmsnorm_bwd: unsupported dtype combination (x=%d, delta=%d, y=%d)", x_dtype, delta_dtype, y_dtype);
  NNB_REQUIRE(rc == 0, "add_rmsnorm_bwd: cannot raise the shared-memory limit");
  NNB_LAUNCH_OK("add_rmsnorm_bwd");
  nnb_launch(dw_reduce_kernel, (N + 31) / 32, 1024, 0, st, (const float*)dw_partial, (float*)dw, blocks, N, accumulate_dw);
  NNB_LAUNCH_OK("rmsnorm_dw_reduce");
  return 0;
}

// ============================================================================ product with a device scalar
// dst[i] (+)= s[0] * src[i], fp32 product, one rounding into T. The gradients of the fused head are made in its forward pass for an
// upstream gradient of one; this is where the backward brings the real one in (it stays on the device). Bound by HBM: 16-byte
// accesses, one vector per thread. 50304 x 768 fp32: 45 us, adding into the gradient buffer about 70 us; the broadcasting
// elementwise kernels of PyTorch (scalar accesses) took 103 and 123 us.
template <typename T, bool ACC>
__global__ void __launch_bounds__(256) scale_kernel(const T* __restrict__ src, const float* __restrict__ scalar, T* __restrict__ dst,
                                                    long long n) {
  nnb_after_previous(src, scalar, dst);
  nnb_release_next();
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const float s = scalar[0];
  if (i + 8 <= n) {
    float a[8], d[8];
    Chunk8<T>::load(src + i, a);
    if (ACC) Chunk8<T>::load(dst + i, d);
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = ACC ? d[e] + s * a[e] : s * a[e];
    Chunk8<T>::store(dst + i, a);
  } else {
    for (long long j = i; j < n; ++j) {
      const float v = s * to_f32(src[j]);
      dst[j] = from_f32<T>(ACC ? to_f32(dst[j]) + v : v);
    }
  }
}

// src, dst: n contiguous elements of one dtype, 16-byte aligned; scalar: fp32 on the device; accumulate adds to dst.
extern "C" int nnb_scale(const void* src, const void* scalar, void* dst, long long n, int dtype, int accumulate, cudaStream_t st) {
  NNB_REQUIRE(n >= 0 && nnb_aligned16(src) && nnb_aligned16(dst), "scale: operands must be 16-byte aligned");
  NNB_REQUIRE(dtype == NNB_F32 || dtype == NNB_BF16 || dtype == NNB_F16, "scale: unsupported dtype code %d", dtype);
  if (n == 0) return 0;
  const unsigned blocks = (unsigned)((n + 2047) / 2048);
#define NNB_SCALE(T)                                                                                              \
  if (accumulate) nnb_launch(scale_kernel<T, true>, blocks, 256, 0, st, (const T*)src, (const float*)scalar, (T*)dst, n); \
  else nnb_launch(scale_kernel<T, false>, blocks, 256, 0, st, (const T*)src, (const float*)scalar, (T*)dst, n)
  if (dtype == NNB_F32) { NNB_SCALE(float); }
  else if (dtype == NNB_BF16) { NNB_SCALE(__nv_bfloat16); }
  else { NNB_SCALE(__half); }
#undef NNB_SCALE
  NNB_LAUNCH_OK("scale");
  return 0;
}

// ============================================================================ RoPE on packed QKV
// in/out: [M, row_stride] with (n_rot_heads) rotated heads of hd columns followed by n_copy_cols
// columns copied through (V). Row m uses table row (m % T). sin_sign = -1 gives the inverse (backward).
template <typename T>
__global__ void rope_packed_kernel(const T* __restrict__ in, T* __restrict__ out, const float* __restrict__ cos_t,
                                   const float* __restrict__ sin_t, long long M, int T_len, int n_rot_heads, int hd,
                                   int n_copy_cols, long long in_stride, long long out_stride, float sin_sign) {
  nnb_after_previous(in, out, cos_t, sin_t);
  nnb_release_next();
  const int half = hd >> 1, vec_per_half = half >> 3;
  const int rot_items = n_rot_heads * vec_per_half, copy_items = n_copy_cols >> 3;
  const int items = rot_items + copy_items;
  const long long total = M * items;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long m = idx / items;
    const int it = (int)(idx - m * items);
    const T* src = in + m * in_stride;
    T* dst = out + m * out_stride;
    if (it < rot_items) {
      const int head = it / vec_per_half, j = (it - head * vec_per_half) * 8;
      const int t = (int)(m % T_len);
      float a[8], b[8], c[8], s[8], o1[8], o2[8];
      Chunk8<T>::load(src + head * hd + j, a);
      Chunk8<T>::load(src + head * hd + half + j, b);
      Chunk8<float>::load(cos_t + (size_t)t * half + j, c);
      Chunk8<float>::load(sin_t + (size_t)t * half + j, s);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float sn = s[i] * sin_sign;
        o1[i] = a[i] * c[i] - b[i] * sn;
        o2[i] = a[i] * sn + b[i] * c[i];
      }
      Chunk8<T>::store(dst + head * hd + j, o1);
      Chunk8<T>::store(dst + head * hd + half + j, o2);
    } else {
      const int col = n_rot_heads * hd + (it - rot_items) * 8;
      float cp[8];
      Chunk8<T>::load(src + col, cp);
      Chunk8<T>::store(dst + col, cp);
    }
  }
}

extern "C" int nnb_rope_packed(const void* in, void* out, const void* cos_t, const void* sin_t, long long M, int T_len,
                               int n_rot_heads, int hd, int n_copy_cols, long long in_stride, long long out_stride,
                               float sin_sign, int dtype, cudaStream_t st) {
  NNB_REQUIRE(hd % 16 == 0, "rope: head_dim=%d must be a multiple of 16", hd);
  NNB_REQUIRE(n_copy_cols % 8 == 0 && in_stride % 8 == 0 && out_stride % 8 == 0, "rope: strides/cols must be multiples of 8");
  NNB_REQUIRE(nnb_aligned16(in) && nnb_aligned16(out) && nnb_aligned16(cos_t) && nnb_aligned16(sin_t), "rope: unaligned pointer");
  if (M == 0) return 0;
  const long long items = M * ((long long)n_rot_heads * (hd / 16) + n_copy_cols / 8);
  const int blocks = (int)min((items + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(dtype, T, {
    nnb_launch(rope_packed_kernel<T>, blocks, 256, 0, st, (const T*)in, (T*)out, (const float*)cos_t, (const float*)sin_t, M,
                                                  T_len, n_rot_heads, hd, n_copy_cols, in_stride, out_stride, sin_sign);
  });
  NNB_LAUNCH_OK("rope_packed");
  return 0;
}

// ============================================================================ SwiGLU
// out = silu(g) * u, rows of F columns; g, u, out with independent row strides (packed gate||up works).
template <typename T>
__global__ void swiglu_fwd_kernel(const T* __restrict__ g, const T* __restrict__ u, T* __restrict__ out, long long M,
                                  int F, long long g_stride, long long u_stride, long long o_stride) {
  nnb_after_previous(g, u, out);
  nnb_release_next();
  const int vec = F >> 3;
  const long long total = M * vec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long m = idx / vec;
    const int j = (int)(idx - m * vec) * 8;
    float a[8], b[8];
    Chunk8<T>::load(g + m * g_stride + j, a);
    Chunk8<T>::load(u + m * u_stride + j, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = a[i] / (1.f + __expf(-a[i])) * b[i];
    Chunk8<T>::store(out + m * o_stride + j, a);
  }
}

// dg = dy*u*s*(1 + g*(1-s)), du = dy*g*s with s = sigmoid(g) recomputed (only g, u are saved).
template <typename T>
__global__ void swiglu_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ g, const T* __restrict__ u,
                                  T* __restrict__ dg, T* __restrict__ du, long long M, int F, long long dy_stride,
                                  long long g_stride, long long u_stride, long long dg_stride, long long du_stride) {
  nnb_after_previous(dy, g, u, dg, du);
  nnb_release_next();
  const int vec = F >> 3;
  const long long total = M * vec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long m = idx / vec;
    const int j = (int)(idx - m * vec) * 8;
    float d[8], a[8], b[8], og[8], ou[8];
    Chunk8<T>::load(dy + m * dy_stride + j, d);
    Chunk8<T>::load(g + m * g_stride + j, a);
    Chunk8<T>::load(u + m * u_stride + j, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = 1.f / (1.f + __expf(-a[i]));
      og[i] = d[i] * b[i] * s * (1.f + a[i] * (1.f - s));
      ou[i] = d[i] * a[i] * s;
    }
    Chunk8<T>::store(dg + m * dg_stride + j, og);
    Chunk8<T>::store(du + m * du_stride + j, ou);
  }
}

extern "C" int nnb_swiglu_fwd(const void* g, const void* u, void* out, long long M, int F, long long g_stride,
                              long long u_stride, long long o_stride, int dtype, cudaStream_t st) {
  NNB_REQUIRE(F % 8 == 0 && g_stride % 8 == 0 && u_stride % 8 == 0 && o_stride % 8 == 0, "swiglu: F and strides must be multiples of 8");
  NNB_REQUIRE(nnb_aligned16(g) && nnb_aligned16(u) && nnb_aligned16(out), "swiglu: unaligned pointer");
  if (M == 0) return 0;
  const int blocks = (int)min((M * (F / 8) + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(dtype, T, {
    nnb_launch(swiglu_fwd_kernel<T>, blocks, 256, 0, st, (const T*)g, (const T*)u, (T*)out, M, F, g_stride, u_stride, o_stride);
  });
  NNB_LAUNCH_OK("swiglu_fwd");
  return 0;
}

extern "C" int nnb_swiglu_bwd(const void* dy, const void* g, const void* u, void* dg, void* du, long long M, int F,
                              long long dy_stride, long long g_stride, long long u_stride, long long dg_stride,
                              long long du_stride, int dtype, cudaStream_t st) {
  NNB_REQUIRE(F % 8 == 0 && dy_stride % 8 == 0 && g_stride % 8 == 0 && u_stride % 8 == 0 && dg_stride % 8 == 0 && du_stride % 8 == 0,
              "swiglu_bwd: F and strides must be multiples of 8");
  if (M == 0) return 0;
  const int blocks = (int)min((M * (F / 8) + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(dtype, T, {
    nnb_launch(swiglu_bwd_kernel<T>, blocks, 256, 0, st, (const T*)dy, (const T*)g, (const T*)u, (T*)dg, (T*)du, M, F, dy_stride,
                                                 g_stride, u_stride, dg_stride, du_stride);
  });
  NNB_LAUNCH_OK("swiglu_bwd");
  return 0;
}

// ============================================================================ embedding
// out[m, :] = W[idx[m], :] (W fp32 master) in the residual dtype.
template <typename TO>
__global__ void embedding_fwd_kernel(const long long* __restrict__ idx, const float* __restrict__ W,
                                     TO* __restrict__ out, long long M, int D, int vocab) {
  nnb_after_previous(idx, W, out);
  nnb_release_next();
  const int vec = D >> 3;
  const long long total = M * vec;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long m = i / vec;
    const int j = (int)(i - m * vec) * 8;
    long long row = idx[m];
    row = row < 0 ? 0 : (row >= vocab ? vocab - 1 : row);
    float v[8];
    Chunk8<float>::load(W + row * D + j, v);
    Chunk8<TO>::store(out + m * D + j, v);
  }
}

// dW[idx[m], :] += dout[m, :] with 16-byte vector reductions (red.global.add.v4.f32): rows that
// repeat inside the batch are summed by the memory system, nothing is sorted.
template <typename TO>
__global__ void embedding_bwd_kernel(const long long* __restrict__ idx, const TO* __restrict__ dout,
                                     float* __restrict__ dW, long long M, int D, int vocab) {
  nnb_after_previous(idx, dout, dW);
  nnb_release_next();
  const int vec = D >> 3;
  const long long total = M * vec;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long m = i / vec;
    const int j = (int)(i - m * vec) * 8;
    long long row = idx[m];
    if (row < 0 || row >= vocab) continue;
    float v[8];
    Chunk8<TO>::load(dout + m * D + j, v);
    float* dst = dW + row * D + j;
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
  }
}

extern "C" int nnb_embedding_fwd(const void* idx, const void* W, void* out, long long M, int D, int vocab,
                                 int out_dtype, cudaStream_t st) {
  NNB_REQUIRE(D % 8 == 0, "embedding: D=%d must be a multiple of 8", D);
  if (M == 0) return 0;
  const int blocks = (int)min((M * (D / 8) + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(out_dtype, TO, {
    nnb_launch(embedding_fwd_kernel<TO>, blocks, 256, 0, st, (const long long*)idx, (const float*)W, (TO*)out, M, D, vocab);
  });
  NNB_LAUNCH_OK("embedding_fwd");
  return 0;
}

extern "C" int nnb_embedding_bwd(const void* idx, const void* dout, void* dW, long long M, int D, int vocab,
                                 int dout_dtype, cudaStream_t st) {
  NNB_REQUIRE(D % 8 == 0, "embedding_bwd: D=%d must be a multiple of 8", D);
  if (M == 0) return 0;
  const int blocks = (int)min((M * (D / 8) + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(dout_dtype, TO, {
    nnb_launch(embedding_bwd_kernel<TO>, blocks, 256, 0, st, (const long long*)idx, (const TO*)dout, (float*)dW, M, D, vocab);
  });
  NNB_LAUNCH_OK("embedding_bwd");
  return 0;
}

// ============================================================================ warm-up add (toolchain smoke test)
__global__ void warmup_add_kernel(const float* a, const float* b, float* c, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) c[i] = a[i] + b[i];
}

extern "C" int nnb_warmup_add(const void* a, const void* b, void* c, long long n, cudaStream_t st) {
  if (n == 0) return 0;
  warmup_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const float*)a, (const float*)b, (float*)c, n);
  NNB_LAUNCH_OK("warmup_add");
  return 0;
}

// ============================================================================ dtype cast (fp32 -> 16-bit shadow)
template <typename TO>
__global__ void cast_from_f32_kernel(const float* __restrict__ in, TO* __restrict__ out, long long n8) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float v[8];
    Chunk8<float>::load(in + i * 8, v);
    Chunk8<TO>::store(out + i * 8, v);
  }
}

extern "C" int nnb_cast_from_f32(const void* in, void* out, long long n, int out_dtype, cudaStream_t st) {
  NNB_REQUIRE(n % 8 == 0, "cast: n must be a multiple of 8");
  if (n == 0) return 0;
  const int blocks = (int)min((n / 8 + 255) / 256, (long long)nnb_num_sms() * 16);
  NNB_DISPATCH(out_dtype, TO, { cast_from_f32_kernel<TO><<<blocks, 256, 0, st>>>((const float*)in, (TO*)out, n / 8); });
  NNB_LAUNCH_OK("cast_from_f32");
  return 0;
}

// Shared host/device helpers for the sm_100a kernel library: error reporting for the extern "C"
// launchers, dtype codes, 16-byte vector load/store helpers and warp reductions.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

// ---- host-side error channel: launchers return 0 or a negative code and leave a message here
extern "C" const char* nnb_last_error();
void nnb_set_error(const char* fmt, ...);

#define NNB_REQUIRE(cond, ...)           \
  do {                                   \
    if (!(cond)) {                       \
      nnb_set_error(__VA_ARGS__);        \
      return -1;                         \
    }                                    \
  } while (0)

#define NNB_LAUNCH_OK(name)                                                      \
  do {                                                                           \
    cudaError_t e_ = cudaGetLastError();                                         \
    if (e_ != cudaSuccess) {                                                     \
      nnb_set_error("%s: launch failed: %s", name, cudaGetErrorString(e_));      \
      return -100;                                                               \
    }                                                                            \
  } while (0)

enum NnbDtype : int { NNB_F32 = 0, NNB_BF16 = 1, NNB_F16 = 2 };

static inline int nnb_num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

// Launch that may begin while the previous kernel of the stream is still running its last blocks: blocks are placed as SMs fall free, set
// themselves up (barriers, tensor memory, descriptors) and stop in nnb_after_previous(), which EVERY kernel launched this way calls
// before it touches global memory. What it returns to is what stream order gives: the previous kernel, and with it everything before
// it, has finished and its writes are visible. A kernel lets its successor in with nnb_release_next() when its own work is nearly
// handed out, not earlier: blocks that wait hold their SM's resources, which kernels of other streams may want.
// An eager step of the 114M model in two micro-batches of 4096 tokens is 574 launches with 1.7 us of idle GPU before each: 12.0 ms
// in plain launches, 11.1 in these (8192 tokens in fp8: 11.6 and 11.1). Not every kernel gains: see nnb_launch_pre_pass.
// `cluster`: CTAs of a cluster along x, 1 for a kernel without clusters (or with its own __cluster_dims__).
template <typename... K, typename... A>
static inline void nnb_launch_clusters(void (*kernel)(K...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);  // (its error is read by NNB_LAUNCH_OK)
}
template <typename... K, typename... A>
static inline void nnb_launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  nnb_launch_clusters(kernel, 1, grid, block, smem, st, args...);
}

static inline bool nnb_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

#ifdef __CUDACC__
// See nnb_launch_clusters. The pointers through which the kernel reads are named here: their values then come out of the statement after
// the wait, so that no load (read-only loads obey no memory clobber) can be moved above it.
template <typename... P>
__device__ __forceinline__ void nnb_after_previous(P&... pointers) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  ((void)[&] { asm volatile("" : "+l"(pointers)); }(), ...);
}
__device__ __forceinline__ void nnb_release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- 8-element (one "chunk") loads/stores converting to/from fp32 registers
template <typename T>
struct Chunk8;

template <>
struct Chunk8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
};

template <>
struct Chunk8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
  }
};

template <>
struct Chunk8<__half> {
  static __device__ __forceinline__ void load(const __half* p, float (&v)[8]) {
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __half22float2(h[i]);
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__half* p, const float (&v)[8]) {
    uint4 raw;
    __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
  }
};

// A chunk in global memory, at 32-byte aligned addresses where WIDE: eight fp32 values are then one access of a whole sector a lane instead of
// two of half a sector.
template <typename T, bool WIDE>
struct GlobalChunk8 : Chunk8<T> {};
template <>
struct GlobalChunk8<float, true> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
  }
};

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Dispatch a dtype code to a type tag: NNB_DISPATCH(code, T, { body using T })
#define NNB_DISPATCH(code, T, ...)                                  \
  switch (code) {                                                   \
    case NNB_F32: { using T = float; __VA_ARGS__; break; }          \
    case NNB_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; } \
    case NNB_F16: { using T = __half; __VA_ARGS__; break; }         \
    default: nnb_set_error("unknown dtype code %d", code); return -2; \
  }
#define NNB_DISPATCH_16(code, T, ...)                               \
  switch (code) {                                                   \
    case NNB_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; } \
    case NNB_F16: { using T = __half; __VA_ARGS__; break; }         \
    default: nnb_set_error("expected a 16-bit float dtype, got code %d", code); return -2; \
  }
#endif

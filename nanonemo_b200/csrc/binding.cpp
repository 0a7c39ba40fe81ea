// Native binding of the operators: argument checks, allocation, launches and autograd nodes without Python in between.
//
// The kernel library keeps its plain extern "C" launchers; this extension (the only translation unit that knows torch's headers) calls
// them from C++. Two layers:
//   raw functions   one launch each on given tensors (gemm, flash_fwd, ...): what the Python launch helpers of nanonemo_b200/ops call.
//   operators       linear, add_rms_norm, flash_attn, qkv_rope_attention, mlp_swiglu with C++ autograd nodes; a whole block without gradients.
// Why: the host set the pace of every call that is not replayed from a graph. A Python launch helper took 12 us (torch.empty, views,
// 15 to 45 converted arguments), a registered operator with its formula 25 to 40 us more in each direction. us a pass, through
// Python / natively: optimizer step of the 114M model in two micro-batches of 4 x 1024 17,300 / 12,100 (11,400 of kernels), scoring 201
// tokens 4,680 / 1,830, attention forward and backward over 2 x 333 tokens 246 / 96, add + norm of 16384 x 768 197 / 95.
//
// An operator serves PLAIN calls only: exact torch.Tensor / Parameter arguments on CUDA, no tangents, and no transform, tracer or
// mode active in this thread. Anything else is answered with NotImplemented and takes the registered operators or the Python
// autograd functions, as every call did before. Backward nodes that belong to the registered operators do the same with their
// upstream gradient: under create_graph=True, or for a gradient that is not plain (is_grads_batched=True), they call the
// registered operators through the dispatcher, which differentiate, batch or refuse as they always have.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <cmath>
#include <map>
#include <mutex>

namespace py = pybind11;
using at::Tensor;
using c10::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

extern "C" {
typedef struct CUstream_st* cudaStream_t;
const char* nnb_last_error();
int nnb_gemm_bf16(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, int, int, int, int, int, void*, cudaStream_t);
int nnb_gemm_rows_rope(const void*, const void*, void*, const void*, const void*, int, int, int, long long, long long, long long, int, int, int, int, int, int, void*, cudaStream_t);
int nnb_gemm_rows_f32w_serves(int, int, int, int);
int nnb_gemm_rows_f32w(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, void*, cudaStream_t);
int nnb_gemm_rows_f32w_swiglu(const void*, const void*, void*, int, int, int, long long, long long, long long, int, void*, cudaStream_t);
int nnb_gemm_swiglu(const void*, const void*, void*, void*, int, int, int, long long, long long, long long, long long, int, void*, cudaStream_t);
int nnb_gemm_swiglu_act(const void*, const void*, void*, int, int, int, long long, long long, long long, int, void*, cudaStream_t);
int nnb_gemm_swiglu_bwd(const void*, const void*, const void*, void*, int, int, int, long long, long long, long long, long long, int, void*, cudaStream_t);
int nnb_gemm_rope(const void*, const void*, void*, const void*, const void*, int, int, int, long long, long long, long long, int, int, int, int, void*, cudaStream_t);
int nnb_gemm_mxfp8(const void*, const void*, const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, int, void*, cudaStream_t);
int nnb_mxfp8_quantize_sw(const void*, long long, void*, long long, void*, void*, long long, void*, int, int, cudaStream_t);
int nnb_mxfp8_swiglu(const void*, long long, void*, long long, void*, void*, long long, void*, int, int, cudaStream_t);
int nnb_mxfp8_swiglu_bwd(const void*, long long, const void*, long long, void*, long long, void*, void*, long long, void*, int, int, cudaStream_t);
int nnb_add_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, void*, int, int, float, int, int, int, cudaStream_t);
int nnb_rmsnorm_bwd_blocks();
int nnb_add_rmsnorm_bwd(const void*, const void*, const void*, const void*, const void*, void*, void*, void*, void*, int, int, int, int, int, int, cudaStream_t);
int nnb_rope_packed(const void*, void*, const void*, const void*, long long, int, int, int, int, long long, long long, float, int, cudaStream_t);
int nnb_swiglu_fwd(const void*, const void*, void*, long long, int, long long, long long, long long, int, cudaStream_t);
int nnb_swiglu_bwd(const void*, const void*, const void*, void*, void*, long long, int, long long, long long, long long, long long, long long, int, cudaStream_t);
int nnb_flash_fwd(const void*, const void*, const void*, void*, void*, int, int, int, int, int, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, float, int, void*, cudaStream_t);
int nnb_flash_bwd(const void*, const void*, const void*, const void*, const void*, const void*, void*, void*, void*, void*, void*, int, int, int, int, int, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, long long, float, int, const void*, const void*, int, void*, cudaStream_t);
}

namespace {

// What the Python helpers raised as AssertionError and TypeError keeps its type.
struct AssertionFailed : std::runtime_error { using std::runtime_error::runtime_error; };
struct WrongType : std::runtime_error { using std::runtime_error::runtime_error; };
#define NNB_ASSERT(cond, msg) do { if (!(cond)) throw AssertionFailed(msg); } while (0)

std::atomic<long long> g_launches{0};

void launched(int rc, const char* name) {
  if (rc != 0) {
    const char* msg = nnb_last_error();
    throw std::runtime_error(std::string(name) + " failed (code " + std::to_string(rc) + "): " + (msg ? msg : "no message"));
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
}
// Launchers that answer 1 when they do not serve the problem (nothing was launched).
bool served(int rc, const char* name) {
  if (rc == 1) return false;
  launched(rc, name);
  return true;
}
cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The status words of the bounded waits, one tensor per device (never freed: kernels in flight may write to it until the process ends).
std::mutex g_status_mutex;
std::map<int, Tensor>& status_map() {
  static auto* m = new std::map<int, Tensor>();
  return *m;
}
Tensor status_tensor(int device) {
  std::lock_guard<std::mutex> lock(g_status_mutex);
  Tensor& t = status_map()[device];
  if (!t.defined()) {
    c10::impl::ExcludeDispatchKeyGuard no_modes(c10::DispatchKeySet(c10::DispatchKey::Python));
    at::NoGradGuard no_grad;
    t = at::zeros({4}, at::device(at::Device(at::kCUDA, (c10::DeviceIndex)device)).dtype(at::kInt));
  }
  return t;
}
void* status_of(const Tensor& like) { return status_tensor(like.get_device()).data_ptr(); }

// A kernel that is given pageable host memory faults, and the context is lost.
void reachable(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->defined() && !t->is_cuda() && !(t->is_cpu() && t->is_pinned())) throw AssertionFailed("the GPU cannot reach an operand on " + t->device().str());
}

int code_of(at::ScalarType t) {  // -1: no operand format of the kernels
  return t == at::kFloat ? 0 : t == at::kBFloat16 ? 1 : t == at::kHalf ? 2 : -1;
}
int code16(at::ScalarType t) { const int c = code_of(t); return c >= 1 ? c : -1; }
int code_any(const Tensor& t) {
  const int c = code_of(t.scalar_type());
  if (c < 0) throw WrongType(std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
  return c;
}

Tensor rowmajor2d(Tensor t) {
  if (t.dim() != 2) t = t.reshape({-1, t.size(-1)});
  if (t.stride(1) != 1 || (t.stride(0) * (int64_t)t.element_size()) % 16 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) t = t.contiguous();
  return t;
}
Tensor rows2d(const Tensor& t) { return t.dim() == 2 ? t : t.reshape({-1, t.size(-1)}); }
Tensor as_dtype(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }
Tensor dense_rows(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
Tensor empty(at::IntArrayRef size, at::ScalarType dt, const Tensor& like) { return at::empty(size, like.options().dtype(dt).requires_grad(false).memory_format(std::nullopt)); }

// ------------------------------------------------------------------------------------------------ raw functions
// (A kernel takes one of the two for both operands: it would read past the end of the shorter one.)
void inner_dimensions(int64_t a, int64_t b) { NNB_ASSERT(a == b, "inner dimensions differ: " + std::to_string(a) + " vs " + std::to_string(b)); }

Tensor gemm(Tensor a, Tensor b, bool a_mn, bool b_mn, const optional<Tensor>& out_, optional<at::ScalarType> out_dtype, bool accumulate, int k_splits, int bn, int max_ctas) {
  a = rowmajor2d(std::move(a));
  b = rowmajor2d(std::move(b));
  reachable({&a, &b});
  if (out_ && out_->defined()) reachable({&a, &*out_});
  NNB_ASSERT(a.scalar_type() == b.scalar_type() && code16(a.scalar_type()) > 0,
             std::string("gemm needs matching bf16/fp16 inputs, got ") + c10::toString(a.scalar_type()) + "/" + c10::toString(b.scalar_type()));
  const int64_t K = a_mn ? a.size(0) : a.size(1), M = a_mn ? a.size(1) : a.size(0);
  const int64_t Kb = b_mn ? b.size(0) : b.size(1), N = b_mn ? b.size(1) : b.size(0);
  inner_dimensions(K, Kb);
  const bool given = out_.has_value() && out_->defined();
  const at::ScalarType dt = out_dtype ? *out_dtype : given ? out_->scalar_type() : a.scalar_type();
  NNB_ASSERT(dt == a.scalar_type() || dt == at::kFloat, "gemm: the output is of the operands' dtype or fp32");
  NNB_ASSERT(given || !accumulate, "gemm: accumulate needs an output");
  Tensor out = given ? *out_ : empty({M, N}, dt, a);
  NNB_ASSERT(out.dim() == 2 && out.size(0) == M && out.size(1) == N && out.stride(1) == 1 && out.scalar_type() == dt, "gemm: the output does not fit");
  launched(nnb_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn, code16(a.scalar_type()),
                         dt == at::kFloat, accumulate, k_splits, bn, max_ctas, status_of(a), stream()), "nnb_gemm_bf16");
  return out;
}
Tensor gemm_nt(const Tensor& a, const Tensor& b, bool b_mn = false) { return gemm(a, b, false, b_mn, std::nullopt, std::nullopt, false, 0, 0, 0); }

// x2 [M, K] @ w_gu [2 F, K]^T -> (gu, act), (undefined, act) without `keep`, or two undefined tensors where the CTA-pair kernel does not serve the shape
std::pair<Tensor, Tensor> gemm_swiglu(const Tensor& x2, const Tensor& w, bool keep) {
  reachable({&x2, &w});
  const int64_t M = x2.size(0), K = x2.size(1), F = w.size(0) / 2;
  if (M < 256 || F % 128 || w.stride(1) != 1 || x2.stride(1) != 1) return {};
  inner_dimensions(K, w.size(1));
  Tensor gu = keep ? empty({M, 2 * F}, x2.scalar_type(), x2) : Tensor(), act = empty({M, F}, x2.scalar_type(), x2);
  const int code = code16(x2.scalar_type());
  NNB_ASSERT(code > 0 && w.scalar_type() == x2.scalar_type(), "gemm_swiglu needs bf16 or fp16 operands of one dtype");
  const bool ok = keep ? served(nnb_gemm_swiglu(x2.data_ptr(), w.data_ptr(), gu.data_ptr(), act.data_ptr(), (int)M, (int)F, (int)K, x2.stride(0), w.stride(0), 2 * F, F, code,
                                                status_of(x2), stream()), "nnb_gemm_swiglu")
                       : served(nnb_gemm_swiglu_act(x2.data_ptr(), w.data_ptr(), act.data_ptr(), (int)M, (int)F, (int)K, x2.stride(0), w.stride(0), F, code, status_of(x2),
                                                    stream()), "nnb_gemm_swiglu_act");
  if (!ok) return {};
  return {gu, act};
}

Tensor gemm_swiglu_bwd(const Tensor& dy, const Tensor& w, const Tensor& gu) {
  reachable({&dy, &w, &gu});
  const int64_t M = dy.size(0), K = dy.size(1), F = w.size(1);
  if (M < 256 || F < 128 || F % 64 || gu.dim() != 2 || gu.size(0) != M || gu.size(1) != 2 * F || gu.stride(1) != 1 || gu.stride(0) % 8 || w.stride(1) != 1 ||
      dy.stride(1) != 1 || gu.scalar_type() != dy.scalar_type() || w.scalar_type() != dy.scalar_type())
    return Tensor();
  inner_dimensions(K, w.size(0));
  const int code = code16(dy.scalar_type());
  NNB_ASSERT(code > 0, "gemm_swiglu_bwd needs bf16 or fp16 operands");
  Tensor dgu = empty({M, 2 * F}, gu.scalar_type(), gu);
  return served(nnb_gemm_swiglu_bwd(dy.data_ptr(), w.data_ptr(), gu.data_ptr(), dgu.data_ptr(), (int)M, (int)F, (int)K, dy.stride(0), w.stride(0), gu.stride(0), 2 * F, code,
                                    status_of(dy), stream()), "nnb_gemm_swiglu_bwd") ? dgu : Tensor();
}

Tensor gemm_rope(const Tensor& x2, const Tensor& w, const Tensor& cos, const Tensor& sin, int64_t t_len, int64_t rope_cols, int64_t hd) {
  reachable({&x2, &w, &cos, &sin});
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  inner_dimensions(K, w.size(1));
  if ((hd != 64 && hd != 128) || N % hd || rope_cols % hd || w.stride(1) != 1 || x2.stride(1) != 1) return Tensor();
  const int code = code16(x2.scalar_type());
  NNB_ASSERT(code > 0 && w.scalar_type() == x2.scalar_type(), "gemm_rope needs bf16 or fp16 operands of one dtype");
  Tensor out = empty({M, N}, x2.scalar_type(), x2);
  return served(nnb_gemm_rope(x2.data_ptr(), w.data_ptr(), out.data_ptr(), cos.data_ptr(), sin.data_ptr(), (int)M, (int)N, (int)K, x2.stride(0), w.stride(0), N, (int)t_len,
                              (int)rope_cols, (int)hd, code, status_of(x2), stream()), "nnb_gemm_rope") ? out : Tensor();
}

// Products of a few rows with a weight that has no 16-bit copy, straight from its fp32 values (the bits are those of the cast and the usual
// product); undefined where that is not served.
bool from_f32(const Tensor& x2, const Tensor& w) {
  return w.scalar_type() == at::kFloat && w.dim() == 2 && w.stride(1) == 1 && x2.dim() == 2 && x2.stride(1) == 1 && x2.size(1) == w.size(1) && code16(x2.scalar_type()) > 0 &&
         x2.numel() > 0 && w.numel() > 0;
}
bool f32w_serves(int64_t M, int64_t N, int64_t K, int kind) { return nnb_gemm_rows_f32w_serves((int)M, (int)N, (int)K, kind) != 0; }
Tensor gemm_f32w(const Tensor& x2, const Tensor& w) {
  if (!from_f32(x2, w) || !f32w_serves(x2.size(0), w.size(0), w.size(1), 0)) return Tensor();
  reachable({&x2, &w});
  const int64_t M = x2.size(0), N = w.size(0);
  Tensor y = empty({M, N}, x2.scalar_type(), x2);
  return served(nnb_gemm_rows_f32w(x2.data_ptr(), w.data_ptr(), y.data_ptr(), (int)M, (int)N, (int)w.size(1), x2.stride(0), w.stride(0), N, 0, code16(x2.scalar_type()), status_of(x2),
                                   stream()), "nnb_gemm_rows_f32w") ? y : Tensor();
}
// dy2 w, the input gradient of such a product
Tensor gemm_f32w_dgrad(const Tensor& dy2, const Tensor& w) {
  if (w.scalar_type() != at::kFloat || w.dim() != 2 || w.stride(1) != 1 || dy2.dim() != 2 || dy2.stride(1) != 1 || dy2.size(1) != w.size(0) || code16(dy2.scalar_type()) < 0 || dy2.numel() == 0 ||
      w.numel() == 0 || !f32w_serves(dy2.size(0), w.size(1), w.size(0), 2))
    return Tensor();
  reachable({&dy2, &w});
  const int64_t M = dy2.size(0), N = w.size(1);
  Tensor dx = empty({M, N}, dy2.scalar_type(), dy2);
  return served(nnb_gemm_rows_f32w(dy2.data_ptr(), w.data_ptr(), dx.data_ptr(), (int)M, (int)N, (int)w.size(0), dy2.stride(0), w.stride(0), N, 1, code16(dy2.scalar_type()), status_of(dy2),
                                   stream()), "nnb_gemm_rows_f32w") ? dx : Tensor();
}
Tensor gemm_f32w_swiglu(const Tensor& x2, const Tensor& w) {
  if (!from_f32(x2, w) || w.size(0) % 2 || !f32w_serves(x2.size(0), w.size(0) / 2, w.size(1), 1)) return Tensor();
  reachable({&x2, &w});
  const int64_t M = x2.size(0), F = w.size(0) / 2;
  Tensor act = empty({M, F}, x2.scalar_type(), x2);
  return served(nnb_gemm_rows_f32w_swiglu(x2.data_ptr(), w.data_ptr(), act.data_ptr(), (int)M, (int)F, (int)w.size(1), x2.stride(0), w.stride(0), F, code16(x2.scalar_type()),
                                          status_of(x2), stream()), "nnb_gemm_rows_f32w_swiglu") ? act : Tensor();
}
Tensor gemm_f32w_rope(const Tensor& x2, const Tensor& w, const Tensor& cos, const Tensor& sin, int64_t t_len, int64_t rope_cols, int64_t hd) {
  if (!from_f32(x2, w) || (hd != 64 && hd != 128) || w.size(0) % hd || rope_cols % hd || !f32w_serves(x2.size(0), w.size(0), w.size(1), 0)) return Tensor();
  reachable({&x2, &w, &cos, &sin});
  const int64_t M = x2.size(0), N = w.size(0);
  Tensor y = empty({M, N}, x2.scalar_type(), x2);
  return served(nnb_gemm_rows_rope(x2.data_ptr(), w.data_ptr(), y.data_ptr(), cos.data_ptr(), sin.data_ptr(), (int)M, (int)N, (int)w.size(1), x2.stride(0), w.stride(0), N, (int)t_len,
                                   (int)rope_cols, (int)hd, code16(x2.scalar_type()), /*f32w=*/1, 16, status_of(x2), stream()), "nnb_gemm_rows_rope") ? y : Tensor();
}

void rope_packed(const Tensor& x2, const Tensor& out2, const Tensor& cos, const Tensor& sin, int64_t T, int64_t n_rot, int64_t hd, int64_t n_copy, double sign) {
  reachable({&x2, &out2, &cos, &sin});
  launched(nnb_rope_packed(x2.data_ptr(), out2.data_ptr(), cos.data_ptr(), sin.data_ptr(), x2.size(0), (int)T, (int)n_rot, (int)hd, (int)n_copy, x2.stride(0), out2.stride(0),
                           (float)sign, code_any(x2), stream()), "nnb_rope_packed");
}
void swiglu_fwd(const Tensor& g, const Tensor& u, const Tensor& out) {
  reachable({&g, &u, &out});
  launched(nnb_swiglu_fwd(g.data_ptr(), u.data_ptr(), out.data_ptr(), out.size(0), (int)out.size(1), g.stride(0), u.stride(0), out.stride(0), code_any(out), stream()), "nnb_swiglu_fwd");
}
void swiglu_bwd(const Tensor& dy, const Tensor& g, const Tensor& u, const Tensor& dg, const Tensor& du) {
  reachable({&dy, &g, &u, &dg, &du});
  launched(nnb_swiglu_bwd(dy.data_ptr(), g.data_ptr(), u.data_ptr(), dg.data_ptr(), du.data_ptr(), dy.size(0), (int)dy.size(1), dy.stride(0), g.stride(0), u.stride(0), dg.stride(0),
                          du.stride(0), code_any(dy), stream()), "nnb_swiglu_bwd");
}

// (y, h, rstd) in two dimensions; h is x2 itself without a delta
std::tuple<Tensor, Tensor, Tensor> rms_fwd(const Tensor& x, const optional<Tensor>& delta, const Tensor& weight, double eps, at::ScalarType y_dt) {
  const int64_t N = x.size(-1);
  Tensor x2 = x.reshape({-1, N}).contiguous(), d2;
  if (delta && delta->defined()) d2 = delta->reshape({-1, N}).contiguous();
  const int64_t M = x2.size(0);
  reachable({&x2, &d2, &weight});
  const Tensor w = as_dtype(weight, at::kFloat);
  Tensor y = empty({M, N}, y_dt, x), h = d2.defined() ? empty({M, N}, x2.scalar_type(), x) : x2, rstd = empty({M}, at::kFloat, x);
  const int y_code = code_any(y);
  launched(nnb_add_rmsnorm_fwd(x2.data_ptr(), d2.defined() ? d2.data_ptr() : nullptr, w.data_ptr(), y.data_ptr(), h.data_ptr(), rstd.data_ptr(), (int)M, (int)N, (float)eps, code_any(x2),
                               d2.defined() ? code_any(d2) : y_code, y_code, stream()), "nnb_add_rmsnorm_fwd");
  return {y, h, rstd};
}

// (dx, ddelta or undefined, dw); ddelta is dx where their dtypes agree
std::tuple<Tensor, Tensor, Tensor> rms_bwd(const Tensor& dy, const Tensor& h, const Tensor& rstd, const Tensor& weight, const optional<Tensor>& dres, optional<at::ScalarType> delta_dt,
                                           const optional<Tensor>& dw_out, bool accumulate) {
  const int64_t N = h.size(-1);
  const Tensor h2 = h.reshape({-1, N}), dy2 = dy.reshape({-1, N}).contiguous();
  const int64_t M = h2.size(0);
  Tensor dr2;
  if (dres && dres->defined()) dr2 = as_dtype(dres->reshape({-1, N}).contiguous(), h2.scalar_type());
  reachable({&h2, &dy2, &dr2, &rstd, &weight});
  if (dw_out && dw_out->defined()) reachable({&h2, &*dw_out});
  const Tensor w = as_dtype(weight, at::kFloat);
  Tensor dx = at::empty_like(h2), ddelta;
  if (delta_dt && *delta_dt != h2.scalar_type()) ddelta = empty({M, N}, *delta_dt, h);
  const Tensor partial = empty({nnb_rmsnorm_bwd_blocks(), N}, at::kFloat, h);
  const Tensor dw = dw_out && dw_out->defined() ? *dw_out : empty({N}, at::kFloat, h);
  const int dy_code = code_any(dy2);
  int d_code = dy_code;
  if (delta_dt && (d_code = code_of(*delta_dt)) < 0) throw WrongType("add_rmsnorm_bwd: unsupported dtype of the delta");
  launched(nnb_add_rmsnorm_bwd(dy2.data_ptr(), h2.data_ptr(), rstd.data_ptr(), w.data_ptr(), dr2.defined() ? dr2.data_ptr() : nullptr, dx.data_ptr(),
                               ddelta.defined() ? ddelta.data_ptr() : nullptr, dw.data_ptr(), partial.data_ptr(), (int)M, (int)N, code_any(h2), d_code, dy_code, accumulate, stream()),
           "nnb_add_rmsnorm_bwd");
  dx = dx.view(h.sizes());
  if (ddelta.defined()) ddelta = ddelta.view(h.sizes());
  else if (delta_dt) ddelta = dx;
  return {dx, ddelta, dw};
}

int attention_code(std::initializer_list<const Tensor*> ts) {
  const at::ScalarType dt = (*ts.begin())->scalar_type();
  for (const Tensor* t : ts) {
    if (code16(dt) < 0 || t->scalar_type() != dt) throw WrongType("attention kernels take bf16 or fp16 operands of one dtype");
    NNB_ASSERT(t->stride(-1) == 1, "last dimension must be contiguous");
  }
  return code16(dt);
}
#define NNB_STRIDES(t) (t).stride(0), (t).stride(1), (t).stride(2)

// q, o: [B, T, H, hd] views; k, v: [B, T, KVH, hd] views
Tensor flash_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, double scale) {
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), hd = q.size(3), KVH = k.size(2);
  reachable({&q, &k, &v, &o});
  const int code = attention_code({&q, &k, &v, &o});
  Tensor lse = empty({B, H, T}, at::kFloat, q);
  launched(nnb_flash_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), (int)B, (int)T, (int)H, (int)KVH, (int)hd, NNB_STRIDES(q), NNB_STRIDES(k), NNB_STRIDES(v),
                         NNB_STRIDES(o), (float)scale, code, status_of(q), stream()), "nnb_flash_fwd");
  return lse;
}
void flash_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& dout, const Tensor& dq, const Tensor& dk, const Tensor& dv, double scale,
               const optional<Tensor>& cos, const optional<Tensor>& sin, bool in_order) {
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), hd = q.size(3), KVH = k.size(2);
  reachable({&q, &k, &v, &o, &lse, &dout, &dq, &dk, &dv});
  if (cos && sin) reachable({&q, &*cos, &*sin});
  const int code = attention_code({&q, &k, &v, &o, &dout, &dq, &dk, &dv});
  const Tensor delta = empty({B, H, T}, at::kFloat, q);     // rowsum(dO * O), computed by the launcher's pre-pass
  const Tensor dq_acc = empty({B, T, H, hd}, at::kFloat, q);  // cleared by the pre-pass
  launched(nnb_flash_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dout.data_ptr(), lse.data_ptr(), delta.data_ptr(), dq_acc.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                         dv.data_ptr(), (int)B, (int)T, (int)H, (int)KVH, (int)hd, NNB_STRIDES(q), NNB_STRIDES(k), NNB_STRIDES(v), NNB_STRIDES(o), NNB_STRIDES(dout), NNB_STRIDES(dq),
                         NNB_STRIDES(dk), NNB_STRIDES(dv), (float)scale, code, cos ? cos->data_ptr() : nullptr, sin ? sin->data_ptr() : nullptr, in_order, status_of(q), stream()),
           "nnb_flash_bwd");
}

// MXFP8: quantised copies (see nanonemo_b200/fp8) and the block-scaled product
struct Quantized {
  Tensor q, sf, qt, sft;
  Quantized(int64_t R, int64_t C, bool rowwise, bool colwise, const Tensor& like) {
    const int64_t scales = (R / 128) * (C / 128) * 512;
    if (rowwise) { q = empty({R, C}, at::kByte, like); sf = empty({scales}, at::kByte, like); }
    if (colwise) { qt = empty({C, R}, at::kByte, like); sft = empty({scales}, at::kByte, like); }
  }
  static void* at_(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
};
Quantized quantize_mx(const Tensor& x, bool rowwise, bool colwise) {
  reachable({&x});
  NNB_ASSERT(x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.stride(1) == 1, "quantize_mx takes bf16 rows");
  const int64_t R = x.size(0), C = x.size(1);
  Quantized o(R, C, rowwise, colwise, x);
  launched(nnb_mxfp8_quantize_sw(x.data_ptr(), x.stride(0), o.at_(o.q), C, o.at_(o.sf), o.at_(o.qt), R, o.at_(o.sft), (int)R, (int)C, stream()), "nnb_mxfp8_quantize_sw");
  return o;
}
// of the activation silu(gate) * up of a packed projection, and of the projection's gradient for a gradient of the activation
Quantized swiglu_mx(const Tensor& gu, bool rowwise, bool colwise) {
  reachable({&gu});
  NNB_ASSERT(gu.dim() == 2 && gu.scalar_type() == at::kBFloat16 && gu.stride(1) == 1 && gu.size(1) % 2 == 0, "swiglu_mx takes bf16 rows");
  const int64_t R = gu.size(0), F = gu.size(1) / 2;
  Quantized o(R, F, rowwise, colwise, gu);
  launched(nnb_mxfp8_swiglu(gu.data_ptr(), gu.stride(0), o.at_(o.q), F, o.at_(o.sf), o.at_(o.qt), R, o.at_(o.sft), (int)R, (int)F, stream()), "nnb_mxfp8_swiglu");
  return o;
}
Quantized swiglu_bwd_mx(const Tensor& dact, const Tensor& gu, bool rowwise, bool colwise) {
  reachable({&dact, &gu});
  NNB_ASSERT(gu.dim() == 2 && gu.scalar_type() == at::kBFloat16 && gu.stride(1) == 1 && dact.dim() == 2 && dact.scalar_type() == at::kBFloat16 && dact.stride(1) == 1 &&
             dact.size(0) == gu.size(0) && 2 * dact.size(1) == gu.size(1), "swiglu_bwd_mx takes bf16 rows that fit");
  const int64_t R = gu.size(0), F = dact.size(1);
  Quantized o(R, 2 * F, rowwise, colwise, gu);
  launched(nnb_mxfp8_swiglu_bwd(dact.data_ptr(), dact.stride(0), gu.data_ptr(), gu.stride(0), o.at_(o.q), 2 * F, o.at_(o.sf), o.at_(o.qt), R, o.at_(o.sft), (int)R, (int)F, stream()),
           "nnb_mxfp8_swiglu_bwd");
  return o;
}
Tensor gemm_mxfp8(const Tensor& aq, const Tensor& asf, const Tensor& bq, const Tensor& bsf, const optional<Tensor>& out_, at::ScalarType out_dtype, bool accumulate, int k_splits) {
  reachable({&aq, &asf, &bq, &bsf});
  if (out_ && out_->defined()) reachable({&aq, &*out_});
  const int64_t M = aq.size(0), K = aq.size(1), N = bq.size(0);
  NNB_ASSERT(bq.size(1) == K && aq.scalar_type() == at::kByte && bq.scalar_type() == at::kByte, "gemm_mxfp8: operands do not fit");
  const bool given = out_.has_value() && out_->defined();
  NNB_ASSERT(given || !accumulate, "gemm_mxfp8: accumulate needs an output");
  Tensor out = given ? *out_ : empty({M, N}, out_dtype, aq);
  NNB_ASSERT(out.dim() == 2 && out.size(0) == M && out.size(1) == N && out.stride(1) == 1 && (out.scalar_type() == at::kBFloat16 || out.scalar_type() == at::kFloat), "gemm_mxfp8: the output does not fit");
  launched(nnb_gemm_mxfp8(aq.data_ptr(), asf.data_ptr(), bq.data_ptr(), bsf.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, aq.stride(0), bq.stride(0), out.stride(0),
                          out.scalar_type() == at::kFloat, accumulate, k_splits, 0, status_of(aq), stream()), "nnb_gemm_mxfp8");
  return out;
}

// ------------------------------------------------------------------------------------------------ plain calls
PyObject* g_parameter_type = nullptr;

bool plain_tensor(const Tensor& t) {
  static const uint64_t allowed = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutocastCUDA}).raw_repr();
  return t.defined() && t.is_cuda() && (t.key_set().raw_repr() & ~allowed) == 0;
}
bool plain_arg(py::handle h) {
  if (Py_TYPE(h.ptr()) != (PyTypeObject*)THPVariableClass && (PyObject*)Py_TYPE(h.ptr()) != g_parameter_type) return false;
  const Tensor& t = THPVariable_Unpack(h.ptr());
  return plain_tensor(t) && !t._fw_grad(/*level=*/0).defined();
}
bool plain_thread() {  // no transform, tracer, mode or functional layer is active
  static const uint64_t allowed = (c10::default_included_set | c10::autocast_dispatch_keyset).raw_repr();
  return (c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~allowed) == 0 && !c10::impl::dispatch_mode_enabled() && !at::impl::torch_function_mode_enabled();
}
template <typename... H>
bool plain(H... h) { return plain_thread() && (plain_arg(h) && ...); }

py::object attribute(py::handle obj, const char* name) {  // None where it is missing
  PyObject* r = PyObject_GetAttrString(obj.ptr(), name);
  if (r == nullptr) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw py::error_already_set();
    PyErr_Clear();
    return py::none();
  }
  return py::reinterpret_steal<py::object>(r);
}
Tensor tensor_or_undefined(const py::object& o) { return THPVariable_Check(o.ptr()) ? THPVariable_Unpack(o.ptr()) : Tensor(); }

at::ScalarType compute_dtype() {
  if (at::autocast::is_autocast_enabled(at::kCUDA)) {
    const at::ScalarType dt = at::autocast::get_autocast_dtype(at::kCUDA);
    if (code16(dt) > 0) return dt;
  }
  return at::kBFloat16;
}

// A weight as an operator sees it: its 16-bit copy when the engine keeps one, and whether it belongs to the engine at all.
struct Weight {
  Tensor shadow;
  bool engine;
  Weight(py::handle w) : shadow(tensor_or_undefined(attribute(w, "_shadow"))) { engine = shadow.defined() || !attribute(w, "_main_grad").is_none(); }
  bool has(at::ScalarType dt) const { return shadow.defined() && shadow.scalar_type() == dt; }
  Tensor in(const Tensor& w, at::ScalarType dt) const { return has(dt) ? shadow : as_dtype(w.detach(), dt); }
};
// x2 w^T for a weight without a 16-bit copy
Tensor weight_product(const Tensor& x2, const Tensor& weight) {
  const Tensor w = weight.detach(), y = gemm_f32w(x2, w);
  return y.defined() ? y : gemm_nt(x2, as_dtype(w, x2.scalar_type()));
}

// dW of an engine weight goes into the flat gradient buffer, and the strategy hears of it, in every backward pass through a weight that is
// trained, also one that asks for other gradients only: as with the Python autograd functions, whose needs_input_grad is fixed in the
// forward pass (needs_input_grad here is what the running pass asks for). Everything is read from the weight's
// Python object when the backward runs (a saved-tensor hook may have put another tensor in its place).
struct MainGrad {
  Tensor main;
  py::object cb;
  bool tied = false;
  explicit MainGrad(const Tensor& weight) {
    py::gil_scoped_acquire gil;
    py::object w = py::reinterpret_steal<py::object>(THPVariable_Wrap(weight));
    main = tensor_or_undefined(attribute(w, "_main_grad"));
    if (main.defined() && main.scalar_type() != at::kFloat) main = Tensor();
    if (main.defined()) {
      cb = attribute(w, "_grad_ready_cb");
      if (cb.is_none()) cb.release().dec_ref();
      else tied = py::bool_(attribute(w, "_tied_embedding"));
    }
  }
  ~MainGrad() {
    if (cb) {
      py::gil_scoped_acquire gil;
      cb.release().dec_ref();
    }
  }
  void ready(const Tensor& weight) {
    if (!cb) return;
    py::gil_scoped_acquire gil;
    cb(py::reinterpret_steal<py::object>(THPVariable_Wrap(weight)), true);
  }
};

// dy2^T @ x2 into the flat buffer (undefined result) or as a gradient of the weight's dtype
Tensor weight_gradient(const Tensor& dy2, const Tensor& x2, const Tensor& weight, bool engine) {
  if (engine) {
    MainGrad mg(weight);
    if (mg.main.defined()) {
      gemm(dy2, x2, true, true, mg.main, std::nullopt, true, 0, 0, 0);
      if (!mg.tied) mg.ready(weight);  // a tied head weight is complete only after the embedding backward
      return Tensor();
    }
  }
  return as_dtype(gemm(dy2, x2, true, true, std::nullopt, at::kFloat, false, 0, 0, 0), weight.scalar_type());
}

// Must a node of a registered operator go through the dispatcher? (create_graph=True, or a gradient that is not plain)
bool through_dispatcher(const Tensor& a, const Tensor& b = Tensor()) {
  return at::GradMode::is_enabled() || !plain_thread() || !plain_tensor(a) || (b.defined() && !plain_tensor(b));
}
void engine_gradient(const Tensor& g) { TORCH_CHECK(plain_tensor(g), "this operator's backward takes plain CUDA gradients only"); }

c10::OperatorHandle registered(const char* name) { return c10::Dispatcher::singleton().findSchemaOrThrow(name, ""); }
Tensor call_matmul_nt(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, bool f32) {
  static auto op = registered("nanonemo_b200::matmul_nt").typed<Tensor(const Tensor&, const Tensor&, bool, bool, bool)>();
  return op.call(a, b, a_mn, b_mn, f32);
}

// An output that is a reshaped new tensor and no view of anything, as far as autograd can see (in-place use stays open).
template <typename F>
Tensor fresh(F make) {
  at::AutoDispatchBelowADInplaceOrView guard;
  return make();
}
std::vector<int64_t> with_last(at::IntArrayRef sizes, int64_t last) {
  std::vector<int64_t> s(sizes.begin(), sizes.end());
  s.back() = last;
  return s;
}

// ------------------------------------------------------------------------------------------------ operators
// x: any shape and dtype where the engine's weight is (nothing differentiates its gradients); otherwise the 16-bit rows, made before the
// node, so that its saved tensor leads back to the caller's input under create_graph. w16: none where the weight has no 16-bit copy.
struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const optional<Tensor>& w16, bool engine, const std::vector<int64_t>& y_sizes) {
    const Tensor x2 = engine ? rowmajor2d(as_dtype(rows2d(x), w16->scalar_type())) : x;
    Tensor y = w16 ? gemm_nt(x2, *w16) : weight_product(x2, weight);
    ctx->save_for_backward({x2, weight});
    if (engine) ctx->saved_data["w16"] = *w16;
    ctx->saved_data["x_sizes"] = x.sizes().vec();
    ctx->saved_data["x_dtype"] = (int64_t)x.scalar_type();
    ctx->saved_data["engine"] = engine;
    ctx->saved_data["trained"] = weight.requires_grad();
    return fresh([&] { return y.view(y_sizes); });
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &weight = saved[1];
    const bool engine = ctx->saved_data["engine"].toBool();
    const auto x_sizes = ctx->saved_data["x_sizes"].toIntVector();
    const auto x_dtype = (at::ScalarType)ctx->saved_data["x_dtype"].toInt();
    const bool need_dx = ctx->needs_input_grad(0), need_dw = engine ? ctx->saved_data["trained"].toBool() : ctx->needs_input_grad(1);
    Tensor dy2 = as_dtype(rows2d(grads[0]), x2.scalar_type()), dx, dw;
    if (!engine && through_dispatcher(grads[0])) {
      dy2 = dy2.contiguous();  // (both, as the registered formula has it: what it refuses to differentiate further is refused here too)
      dx = call_matmul_nt(dy2, as_dtype(weight, x2.scalar_type()), false, true, false);
      dw = as_dtype(call_matmul_nt(dy2, x2, true, true, true), weight.scalar_type());
    } else {
      if (engine) engine_gradient(grads[0]);
      dy2 = rowmajor2d(dy2);
      if (need_dx && !engine) dx = gemm_f32w_dgrad(dy2, weight.detach());
      if (need_dx && !dx.defined()) dx = gemm_nt(dy2, engine ? ctx->saved_data["w16"].toTensor() : as_dtype(weight, x2.scalar_type()), true);
      if (need_dw) dw = weight_gradient(dy2, x2, weight, engine);
    }
    if (dx.defined()) dx = as_dtype(dx.view(x_sizes), x_dtype);
    return {dx, dw, Tensor(), Tensor(), Tensor()};
  }
};

py::object linear(py::handle x_, py::handle weight_) {
  if (!plain(x_, weight_)) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  const Tensor x = THPVariable_Unpack(x_.ptr()), weight = THPVariable_Unpack(weight_.ptr());
  const Weight w(weight_);
  Tensor y;
  {
    py::gil_scoped_release nogil;
    const at::ScalarType dt = compute_dtype();
    const optional<Tensor> w16 = w.engine ? optional<Tensor>(w.in(weight, dt)) : std::nullopt;
    y = LinearFn::apply(w.engine ? x : rowmajor2d(as_dtype(rows2d(x), dt)), weight, w16, w.engine, with_last(x.sizes(), weight.size(0)));
  }
  return py::cast(y);
}

struct AddRMSNormFn : torch::autograd::Function<AddRMSNormFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& delta, const Tensor& weight, double eps, int64_t y_dt, bool engine) {
    auto [y, h, rstd] = rms_fwd(x, delta, weight, eps, (at::ScalarType)y_dt);
    const bool has_delta = delta.has_value();
    y = fresh([&, y2 = y] { return y2.view(x.sizes()); });
    if (has_delta) h = fresh([&, h2 = h] { return h2.view(x.sizes()); });
    else h = engine ? h.view(x.sizes()) : x.clone(at::MemoryFormat::Contiguous);
    ctx->save_for_backward({h, rstd, weight});
    ctx->saved_data["has_delta"] = has_delta;
    ctx->saved_data["delta"] = has_delta ? (int64_t)delta->scalar_type() : (int64_t)y_dt;
    ctx->saved_data["y"] = y_dt;
    ctx->saved_data["engine"] = engine;
    ctx->set_materialize_grads(false);
    return {y, h};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &rstd = saved[1], &weight = saved[2];
    const bool has_delta = ctx->saved_data["has_delta"].toBool(), engine = ctx->saved_data["engine"].toBool();
    const auto delta_dt = (at::ScalarType)ctx->saved_data["delta"].toInt();
    Tensor dy = grads[0], dh = grads[1];
    if (!dy.defined() && !dh.defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    if (!dy.defined()) dy = at::zeros(h.sizes(), h.options().dtype((at::ScalarType)ctx->saved_data["y"].toInt()));
    Tensor dx, ddelta, dw;
    if (!engine && through_dispatcher(dy, dh)) {
      static auto op = registered("nanonemo_b200::add_rms_norm_bwd").typed<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const optional<Tensor>&, const Tensor&, const Tensor&, const Tensor&, int64_t)>();
      std::tie(dx, ddelta, dw) = op.call(dy.contiguous(), dh.defined() ? optional<Tensor>(dh.contiguous()) : std::nullopt, h, rstd, weight, code_of(delta_dt));
      dw = as_dtype(dw, weight.scalar_type());
    } else if (engine) {
      engine_gradient(dy);
      if (dh.defined()) engine_gradient(dh);
      const optional<at::ScalarType> dd = has_delta ? optional<at::ScalarType>(delta_dt) : std::nullopt;
      MainGrad mg(weight);
      std::tie(dx, ddelta, dw) = rms_bwd(dy, h, rstd, weight, dh, dd, mg.main, mg.main.defined());
      if (mg.main.defined()) {
        mg.ready(weight);
        dw = Tensor();
      } else {
        dw = as_dtype(dw, weight.scalar_type());
      }
    } else {
      std::tie(dx, ddelta, dw) = rms_bwd(dy, h, rstd, weight, dh, has_delta ? optional<at::ScalarType>(delta_dt) : std::nullopt, std::nullopt, false);
      if (ddelta.defined() && ddelta.is_same(dx)) ddelta = dx.clone();
      dw = as_dtype(dw, weight.scalar_type());
    }
    return {dx, has_delta ? ddelta : Tensor(), dw, Tensor(), Tensor(), Tensor()};
  }
};

py::object add_rms_norm(py::handle x_, py::handle delta_, py::handle weight_, double eps) {
  const bool has_delta = !delta_.is_none();
  if (!plain(x_, weight_) || (has_delta && !plain_arg(delta_))) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  Tensor x = THPVariable_Unpack(x_.ptr()), delta = has_delta ? THPVariable_Unpack(delta_.ptr()) : Tensor();
  const Tensor weight = THPVariable_Unpack(weight_.ptr());
  const bool engine = !attribute(weight_, "_main_grad").is_none();
  const at::ScalarType y_dt = at::autocast::is_autocast_enabled(at::kCUDA) ? at::autocast::get_autocast_dtype(at::kCUDA) : has_delta ? delta.scalar_type() : x.scalar_type();
  if (code_of(y_dt) < 0) return py::reinterpret_borrow<py::object>(Py_NotImplemented);  // refused there
  variable_list out;
  {
    py::gil_scoped_release nogil;
    if (has_delta) delta = as_dtype(delta, y_dt);
    if (x.scalar_type() != at::kFloat && x.scalar_type() != y_dt) x = x.to(at::kFloat);
    out = AddRMSNormFn::apply(x, has_delta ? optional<Tensor>(delta) : std::nullopt, weight, eps, (int64_t)y_dt, engine);
  }
  return py::make_tuple(out[0], out[1]);
}

Tensor bthd(const Tensor& t_) {  // (B, heads, T, hd) -> the kernel's [B, T, heads, hd] view; copied only when strides or alignment rule it out
  const Tensor t = t_.transpose(1, 2);
  const bool ok = t.stride(-1) == 1 && (t.stride(0) * 2) % 16 == 0 && (t.stride(1) * 2) % 16 == 0 && (t.stride(2) * 2) % 16 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  return ok ? t : t.contiguous();
}

struct FlashAttnFn : torch::autograd::Function<FlashAttnFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v) {
    const Tensor qt = bthd(q), kt = bthd(k), vt = bthd(v), o = empty(qt.sizes(), q.scalar_type(), q);
    const Tensor lse = flash_fwd(qt, kt, vt, o, 1.0 / std::sqrt((double)qt.size(3)));
    const Tensor out = fresh([&] { return o.transpose(1, 2); });
    ctx->save_for_backward({q, k, v, out, lse});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor dout = as_dtype(grads[0], s[0].scalar_type());
    if (through_dispatcher(grads[0])) {
      static auto op = registered("nanonemo_b200::flash_attn_bwd").typed<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&)>();
      auto [dq, dk, dv] = op.call(dout, s[0], s[1], s[2], s[3], s[4]);
      return {dq, dk, dv};
    }
    const Tensor qt = bthd(s[0]), kt = bthd(s[1]), vt = bthd(s[2]), ot = bthd(s[3]), dt = bthd(dout);
    const Tensor dq = empty(qt.sizes(), qt.scalar_type(), qt), dk = empty(kt.sizes(), qt.scalar_type(), qt), dv = empty(vt.sizes(), qt.scalar_type(), qt);
    flash_bwd(qt, kt, vt, ot, s[4], dt, dq, dk, dv, 1.0 / std::sqrt((double)qt.size(3)), std::nullopt, std::nullopt, false);
    return {dq.transpose(1, 2), dk.transpose(1, 2), dv.transpose(1, 2)};
  }
};

py::object flash_attn(py::handle q_, py::handle k_, py::handle v_) {
  if (!plain(q_, k_, v_)) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  const Tensor q = THPVariable_Unpack(q_.ptr()), k = THPVariable_Unpack(k_.ptr()), v = THPVariable_Unpack(v_.ptr());
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  Tensor o;
  {
    py::gil_scoped_release nogil;
    const at::ScalarType dt = code16(q.scalar_type()) > 0 ? q.scalar_type() : at::kBFloat16;  // fp32 goes through bf16 and back
    o = as_dtype(FlashAttnFn::apply(as_dtype(q, dt), as_dtype(k, dt), as_dtype(v, dt)), q.scalar_type());
  }
  return py::cast(o);
}

struct Heads {
  Tensor q, k, v;
  Heads(const Tensor& qkv, int64_t B, int64_t T, int64_t H, int64_t KVH, int64_t hd)  // qkv: [B T, (H + 2 KVH) hd] contiguous
      : q(part(qkv, B, T, 0, H, hd)), k(part(qkv, B, T, H, KVH, hd)), v(part(qkv, B, T, H + KVH, KVH, hd)) {}
  static Tensor part(const Tensor& t, int64_t B, int64_t T, int64_t first, int64_t heads, int64_t hd) {
    const int64_t row = t.stride(0);
    return t.as_strided({B, T, heads, hd}, {T * row, row, hd, 1}, t.storage_offset() + first * hd);
  }
};

// Engine weights, or calls without gradients: projection + RoPE (GEMM epilogue) + attention as one node
struct QKVRopeAttentionFn : torch::autograd::Function<QKVRopeAttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& w16, const Tensor& cos, const Tensor& sin, int64_t H, int64_t KVH, int64_t hd) {
    const int64_t B = x.size(0), T = x.size(1);
    const at::ScalarType dt = w16.scalar_type();
    const Tensor x2 = rowmajor2d(as_dtype(rows2d(x), dt));
    Tensor qkv = gemm_rope(x2, w16, cos, sin, T, (H + KVH) * hd, hd);
    if (!qkv.defined()) {
      qkv = gemm_nt(x2, w16);
      rope_packed(qkv, qkv, cos, sin, T, H + KVH, hd, 0, 1.0);  // rotates Q and K in place, V untouched
    }
    const Heads p(qkv, B, T, H, KVH, hd);
    const Tensor o = empty({B, T, H, hd}, dt, x);
    const Tensor lse = flash_fwd(p.q, p.k, p.v, o, 1.0 / std::sqrt((double)hd));
    ctx->save_for_backward({x2, weight, qkv, o, lse, cos, sin});
    ctx->saved_data["w16"] = w16;
    ctx->saved_data["meta"] = std::vector<int64_t>{B, T, H, KVH, hd, (int64_t)x.scalar_type()};
    ctx->saved_data["x_sizes"] = x.sizes().vec();
    ctx->saved_data["trained"] = weight.requires_grad();
    return fresh([&] { return o.view({B, T, H * hd}); });
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &weight = s[1], &qkv = s[2], &o = s[3], &lse = s[4], &cos = s[5], &sin = s[6];
    const auto m = ctx->saved_data["meta"].toIntVector();
    const int64_t B = m[0], T = m[1], H = m[2], KVH = m[3], hd = m[4];
    engine_gradient(grads[0]);
    Tensor dout = grads[0].reshape({B, T, H, hd});
    if (dout.stride(-1) != 1 || dout.scalar_type() != qkv.scalar_type()) dout = dout.to(qkv.scalar_type()).contiguous();
    const Tensor dqkv = at::empty_like(qkv);
    const Heads p(qkv, B, T, H, KVH, hd), d(dqkv, B, T, H, KVH, hd);
    const double scale = 1.0 / std::sqrt((double)hd);
    const char* route = std::getenv("NANONEMO_FLASH_BWD");
    if (hd == 64 && !(route && route[0] == 't')) {  // this backward kernel un-rotates dQ and dK itself
      flash_bwd(p.q, p.k, p.v, o, lse, dout, d.q, d.k, d.v, scale, cos, sin, false);
    } else {
      flash_bwd(p.q, p.k, p.v, o, lse, dout, d.q, d.k, d.v, scale, std::nullopt, std::nullopt, false);
      rope_packed(dqkv, dqkv, cos, sin, T, H + KVH, hd, 0, -1.0);
    }
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) dx = as_dtype(gemm_nt(dqkv, ctx->saved_data["w16"].toTensor(), true).view(ctx->saved_data["x_sizes"].toIntVector()), (at::ScalarType)m[5]);
    if (ctx->saved_data["trained"].toBool()) dw = weight_gradient(dqkv, x2, weight, true);
    return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

bool wants_gradient(std::initializer_list<const Tensor*> ts) {
  if (at::GradMode::is_enabled())
    for (const Tensor* t : ts)
      if (t->requires_grad()) return true;
  return false;
}

Tensor rope_table(const Tensor& t, int64_t T) { return as_dtype(t.slice(0, 0, T), at::kFloat).contiguous(); }

// Projection, RoPE and attention where nobody asks for a gradient
Tensor attention_rows(const Tensor& x, const Tensor& weight, const Weight& w, const Tensor& cos, const Tensor& sin, int64_t H, int64_t KVH, int64_t hd) {
  const int64_t B = x.size(0), T = x.size(1), cols = (H + KVH) * hd;
  const at::ScalarType dt = compute_dtype();
  const Tensor x2 = rowmajor2d(as_dtype(rows2d(x), dt));
  Tensor qkv = w.engine ? Tensor() : gemm_f32w_rope(x2, weight.detach(), cos, sin, T, cols, hd);
  if (!qkv.defined()) {
    const Tensor w16 = w.in(weight, dt);
    qkv = gemm_rope(x2, w16, cos, sin, T, cols, hd);
    if (!qkv.defined()) {
      qkv = gemm_nt(x2, w16);
      rope_packed(qkv, qkv, cos, sin, T, H + KVH, hd, 0, 1.0);
    }
  }
  const Heads p(qkv, B, T, H, KVH, hd);
  const Tensor o = empty({B, T, H, hd}, dt, x);
  flash_fwd(p.q, p.k, p.v, o, 1.0 / std::sqrt((double)hd));
  return o.view({B, T, H * hd});
}

py::object qkv_rope_attention(py::handle x_, py::handle weight_, py::handle cos_, py::handle sin_, int64_t H, int64_t KVH, int64_t hd) {
  if (!plain(x_, weight_, cos_, sin_)) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  const Tensor x = THPVariable_Unpack(x_.ptr()), weight = THPVariable_Unpack(weight_.ptr());
  const Weight w(weight_);
  if (x.dim() != 3 || !attribute(weight_, "_gather_in_gemm").is_none() || (!w.engine && wants_gradient({&x, &weight}))) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  Tensor cos = THPVariable_Unpack(cos_.ptr()), sin = THPVariable_Unpack(sin_.ptr()), y;
  {
    py::gil_scoped_release nogil;
    cos = rope_table(cos, x.size(1));
    sin = rope_table(sin, x.size(1));
    y = wants_gradient({&x, &weight}) ? QKVRopeAttentionFn::apply(x, weight, w.in(weight, compute_dtype()), cos, sin, H, KVH, hd)
                                      : attention_rows(x, weight, w, cos, sin, H, KVH, hd);
  }
  return py::cast(y);
}

// (gu, act) of the gate and up projection, gu only where it is kept or has to be made: in one launch, or in two where the fused kernel does not serve
std::pair<Tensor, Tensor> gate_up(const Tensor& x2, const Tensor& w16, bool keep) {
  auto r = gemm_swiglu(x2, w16, keep);
  if (r.second.defined()) return r;
  const int64_t F = w16.size(0) / 2;
  r = {gemm_nt(x2, w16), empty({x2.size(0), F}, w16.scalar_type(), x2)};
  swiglu_fwd(r.first.narrow(1, 0, F), r.first.narrow(1, F, F), r.second);
  return r;
}

// The SwiGLU feed-forward as one node (engine weights)
struct MLPFn : torch::autograd::Function<MLPFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_gu, const Tensor& w_down, const Tensor& gu16, const Tensor& down16) {
    const Tensor x2 = rowmajor2d(as_dtype(rows2d(x), gu16.scalar_type()));
    auto [gu, act] = gate_up(x2, gu16, true);
    Tensor y = gemm_nt(act, down16);
    ctx->save_for_backward({x2, w_gu, w_down, gu, act});
    ctx->saved_data["gu16"] = gu16;
    ctx->saved_data["down16"] = down16;
    ctx->saved_data["x_sizes"] = x.sizes().vec();
    ctx->saved_data["x_dtype"] = (int64_t)x.scalar_type();
    ctx->saved_data["trained"] = std::vector<int64_t>{w_gu.requires_grad(), w_down.requires_grad()};
    return fresh([&] { return y.view(with_last(x.sizes(), w_down.size(0))); });
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w_gu = s[1], &w_down = s[2], &gu = s[3], &act = s[4];
    const Tensor gu16 = ctx->saved_data["gu16"].toTensor(), down16 = ctx->saved_data["down16"].toTensor();
    engine_gradient(grads[0]);
    const int64_t F = gu.size(1) / 2;
    const Tensor dy2 = rowmajor2d(as_dtype(rows2d(grads[0]), gu.scalar_type()));
    Tensor dgu = gemm_swiglu_bwd(dy2, down16, gu);
    if (!dgu.defined()) {
      const Tensor dact = gemm_nt(dy2, down16, true);
      dgu = at::empty_like(gu);
      swiglu_bwd(dact, gu.narrow(1, 0, F), gu.narrow(1, F, F), dgu.narrow(1, 0, F), dgu.narrow(1, F, F));
    }
    const auto trained = ctx->saved_data["trained"].toIntVector();
    Tensor dx, dw_gu, dw_down;
    if (trained[1]) dw_down = weight_gradient(dy2, act, w_down, true);
    if (ctx->needs_input_grad(0)) dx = as_dtype(gemm_nt(dgu, gu16, true).view(ctx->saved_data["x_sizes"].toIntVector()), (at::ScalarType)ctx->saved_data["x_dtype"].toInt());
    if (trained[0]) dw_gu = weight_gradient(dgu, x2, w_gu, true);
    return {dx, dw_gu, dw_down, Tensor(), Tensor()};
  }
};

// The same where nobody will ask for the projection: where one launch serves, only the activation leaves it
Tensor mlp_rows(const Tensor& x, const Tensor& w_gu, const Weight& gu, const Tensor& w_down, const Weight& down) {
  const at::ScalarType dt = compute_dtype();
  const Tensor x2 = rowmajor2d(as_dtype(rows2d(x), dt));
  Tensor act = gu.has(dt) ? Tensor() : gemm_f32w_swiglu(x2, w_gu.detach());
  if (!act.defined()) act = gate_up(x2, gu.in(w_gu, dt), false).second;
  return (down.has(dt) ? gemm_nt(act, down.shadow) : weight_product(act, w_down)).view(with_last(x.sizes(), w_down.size(0)));
}

py::object mlp_swiglu(py::handle x_, py::handle gu_, py::handle down_) {
  if (!plain(x_, gu_, down_)) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  const Tensor x = THPVariable_Unpack(x_.ptr()), w_gu = THPVariable_Unpack(gu_.ptr()), w_down = THPVariable_Unpack(down_.ptr());
  const Weight gu(gu_), down(down_);
  const bool grad = wants_gradient({&x, &w_gu, &w_down});
  if (grad && !(gu.engine && down.engine && attribute(gu_, "_gather_in_gemm").is_none())) return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  Tensor y;
  {
    py::gil_scoped_release nogil;
    const at::ScalarType dt = compute_dtype();
    y = grad ? MLPFn::apply(x, w_gu, w_down, gu.in(w_gu, dt), down.in(w_down, dt)) : mlp_rows(x, w_gu, gu, w_down, down);
  }
  return py::cast(y);
}

// The block of few rows with fp32 weights and an fp32 residual stream (scoring a short text with a loaded model): seven launches into one
// workspace, as raw pointers; 12 tensors, their views and the checks of each operator took 38 us a block beside 17 for the launches. False,
// with nothing launched, where it does not serve.
struct BlockShape { int64_t B, T, D, H, KVH, hd, F; };
bool block_of_few_rows(const Tensor& x, const Tensor& delta, const Tensor& norm1, double eps1, const Tensor& wqkv, const Tensor& wo, const Tensor& norm2, double eps2, const Tensor& w_gu,
                       const Tensor& w_down, const Tensor& cos, const Tensor& sin, const BlockShape& s, at::ScalarType dt, Tensor& h_out, Tensor& y_out) {
  const int code = code16(dt);
  const int64_t M = s.B * s.T, Q = (s.H + 2 * s.KVH) * s.hd, A = s.H * s.hd;
  auto fits = [](const Tensor& t, at::ScalarType type, at::IntArrayRef sizes) {
    return t.scalar_type() == type && t.sizes() == sizes && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  };
  auto serves = [&](int64_t n, int64_t k, int kind) { return f32w_serves(M, n, k, kind); };
  auto table = [&](const Tensor& t) {
    return t.dim() == 2 && t.scalar_type() == at::kFloat && t.is_contiguous() && t.size(0) >= s.T && t.size(1) == s.hd / 2 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  };
  if (code < 0 || M < 1 || M > 4096 || s.D % 8 || s.D > 2048 || s.F % 16 || (s.hd != 64 && s.hd != 128) || s.KVH < 1 || s.H % s.KVH || !fits(x, at::kFloat, {s.B, s.T, s.D}) ||
      (delta.defined() && !fits(delta, dt, {s.B, s.T, s.D})) || !fits(norm1, at::kFloat, {s.D}) || !fits(norm2, at::kFloat, {s.D}) || !fits(wqkv, at::kFloat, {Q, s.D}) ||
      !fits(wo, at::kFloat, {s.D, A}) || !fits(w_gu, at::kFloat, {2 * s.F, s.D}) || !fits(w_down, at::kFloat, {s.D, s.F}) || !table(cos) || !table(sin) || !serves(Q, s.D, 0) ||
      !serves(s.D, A, 0) || !serves(s.F, s.D, 1) || !serves(s.D, s.F, 0))
    return false;
  int64_t bytes = 0;
  auto room = [&](int64_t n) { const int64_t at = bytes; bytes += (n + 255) / 256 * 256; return at; };
  const int64_t at_n = room(M * s.D * 2), at_h = room(M * s.D * 4), at_qkv = room(M * Q * 2), at_o = room(M * A * 2), at_p = room(M * s.D * 2), at_act = room(M * s.F * 2),
                at_rstd = room(M * 4), at_lse = room(M * s.H * 4);
  const Tensor space = empty({bytes}, at::kByte, x);
  char* base = static_cast<char*>(space.data_ptr());
  h_out = empty({s.B, s.T, s.D}, at::kFloat, x);
  y_out = empty({s.B, s.T, s.D}, dt, x);
  void *n = base + at_n, *qkv = base + at_qkv, *o = base + at_o, *p = base + at_p, *act = base + at_act, *rstd = base + at_rstd, *status = status_of(x);
  const void* h = delta.defined() ? base + at_h : x.data_ptr();
  const cudaStream_t st = stream();
  const int m = (int)M, d = (int)s.D, q = (int)Q, a = (int)A, f = (int)s.F;
  const long long row = Q, heads = s.hd;
  char* v = static_cast<char*>(qkv);
  launched(nnb_add_rmsnorm_fwd(x.data_ptr(), delta.defined() ? delta.data_ptr() : nullptr, norm1.data_ptr(), n, const_cast<void*>(h), rstd, m, d, (float)eps1, 0, code, code, st), "nnb_add_rmsnorm_fwd");
  launched(nnb_gemm_rows_rope(n, wqkv.data_ptr(), qkv, cos.data_ptr(), sin.data_ptr(), m, q, d, d, d, q, (int)s.T, (int)((s.H + s.KVH) * s.hd), (int)s.hd, code, 1, 16, status, st),
           "nnb_gemm_rows_rope");
  launched(nnb_flash_fwd(v, v + 2 * A, v + 2 * (A + s.KVH * s.hd), o, base + at_lse, (int)s.B, (int)s.T, (int)s.H, (int)s.KVH, (int)s.hd, s.T * row, row, heads, s.T * row, row, heads, s.T * row,
                         row, heads, s.T * A, A, heads, (float)(1.0 / std::sqrt((double)s.hd)), code, status, st), "nnb_flash_fwd");
  launched(nnb_gemm_rows_f32w(o, wo.data_ptr(), p, m, d, a, a, a, d, 0, code, status, st), "nnb_gemm_rows_f32w");
  launched(nnb_add_rmsnorm_fwd(h, p, norm2.data_ptr(), n, h_out.data_ptr(), rstd, m, d, (float)eps2, 0, code, code, st), "nnb_add_rmsnorm_fwd");
  launched(nnb_gemm_rows_f32w_swiglu(n, w_gu.data_ptr(), act, m, f, d, d, d, f, code, status, st), "nnb_gemm_rows_f32w_swiglu");
  launched(nnb_gemm_rows_f32w(act, w_down.data_ptr(), y_out.data_ptr(), m, d, f, f, f, d, 0, code, status, st), "nnb_gemm_rows_f32w");
  return true;
}

// A transformer block where nobody asks for gradients (models/layers.py: Block), as one call: the launches are those of the operators it
// consists of, without the Python between them, which took as long as the kernels of a short text: scoring 201 tokens through 12 blocks
// 1116 us, now 615 (583 of them kernels). (x, delta) -> (x', delta'), delta not yet added to x.
py::object decoder_block(py::handle x_, py::handle delta_, py::handle norm1_, double eps1, py::handle wqkv_, py::handle wo_, py::handle norm2_, double eps2, py::handle gu_, py::handle down_,
                         py::handle cos_, py::handle sin_, int64_t H, int64_t KVH, int64_t hd) {
  const bool has_delta = !delta_.is_none();
  if (at::GradMode::is_enabled() || !plain(x_, norm1_, wqkv_, wo_, norm2_, gu_, down_, cos_, sin_) || (has_delta && !plain_arg(delta_)))
    return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  const Tensor x = THPVariable_Unpack(x_.ptr()), delta = has_delta ? THPVariable_Unpack(delta_.ptr()) : Tensor(), norm1 = THPVariable_Unpack(norm1_.ptr()),
               wqkv = THPVariable_Unpack(wqkv_.ptr()), wo = THPVariable_Unpack(wo_.ptr()), norm2 = THPVariable_Unpack(norm2_.ptr()), w_gu = THPVariable_Unpack(gu_.ptr()),
               w_down = THPVariable_Unpack(down_.ptr()), cos_t = THPVariable_Unpack(cos_.ptr()), sin_t = THPVariable_Unpack(sin_.ptr());
  const Weight qkv(wqkv_), out(wo_), gu(gu_), down(down_);
  const bool amp = at::autocast::is_autocast_enabled(at::kCUDA);
  const at::ScalarType y_dt = amp ? at::autocast::get_autocast_dtype(at::kCUDA) : has_delta ? delta.scalar_type() : x.scalar_type();
  if (x.dim() != 3 || code_of(y_dt) < 0 || !attribute(wqkv_, "_gather_in_gemm").is_none() || !attribute(gu_, "_gather_in_gemm").is_none())
    return py::reinterpret_borrow<py::object>(Py_NotImplemented);
  Tensor h, y;
  {
    py::gil_scoped_release nogil;
    const at::ScalarType dt = compute_dtype();
    const bool done = !(qkv.engine || out.engine || gu.engine || down.engine) && y_dt == dt && w_gu.dim() == 2 &&
                      block_of_few_rows(x, delta, norm1, eps1, wqkv, wo, norm2, eps2, w_gu, w_down, cos_t, sin_t, {x.size(0), x.size(1), x.size(2), H, KVH, hd, w_gu.size(0) / 2}, dt, h, y);
    if (!done) {
      auto norm = [&](const Tensor& r, const Tensor& d, const Tensor& w, double eps) {  // add_rms_norm
        const at::ScalarType to = amp ? y_dt : d.defined() ? d.scalar_type() : r.scalar_type();
        const Tensor rr = r.scalar_type() != at::kFloat && r.scalar_type() != to ? r.to(at::kFloat) : r;
        auto [yy, hh, rstd] = rms_fwd(rr, d.defined() ? optional<Tensor>(as_dtype(d, to)) : std::nullopt, w, eps, to);
        return std::make_pair(yy.view(r.sizes()), hh.view(r.sizes()));
      };
      auto [n1, h1] = norm(x, delta, norm1, eps1);
      const Tensor a = attention_rows(n1, wqkv, qkv, rope_table(cos_t, x.size(1)), rope_table(sin_t, x.size(1)), H, KVH, hd);
      const Tensor a2 = rowmajor2d(as_dtype(rows2d(a), dt)), p = (out.engine ? gemm_nt(a2, out.in(wo, dt)) : weight_product(a2, wo)).view(with_last(a.sizes(), wo.size(0)));
      auto [n2, h2] = norm(h1, p, norm2, eps2);
      h = h2;
      y = mlp_rows(n2, w_gu, gu, w_down, down);
    }
  }
  return py::make_tuple(h, y);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const AssertionFailed& e) {
      PyErr_SetString(PyExc_AssertionError, e.what());
    } catch (const WrongType& e) {
      PyErr_SetString(PyExc_TypeError, e.what());
    }
  });
  g_parameter_type = py::object(py::module_::import("torch.nn.parameter").attr("Parameter")).release().ptr();  // (held for good)
  const auto nogil = py::call_guard<py::gil_scoped_release>();
  m.def("launches", [] { return g_launches.load(); });
  m.def("status_tensor", &status_tensor, nogil);
  m.def("status_tensors", [] {
    std::lock_guard<std::mutex> lock(g_status_mutex);
    std::vector<Tensor> v;
    for (auto& e : status_map())
      if (e.second.defined()) v.push_back(e.second);
    return v;
  });
  auto opt = [](const Tensor& t) { return t.defined() ? optional<Tensor>(t) : std::nullopt; };
  m.def("gemm", &gemm, nogil);
  m.def("gemm_swiglu", [](const Tensor& x, const Tensor& w) -> optional<std::pair<Tensor, Tensor>> {
    auto r = gemm_swiglu(x, w, true);
    return r.second.defined() ? optional<std::pair<Tensor, Tensor>>(r) : std::nullopt;
  }, nogil);
  m.def("gemm_swiglu_act", [opt](const Tensor& x, const Tensor& w) { return opt(gemm_swiglu(x, w, false).second); }, nogil);
  m.def("gemm_swiglu_bwd", [opt](const Tensor& dy, const Tensor& w, const Tensor& gu) { return opt(gemm_swiglu_bwd(dy, w, gu)); }, nogil);
  m.def("gemm_rope", [opt](const Tensor& x, const Tensor& w, const Tensor& c, const Tensor& s, int64_t t, int64_t cols, int64_t hd) { return opt(gemm_rope(x, w, c, s, t, cols, hd)); }, nogil);
  m.def("rope_packed", &rope_packed, nogil);
  m.def("swiglu_fwd", &swiglu_fwd, nogil);
  m.def("swiglu_bwd", &swiglu_bwd, nogil);
  m.def("rms_fwd", [](const Tensor& x, const optional<Tensor>& d, const Tensor& w, double eps, at::ScalarType y) {
    auto [yy, h, r] = rms_fwd(x, d, w, eps, y);
    return std::make_tuple(yy.view(x.sizes()), h.view(x.sizes()), r);
  }, nogil);
  m.def("rms_bwd", [](const Tensor& dy, const Tensor& h, const Tensor& rstd, const Tensor& w, const optional<Tensor>& dres, optional<at::ScalarType> delta, const optional<Tensor>& dw_out,
                      bool accumulate) {
    auto [dx, dd, dw] = rms_bwd(dy, h, rstd, w, dres, delta, dw_out, accumulate);
    return std::make_tuple(dx, dd.defined() ? optional<Tensor>(dd) : std::nullopt, dw);
  }, nogil);
  m.def("flash_fwd", &flash_fwd, nogil);
  m.def("flash_bwd", &flash_bwd, nogil);
  auto four = [opt](const Quantized& o) { return std::make_tuple(opt(o.q), opt(o.sf), opt(o.qt), opt(o.sft)); };
  m.def("quantize_mx", [four](const Tensor& x, bool r, bool c) { return four(quantize_mx(x, r, c)); }, nogil);
  m.def("swiglu_mx", [four](const Tensor& gu, bool r, bool c) { return four(swiglu_mx(gu, r, c)); }, nogil);
  m.def("swiglu_bwd_mx", [four](const Tensor& dact, const Tensor& gu, bool r, bool c) { return four(swiglu_bwd_mx(dact, gu, r, c)); }, nogil);
  m.def("gemm_mxfp8", &gemm_mxfp8, nogil);
  m.def("linear", &linear);
  m.def("add_rms_norm", &add_rms_norm);
  m.def("flash_attn", &flash_attn);
  m.def("qkv_rope_attention", &qkv_rope_attention);
  m.def("mlp_swiglu", &mlp_swiglu);
  m.def("decoder_block", &decoder_block);
}

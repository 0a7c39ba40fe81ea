"""tcgen05 GEMM front end (csrc/gemm.cu) and the ``linear`` built on it.

``gemm(a, b, ...)`` computes ``D[M, N] (+)= A[M, K] @ B[N, K]^T`` for 16-bit inputs with fp32
accumulation. Each operand can be given K-major (as ``[rows, K]``) or MN-major (the transposed
storage ``[K, rows]``), which is what lets the three GEMMs of a linear layer run without a
transposed copy of the weight or of any activation:

    fprop  y  = x @ W^T       a = x  [M, K]            b = W  [N, K]
    dgrad  dx = dy @ W        a = dy [M, N_out]        b = W  [N_out, K_in] read as B^T (MN-major)
    wgrad  dW += dy^T @ x     a = dy read as A^T, b = x read as B^T, fp32 out, split-K, reduce-add

``linear_sm100(x, weight)`` is the autograd function: the weight is the fp32 master parameter; the
16-bit copy it multiplies with is ``weight._shadow`` (maintained by the flat parameter store and
rewritten by the fused AdamW kernel) or a cast made on the fly; the weight gradient is accumulated
in fp32 directly into the flat gradient buffer when there is one.
"""

import torch
from torch.autograd.forward_ad import unpack_dual

from nanonemo_b200.ops import _lib

_CODE = {torch.bfloat16: 1, torch.float16: 2}


def status_tensor(device) -> torch.Tensor:
    """The status words of the bounded waits on a device (one tensor per device, owned by the binding)."""
    device = torch.device(device)
    return _lib.native().status_tensor(torch.cuda.current_device() if device.index is None else device.index)


def check_status(device=None):
    """Raise if any GEMM launched so far on `device` gave up on a bounded wait (synchronises)."""
    for t in _lib.native().status_tensors():
        code, role, block, item = t.tolist()
        if code != 0:
            t.zero_()
            raise RuntimeError(f"tcgen05 GEMM gave up waiting: role={role} (1 producer, 2 mma, 3 epilogue) block={block} item={item}")


def _rowmajor2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        t = t.reshape(-1, t.shape[-1])
    if t.stride(1) != 1 or (t.stride(0) * t.element_size()) % 16 or t.data_ptr() % 16:
        t = t.contiguous()
    return t


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False, out: torch.Tensor | None = None,
         out_dtype: torch.dtype | None = None, accumulate: bool = False, k_splits: int = 0, bn: int = 0,
         max_ctas: int = 0) -> torch.Tensor:
    """a: [M, K] (or [K, M] when a_mn); b: [N, K] (or [K, N] when b_mn) -> out [M, N]."""
    return _lib.native().gemm(a, b, a_mn, b_mn, out, out_dtype, accumulate, k_splits, bn, max_ctas)


def _fused_call(name: str, *args) -> bool:
    """Launch a GEMM with a fused epilogue; False when the CTA-pair kernel does not serve the shape (the caller then runs
    the plain GEMM followed by the stand-alone elementwise kernel)."""
    return _lib.call_rc(name, *args) == 0


def gemm_swiglu(x2: torch.Tensor, w_gu: torch.Tensor):
    """x2 [M, K] @ w_gu [2F, K]^T with the SwiGLU activation in the epilogue -> (gu [M, 2F], act [M, F]) or None."""
    return _lib.native().gemm_swiglu(x2, w_gu)


def gemm_swiglu_act(x2: torch.Tensor, w_gu: torch.Tensor):
    """The activation of ``gemm_swiglu`` alone (the projection never reaches memory) -> act [M, F] or None."""
    return _lib.native().gemm_swiglu_act(x2, w_gu)


def gemm_swiglu_bwd(dy2: torch.Tensor, w_down: torch.Tensor, gu: torch.Tensor):
    """SwiGLU backward inside the down projection's input-gradient GEMM: dy2 [M, d] @ w_down [d, F] is the gradient of
    act = silu(gate) * up; the epilogue reads the saved projection gu [M, 2F] and writes d(gate) | d(up) [M, 2F] directly
    (the gradient of act is never stored) -> dgu or None when the CTA-pair kernel does not serve the shape."""
    return _lib.native().gemm_swiglu_bwd(dy2, w_down, gu)


def gemm_rope(x2: torch.Tensor, w: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, t_len: int, rope_cols: int, head_dim: int):
    """x2 [M, K] @ w [N, K]^T with rotate-half RoPE on columns [0, rope_cols) in the epilogue (row m at position
    m % t_len; cos / sin fp32 [t_len, head_dim / 2] contiguous) -> [M, N] or None."""
    return _lib.native().gemm_rope(x2, w, cos, sin, t_len, rope_cols, head_dim)


def gemm_ce_stats(x2: torch.Tensor, w: torch.Tensor, out: torch.Tensor):
    """out [M, N] = x2 @ w^T plus partial softmax statistics (max, sum of exp(x - max)) of every row, two parts per
    256-column tile -> stats fp32 [M, 2 ceil(N / 256), 2] or None."""
    M, K = x2.shape
    N = w.shape[0]
    if M < 256 or N < 128 or N % 64:
        return None
    _lib.reachable(x2, w, out)
    stats = torch.empty((M, 2 * ((N + 255) // 256), 2), dtype=torch.float32, device=x2.device)
    ok = _fused_call("nnb_gemm_ce_stats", _lib.ptr(x2), _lib.ptr(w), _lib.ptr(out), _lib.ptr(stats), _lib.i32(M), _lib.i32(N),
                     _lib.i32(K), _lib.i64(x2.stride(0)), _lib.i64(w.stride(0)), _lib.i64(out.stride(0)), _lib.i32(_CODE[x2.dtype]),
                     _lib.ptr(status_tensor(x2.device)), _lib.vp(_lib.stream_ptr()))
    return stats if ok else None


def gemm_ce_loss(x2: torch.Tensor, w: torch.Tensor, targets: torch.Tensor):
    """The statistics of ``gemm_ce_stats`` without the logits, and the logit of every row's target ->
    (stats fp32 [M, 2 ceil(N / 256), 2], target_logit fp32 [M], unwritten where the target is no column) or None."""
    M, K = x2.shape
    N = w.shape[0]
    if M < 256 or N < 128 or N % 64:
        return None
    _lib.reachable(x2, w, targets)
    stats = torch.empty((M, 2 * ((N + 255) // 256), 2), dtype=torch.float32, device=x2.device)
    target_logit = torch.empty(M, dtype=torch.float32, device=x2.device)
    ok = _fused_call("nnb_gemm_ce_loss", _lib.ptr(x2), _lib.ptr(w), _lib.ptr(targets), _lib.ptr(stats), _lib.ptr(target_logit),
                     _lib.i32(M), _lib.i32(N), _lib.i32(K), _lib.i64(x2.stride(0)), _lib.i64(w.stride(0)), _lib.i32(_CODE[x2.dtype]),
                     _lib.ptr(status_tensor(x2.device)), _lib.vp(_lib.stream_ptr()))
    return (stats, target_logit) if ok else None


def compute_dtype() -> torch.dtype:
    if torch.is_autocast_enabled("cuda"):
        dt = torch.get_autocast_dtype("cuda")
        if dt in _CODE:
            return dt
    return torch.bfloat16


def shadow_of(weight: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    sh = getattr(weight, "_shadow", None)
    if sh is not None and sh.dtype == dtype:
        return sh
    return weight.detach().to(dtype)


def no_backward(*tensors: torch.Tensor) -> bool:
    """True when nothing can ask for a derivative of what is computed from these tensors: an operator may then skip what it would
    keep for its backward. Forward-mode tangents count as asking (the autograd functions refuse them, and go on doing so)."""
    if torch.is_grad_enabled() and any(t.requires_grad for t in tensors):
        return False
    return all(unpack_dual(t).tangent is None for t in tensors)


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight):
        dt = compute_dtype()
        w16 = shadow_of(weight, dt)
        x2 = x.reshape(-1, x.shape[-1])
        if x2.dtype != dt:
            x2 = x2.to(dt)
        x2 = _rowmajor2d(x2)
        y = gemm(x2, w16)
        ctx.save_for_backward(x2, weight)
        ctx.w16 = w16
        ctx.x_dtype = x.dtype
        return y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        dx, dw = linear_backward(dy2, x2, weight, ctx.w16, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        if dx is not None:
            dx = dx.view(*dy.shape[:-1], x2.shape[-1])
            if dx.dtype != ctx.x_dtype:
                dx = dx.to(ctx.x_dtype)
        return dx, dw


def linear_backward(dy2, x2, weight, w16, need_dx: bool, need_dw: bool):
    """The two backward GEMMs of ``y = x2 @ w16^T``: returns (dx [M, K] or None, dW for autograd or None).
    When the weight has a slot in the flat gradient buffer (``weight._main_grad``) the weight gradient is accumulated
    there in fp32 by the GEMM epilogue, the strategy is told the gradient is complete (``_grad_ready_cb``) and the
    returned dW is None."""
    if dy2.dtype != x2.dtype:
        dy2 = dy2.to(x2.dtype)
    dy2 = _rowmajor2d(dy2)
    dx = dw = None
    if need_dx:
        dx = gemm(dy2, w16, b_mn=True)  # [M, K_in]
    if need_dw:
        main = getattr(weight, "_main_grad", None)
        if main is not None and main.dtype == torch.float32:
            gemm(dy2, x2, a_mn=True, b_mn=True, out=main, accumulate=True)
            cb = getattr(weight, "_grad_ready_cb", None)
            if cb is not None and not getattr(weight, "_tied_embedding", False):
                cb(weight, True)  # a tied head weight is complete only after the embedding backward
        else:
            dw = gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=torch.float32).to(weight.dtype)
    return dx, dw


def linear_sm100(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """The trainer's linear. A weight that the engine does not know, too (``linear_impl: mxfp8`` outside fp8): its node takes no part in
    second derivatives, where the native one of such a weight is the registered operators', which refuse them."""
    engine = getattr(weight, "_main_grad", None) is not None or getattr(weight, "_shadow", None) is not None
    y = _lib.operator_call("linear", x, weight) if engine or no_backward(x, weight) else NotImplemented
    return y if y is not NotImplemented else _Linear.apply(x, weight)


# ----------------------------------------------------------------------------- GEMMs fused with a collective
class FusedCollectiveGemm:
    """Per-group state for the two single-kernel compute+collective GEMMs (csrc/gemm.cu modes 1 and 2):
    the symmetric flag buffer, the local flag words, the epoch counter and the status words.

    ``gemm_rs(a, b, out)``  row-parallel linear: every rank multiplies its K-slice for ALL rows and each
    output tile is TMA-reduce-added over NVLink into the rank that owns those rows (``out`` is a
    ``SymmetricBuffer`` holding this rank's [M / world, N] shard).
    ``ag_gemm(a_full, b)``  column-parallel linear: ``a_full`` is a ``SymmetricBuffer`` of the FULL
    [M, K] activation in which each rank has written only its own row range; a few CTAs pull the peers'
    ranges in while the rest multiply, starting with the local rows.
    """

    def __init__(self, device, group, rank: int, world: int, max_m_blocks: int = 4096, gather_ctas: int = 16):
        from nanonemo_b200.parallel.symm import SymmetricBuffer

        self.rank, self.world, self.group, self.gather_ctas = rank, world, group, gather_ctas
        words = _lib.lib().nnb_comm_flag_words(max(1, gather_ctas))
        self.flags = SymmetricBuffer(words, torch.int32, device, group)
        self.flags.tensor.zero_()
        self.local_flags = torch.zeros(2 + max_m_blocks, dtype=torch.int32, device=device)
        self.comm_status = torch.zeros(8, dtype=torch.int32, device=device)
        self.epoch = 0
        torch.cuda.synchronize(device)
        torch.distributed.barrier(group)

    def gemm_rs(self, a: torch.Tensor, b: torch.Tensor, out, *, b_mn: bool = False, out_f32: bool = False):
        """a: [M, K_local]; b: [N, K_local] (or [K_local, N] when b_mn); out: SymmetricBuffer viewed as
        [M / world, N]. Returns this rank's reduced shard (valid once the kernel has run)."""
        a, b = _rowmajor2d(a), _rowmajor2d(b)
        M, K = a.shape
        N = b.shape[1] if b_mn else b.shape[0]
        shard = out.tensor.view(-1)[: (M // self.world) * N].view(M // self.world, N)
        shard.zero_()
        self.epoch += 1
        _lib.call("nnb_gemm_rs_bf16", _lib.ptr(a), _lib.ptr(b), out.ptr_array, self.flags.ptr_array, _lib.ptr(self.local_flags),
                  _lib.ptr(self.comm_status), _lib.i32(self.rank), _lib.i32(self.world), _lib.i32(self.epoch), _lib.i32(M),
                  _lib.i32(N), _lib.i32(K), _lib.i64(a.stride(0)), _lib.i64(b.stride(0)), _lib.i64(N), _lib.i32(int(b_mn)),
                  _lib.i32(_CODE[a.dtype]), _lib.i32(int(out_f32)), _lib.ptr(status_tensor(a.device)), _lib.vp(_lib.stream_ptr()))
        return shard

    def ag_gemm(self, a_full, M: int, K: int, b: torch.Tensor, *, b_mn: bool = False, out: torch.Tensor | None = None):
        """a_full: SymmetricBuffer holding [M, K] 16-bit with this rank's rows already written."""
        b = _rowmajor2d(b)
        N = b.shape[1] if b_mn else b.shape[0]
        dtype = a_full.tensor.dtype
        out = out if out is not None else torch.empty((M, N), dtype=dtype, device=b.device)
        self.epoch += 1
        _lib.call("nnb_ag_gemm_bf16", a_full.ptr_array, _lib.ptr(b), _lib.ptr(out), self.flags.ptr_array, _lib.ptr(self.local_flags),
                  _lib.ptr(self.comm_status), _lib.i32(self.rank), _lib.i32(self.world), _lib.i32(self.epoch),
                  _lib.i32(self.gather_ctas), _lib.i32(M), _lib.i32(N), _lib.i32(K), _lib.i64(b.stride(0)), _lib.i64(out.stride(0)),
                  _lib.i32(int(b_mn)), _lib.i32(_CODE[dtype]), _lib.ptr(status_tensor(b.device)), _lib.vp(_lib.stream_ptr()))
        return out

    def gather_b_gemm(self, a: torch.Tensor, wire, src_off_bytes: int, per_bytes: int, unit_dst: torch.Tensor, b_off_bytes: int,
                      N: int, out: torch.Tensor | None = None):
        """a [M, K] @ B[N, K]^T where B sits `b_off_bytes` into a parameter unit sharded over the ranks (`wire`:
        SymmetricBuffer with every rank's shard at `src_off_bytes`, `per_bytes` each). The kernel all-gathers the WHOLE unit
        into `unit_dst` (this rank's unsharded 16-bit copy) while it multiplies: afterwards every parameter of the unit is local."""
        a = _rowmajor2d(a)
        M, K = a.shape
        out = out if out is not None else torch.empty((M, N), dtype=a.dtype, device=a.device)
        chunks = self.world * ((per_bytes + 32767) // 32768)
        assert 2 + chunks <= self.local_flags.numel(), "unit too large for the flag table"
        self.epoch += 1
        _lib.call("nnb_gather_b_gemm_bf16", _lib.ptr(a), wire.ptr_array, _lib.ptr(unit_dst), _lib.ptr(out), self.flags.ptr_array,
                  _lib.ptr(self.local_flags), _lib.ptr(self.comm_status), _lib.i32(self.rank), _lib.i32(self.world), _lib.i32(self.epoch),
                  _lib.i32(self.gather_ctas), _lib.i64(src_off_bytes), _lib.i64(per_bytes), _lib.i64(b_off_bytes), _lib.i32(M), _lib.i32(N),
                  _lib.i32(K), _lib.i64(a.stride(0)), _lib.i64(out.stride(0)), _lib.i32(_CODE[a.dtype]), _lib.ptr(status_tensor(a.device)),
                  _lib.vp(_lib.stream_ptr()))
        return out

    def check_status(self):
        st = self.comm_status.tolist()
        if st[0] != 0:
            self.comm_status.zero_()
            raise RuntimeError(f"fused GEMM collective gave up waiting: code={st[0]} rank={st[1]} peer={st[2]} block={st[3]} epoch={st[4]}")
        check_status()

"""``torch.library`` registration of the sm100 operators: schema + fake (meta) implementation + autograd formula
for each, so they compose with ``torch.compile(fullgraph=True)``, ``opcheck`` and functional transforms — the binding
layer of the reference (nanonemo/kernels/cuda/rmsnorm.py:1-69, flash_attn.py:1-60: ``custom_op`` + ``register_fake`` +
``register_autograd``), on top of the ahead-of-time built library instead of a per-process JIT.

``nanonemo_b200.ops`` routes here what the native operators (csrc/binding.cpp) leave: operators that they do not have, and every call
that is not a plain one (tracing, transforms, tensor subclasses, tangents), unless the parameter involved lives in a flat parameter
store (``weight._main_grad``), where the trainer's variants accumulate weight gradients in place in the flat buffer and report
gradient readiness to the strategy — side effects a functional operator cannot have. The native operators' backward nodes come
here too under create_graph=True and for batched gradients. All routes call the same launchers.

    torch.ops.nanonemo_b200.add_rms_norm(x, delta, weight, eps)              -> (y, h, rstd)
    torch.ops.nanonemo_b200.swiglu(gu)                                       -> act
    torch.ops.nanonemo_b200.rope_qkv(qkv, cos, sin, H, KVH, hd, sign)        -> qkv_rot
    torch.ops.nanonemo_b200.flash_attn_packed(qkv, H, KVH, hd, in_order)     -> (o, lse)
    torch.ops.nanonemo_b200.matmul_nt(a, b, a_mn, b_mn, out_f32)             -> a @ b^T
    torch.ops.nanonemo_b200.linear_w(x2, weight)                             -> x2 @ weight^T (fp32 or 16-bit weight)
    torch.ops.nanonemo_b200.gemm_rope(x2, weight, cos, sin, T, cols, hd)     -> projection with RoPE in the epilogue
    torch.ops.nanonemo_b200.gemm_swiglu(x2, weight)                          -> (gu, act) with SwiGLU in the epilogue
    torch.ops.nanonemo_b200.embedding(idx, weight, fp32_out)                 -> rows
    torch.ops.nanonemo_b200.linear_ce(x2, weight, targets, chunk_rows)       -> (mean loss, dx, dW)
    torch.ops.nanonemo_b200.linear_ce_loss(x2, weight, targets, chunk_rows)  -> mean loss, when no gradient is wanted
    torch.ops.nanonemo_b200.adamw_step(p, g, m, v, shadow, flags, ...)       -> None (mutates its buffers)
"""

import math

import torch
from torch import Tensor
from torch.autograd.forward_ad import unpack_dual

from nanonemo_b200.ops import adamw as adamw_mod, attention, embed as embed_mod, gemm as gemm_mod, linear_ce as ce_mod, rmsnorm, rope, swiglu_act

NS = "nanonemo_b200"


_NO_FORMULA = {}  # operators that have no derivative formula (so far)


def _operator(fn):
    """Register `fn` as the CUDA kernel of operator NS::<its name>, with the schema of its annotations. This is
    ``torch.library.custom_op`` without the wrapper that checks every call's results for aliases of its arguments (the kernels
    below return new tensors only). With custom_op and all else as here, a 201-token forward of the 114M model (87 operator calls)
    takes 5.2 ms instead of 4.55, add + RMSNorm forward and backward 211 us instead of 188.
    Like ``custom_op``, and unlike a bare definition, an operator without a formula stops a backward pass that reaches it: see
    the end of this file."""
    name = f"{NS}::{fn.__name__}"
    torch.library.define(name, torch.library.infer_schema(fn, mutates_args=()), tags=(torch.Tag.pt2_compliant_tag,))
    torch.library.impl(name, "cuda", torch.compiler.disable(fn))
    op = getattr(torch.ops.nanonemo_b200, fn.__name__).default
    _NO_FORMULA[op.name()] = op
    return op


def _fake(op):
    return torch.library.register_fake(op.name())


def _autograd(op, backward, setup_context=None):
    torch.library.register_autograd(op.name(), backward, setup_context=setup_context)
    _NO_FORMULA.pop(op.name())


def _from_formula(op, *args):
    """Call a backward operator from a derivative formula. Outside create_graph=True nothing can be differentiated by what it
    returns, so the call skips the autograd kernel (5 us less on the host), whose only work is to refuse (end of this file)."""
    if torch.is_grad_enabled():
        return op(*args)
    with torch._C._AutoDispatchBelowAutograd():
        return op(*args)


# ----------------------------------------------------------------------------- add + RMSNorm
_DT = {0: torch.float32, 1: torch.bfloat16, 2: torch.float16}
_DT_CODE = {v: k for k, v in _DT.items()}


@_operator
def add_rms_norm(x: Tensor, delta: Tensor | None, weight: Tensor, eps: float, y_code: int = -1) -> tuple[Tensor, Tensor, Tensor]:
    """(y, h, rstd): h = x + delta (x itself without a delta), y = rmsnorm(h) * weight in dtype code y_code (0 fp32, 1 bf16,
    2 fp16; -1 = the delta's dtype, or x's without a delta)."""
    y_dtype = _DT[y_code] if y_code >= 0 else (delta.dtype if delta is not None else x.dtype)
    y, h, rstd = rmsnorm.fwd(x, delta, weight, eps, y_dtype)
    return y, (h if delta is not None else h.clone()), rstd


@_fake(add_rms_norm)
def _(x, delta, weight, eps, y_code=-1):
    y_dtype = _DT[y_code] if y_code >= 0 else (delta.dtype if delta is not None else x.dtype)
    return (x.new_empty(x.shape, dtype=y_dtype), torch.empty_like(x, memory_format=torch.contiguous_format),
            x.new_empty(x.numel() // x.shape[-1], dtype=torch.float32))


@_operator
def add_rms_norm_bwd(dy: Tensor, dh: Tensor | None, h: Tensor, rstd: Tensor, weight: Tensor, delta_code: int) -> tuple[Tensor, Tensor, Tensor]:
    """(dx, ddelta, dw); ddelta has dtype code delta_code (when it equals the residual dtype it is a copy of dx)."""
    dx, ddelta, dw = rmsnorm.bwd(dy, h, rstd, weight, dh, _DT[delta_code])
    return dx, ddelta if ddelta is not dx else dx.clone(), dw


@_fake(add_rms_norm_bwd)
def _(dy, dh, h, rstd, weight, delta_code):
    return torch.empty_like(h), h.new_empty(h.shape, dtype=_DT[delta_code]), weight.new_empty(weight.shape, dtype=torch.float32)


def _arn_setup(ctx, inputs, output):
    x, delta, weight, _, _ = inputs
    y, h, rstd = output
    ctx.save_for_backward(h, rstd, weight)
    ctx.has_delta = delta is not None
    ctx.delta_code = _DT_CODE[delta.dtype if delta is not None else y.dtype]
    ctx.y_dtype = y.dtype
    ctx.set_materialize_grads(False)


def _arn_backward(ctx, dy, dh, _drstd):
    h, rstd, weight = ctx.saved_tensors
    dy = dy.contiguous() if dy is not None else torch.zeros(h.shape, dtype=ctx.y_dtype, device=h.device)
    dx, ddelta, dw = _from_formula(add_rms_norm_bwd, dy, dh.contiguous() if dh is not None else None, h, rstd, weight, ctx.delta_code)
    return dx, (ddelta if ctx.has_delta else None), dw.to(weight.dtype), None, None


_autograd(add_rms_norm, _arn_backward, setup_context=_arn_setup)


# ----------------------------------------------------------------------------- SwiGLU (packed gate || up)
@_operator
def swiglu(gu: Tensor) -> Tensor:
    F = gu.shape[-1] // 2
    gu2 = swiglu_act._rows(gu)
    out = torch.empty((gu2.shape[0], F), dtype=gu.dtype, device=gu.device)
    swiglu_act.fwd_raw(gu2[:, :F], gu2[:, F:], out)
    return out.view(*gu.shape[:-1], F)


@_fake(swiglu)
def _(gu):
    return gu.new_empty((*gu.shape[:-1], gu.shape[-1] // 2))


@_operator
def swiglu_bwd(dy: Tensor, gu: Tensor) -> Tensor:
    F = gu.shape[-1] // 2
    gu2, dy2 = swiglu_act._rows(gu), swiglu_act._rows(dy)
    dgu = torch.empty((gu2.shape[0], 2 * F), dtype=gu.dtype, device=gu.device)
    swiglu_act.bwd_raw(dy2, gu2[:, :F], gu2[:, F:], dgu[:, :F], dgu[:, F:])
    return dgu.view(gu.shape)


@_fake(swiglu_bwd)
def _(dy, gu):
    return torch.empty_like(gu, memory_format=torch.contiguous_format)


_autograd(swiglu, lambda ctx, dy: _from_formula(swiglu_bwd, dy.contiguous(), ctx.saved_tensors[0]),
                         setup_context=lambda ctx, inputs, output: ctx.save_for_backward(inputs[0]))


# ----------------------------------------------------------------------------- RoPE on the packed projection
@_operator
def rope_qkv(qkv: Tensor, cos: Tensor, sin: Tensor, n_heads: int, n_kv_heads: int, head_dim: int, sign: float = 1.0) -> Tensor:
    B, T, C = qkv.shape
    x2 = qkv.reshape(B * T, C)
    x2 = x2 if x2.stride(-1) == 1 else x2.contiguous()
    c, s = rope._tables(cos, sin, T)
    out = torch.empty((B * T, C), dtype=qkv.dtype, device=qkv.device)
    rope.rope_packed_raw(x2, out, c, s, T, n_heads + n_kv_heads, head_dim, n_kv_heads * head_dim, sign)
    return out.view(B, T, C)


@_fake(rope_qkv)
def _(qkv, cos, sin, n_heads, n_kv_heads, head_dim, sign=1.0):
    return torch.empty_like(qkv, memory_format=torch.contiguous_format)


def _rope_setup(ctx, inputs, output):
    _, cos, sin, H, KVH, hd, sign = inputs
    ctx.save_for_backward(cos, sin)
    ctx.meta = (H, KVH, hd, sign)


def _rope_backward(ctx, dout):
    cos, sin = ctx.saved_tensors
    H, KVH, hd, sign = ctx.meta
    return rope_qkv(dout.contiguous(), cos, sin, H, KVH, hd, -sign), None, None, None, None, None, None


_autograd(rope_qkv, _rope_backward, setup_context=_rope_setup)


# ----------------------------------------------------------------------------- FlashAttention on the packed projection
def _split(qkv, H, KVH, hd):
    B, T, _ = qkv.shape
    return (qkv[..., : H * hd].view(B, T, H, hd), qkv[..., H * hd:(H + KVH) * hd].view(B, T, KVH, hd),
            qkv[..., (H + KVH) * hd:].view(B, T, KVH, hd))


@_operator
def flash_attn_packed(qkv: Tensor, n_heads: int, n_kv_heads: int, head_dim: int, in_order: bool = False) -> tuple[Tensor, Tensor]:
    """`in_order` is of the backward pass (``attention.bwd_raw``)."""
    qkv = qkv.contiguous()
    B, T, _ = qkv.shape
    q, k, v = _split(qkv, n_heads, n_kv_heads, head_dim)
    o = torch.empty((B, T, n_heads, head_dim), dtype=qkv.dtype, device=qkv.device)
    lse = attention.fwd_raw(q, k, v, o, 1.0 / math.sqrt(head_dim))
    return o.view(B, T, n_heads * head_dim), lse


@_fake(flash_attn_packed)
def _(qkv, n_heads, n_kv_heads, head_dim, in_order=False):
    B, T, _ = qkv.shape
    return qkv.new_empty((B, T, n_heads * head_dim)), qkv.new_empty((B, n_heads, T), dtype=torch.float32)


@_operator
def flash_attn_packed_bwd(do: Tensor, qkv: Tensor, o: Tensor, lse: Tensor, n_heads: int, n_kv_heads: int, head_dim: int, in_order: bool = False) -> Tensor:
    qkv, do = qkv.contiguous(), do.contiguous()
    B, T, _ = qkv.shape
    q, k, v = _split(qkv, n_heads, n_kv_heads, head_dim)
    dqkv = torch.empty_like(qkv)
    dq, dk, dv = _split(dqkv, n_heads, n_kv_heads, head_dim)
    attention.bwd_raw(q, k, v, o.view(B, T, n_heads, head_dim), lse, do.view(B, T, n_heads, head_dim), dq, dk, dv, 1.0 / math.sqrt(head_dim),
                      in_order=in_order)
    return dqkv


@_fake(flash_attn_packed_bwd)
def _(do, qkv, o, lse, n_heads, n_kv_heads, head_dim, in_order=False):
    return torch.empty_like(qkv, memory_format=torch.contiguous_format)


def _fa_setup(ctx, inputs, output):
    qkv, H, KVH, hd, in_order = inputs
    o, lse = output
    ctx.save_for_backward(qkv, o, lse)
    ctx.meta = (H, KVH, hd, in_order)


def _fa_backward(ctx, do, _dlse):
    qkv, o, lse = ctx.saved_tensors
    return _from_formula(flash_attn_packed_bwd, do, qkv, o, lse, *ctx.meta), None, None, None, None


_autograd(flash_attn_packed, _fa_backward, setup_context=_fa_setup)


# ----------------------------------------------------------------------------- linear (tcgen05 GEMM), 16-bit weight
@_operator
def matmul_nt(a: Tensor, b: Tensor, a_mn: bool = False, b_mn: bool = False, out_f32: bool = False) -> Tensor:
    """a @ b^T with the operand layouts of csrc/gemm.cu (a_mn / b_mn: the operand is stored transposed)."""
    return gemm_mod.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32 if out_f32 else None)


@_fake(matmul_nt)
def _(a, b, a_mn=False, b_mn=False, out_f32=False):
    M = a.shape[1] if a_mn else a.shape[0]
    N = b.shape[1] if b_mn else b.shape[0]
    return a.new_empty((M, N), dtype=torch.float32 if out_f32 else a.dtype)


def _mm_setup(ctx, inputs, output):
    a, b, a_mn, b_mn, out_f32 = inputs
    assert not a_mn and not b_mn, "autograd is defined for the plain a @ b^T form"
    ctx.save_for_backward(a, b)


def _mm_backward(ctx, dy):
    a, b = ctx.saved_tensors
    dy = dy.to(a.dtype).contiguous()
    da = matmul_nt(dy, b, False, True, False)          # dy @ b
    db = matmul_nt(dy, a, True, True, False)           # dy^T @ a
    return da, db, None, None, None


_autograd(matmul_nt, _mm_backward, setup_context=_mm_setup)




# ----------------------------------------------------------------------------- linear with the weight as given (fp32 master or 16-bit)
def _w16(weight: Tensor, dtype: torch.dtype) -> Tensor:
    return weight if weight.dtype == dtype else weight.to(dtype)


@_operator
def linear_w(x2: Tensor, weight: Tensor) -> Tensor:
    """x2 [M, K] (16-bit) @ weight [N, K]^T; an fp32 weight is cast to x2's dtype for the product."""
    return gemm_mod.gemm(x2, _w16(weight, x2.dtype))


@_fake(linear_w)
def _(x2, weight):
    return x2.new_empty((x2.shape[0], weight.shape[0]))


def _linw_setup(ctx, inputs, output):
    ctx.save_for_backward(*inputs)


def _linw_backward(ctx, dy):
    x2, weight = ctx.saved_tensors
    dy = dy.to(x2.dtype).contiguous()
    dx = matmul_nt(dy, _w16(weight, x2.dtype), False, True, False)
    dw = matmul_nt(dy, x2, True, True, True)  # fp32 accumulate and output: the master weight's gradient keeps full precision
    return dx, dw.to(weight.dtype)


_autograd(linear_w, _linw_backward, setup_context=_linw_setup)


def linear(x: Tensor, weight: Tensor) -> Tensor:
    """x [..., K] @ weight [N, K]^T in the autocast dtype (bf16 by default) through the registered operator."""
    dt = gemm_mod.compute_dtype()
    x2 = x.reshape(-1, x.shape[-1])
    x2 = x2 if x2.dtype == dt else x2.to(dt)
    return linear_w(x2.contiguous(), weight).view(*x.shape[:-1], weight.shape[0])


# ----------------------------------------------------------------------------- RoPE on 2-D rows (any column count, in / out of place)
@_operator
def rope_rows(x2: Tensor, cos: Tensor, sin: Tensor, t_len: int, n_rot_heads: int, head_dim: int, sign: float) -> Tensor:
    """Rotate-half on the first n_rot_heads heads of every row (row m at position m % t_len), other columns copied."""
    x2 = x2 if x2.stride(-1) == 1 else x2.contiguous()
    out = torch.empty(x2.shape, dtype=x2.dtype, device=x2.device)
    rope.rope_packed_raw(x2, out, cos, sin, t_len, n_rot_heads, head_dim, x2.shape[1] - n_rot_heads * head_dim, sign)
    return out


@_fake(rope_rows)
def _(x2, cos, sin, t_len, n_rot_heads, head_dim, sign):
    return torch.empty_like(x2, memory_format=torch.contiguous_format)


def _rr_setup(ctx, inputs, output):
    _, cos, sin, t_len, n_rot, hd, sign = inputs
    ctx.save_for_backward(cos, sin)
    ctx.meta = (t_len, n_rot, hd, sign)


def _rr_backward(ctx, dout):
    cos, sin = ctx.saved_tensors
    t_len, n_rot, hd, sign = ctx.meta
    return rope_rows(dout.contiguous(), cos, sin, t_len, n_rot, hd, -sign), None, None, None, None, None, None


_autograd(rope_rows, _rr_backward, setup_context=_rr_setup)


# ----------------------------------------------------------------------------- GEMMs with a fused epilogue
@_operator
def gemm_rope(x2: Tensor, weight: Tensor, cos: Tensor, sin: Tensor, t_len: int, rope_cols: int, head_dim: int) -> Tensor:
    """x2 @ weight^T with RoPE on columns [0, rope_cols) in the GEMM epilogue (plain GEMM + RoPE kernel for shapes the
    fused kernel does not serve: same result)."""
    w16 = _w16(weight, x2.dtype)
    out = gemm_mod.gemm_rope(x2, w16, cos, sin, t_len, rope_cols, head_dim)
    if out is None:
        out = gemm_mod.gemm(x2, w16)
        rope.rope_packed_raw(out, out, cos, sin, t_len, rope_cols // head_dim, head_dim, 0, 1.0)
    return out


@_fake(gemm_rope)
def _(x2, weight, cos, sin, t_len, rope_cols, head_dim):
    return x2.new_empty((x2.shape[0], weight.shape[0]))


def _gr_setup(ctx, inputs, output):
    x2, weight, cos, sin, t_len, rope_cols, hd = inputs
    ctx.save_for_backward(x2, weight, cos, sin)
    ctx.meta = (t_len, rope_cols, hd)


def _gr_backward(ctx, dout):
    x2, weight, cos, sin = ctx.saved_tensors
    t_len, rope_cols, hd = ctx.meta
    draw = rope_rows(dout.to(x2.dtype).contiguous(), cos, sin, t_len, rope_cols // hd, hd, -1.0)
    dx = matmul_nt(draw, _w16(weight, x2.dtype), False, True, False)
    dw = matmul_nt(draw, x2, True, True, True)
    return dx, dw.to(weight.dtype), None, None, None, None, None


_autograd(gemm_rope, _gr_backward, setup_context=_gr_setup)


@_operator
def gemm_swiglu(x2: Tensor, weight: Tensor) -> tuple[Tensor, Tensor]:
    """(gu, act): gu = x2 @ weight^T with gate columns first, act = silu(gate) * up written by the GEMM epilogue."""
    w16 = _w16(weight, x2.dtype)
    fused = gemm_mod.gemm_swiglu(x2, w16)
    if fused is not None:
        return fused
    gu = gemm_mod.gemm(x2, w16)
    F = gu.shape[1] // 2
    act = torch.empty((gu.shape[0], F), dtype=gu.dtype, device=gu.device)
    swiglu_act.fwd_raw(gu[:, :F], gu[:, F:], act)
    return gu, act


@_fake(gemm_swiglu)
def _(x2, weight):
    return x2.new_empty((x2.shape[0], weight.shape[0])), x2.new_empty((x2.shape[0], weight.shape[0] // 2))


def _gs_setup(ctx, inputs, output):
    ctx.save_for_backward(*inputs, output[0])


def _gs_backward(ctx, dgu, dact):
    x2, weight, gu = ctx.saved_tensors
    total = None
    if dact is not None:
        total = _from_formula(swiglu_bwd, dact.to(gu.dtype).contiguous(), gu)
    if dgu is not None:
        total = dgu.to(gu.dtype) if total is None else total + dgu.to(gu.dtype)
    total = total.contiguous()
    dx = matmul_nt(total, _w16(weight, x2.dtype), False, True, False)
    dw = matmul_nt(total, x2, True, True, True)
    return dx, dw.to(weight.dtype)


_autograd(gemm_swiglu, _gs_backward, setup_context=_gs_setup)


# ----------------------------------------------------------------------------- embedding
@_operator
def embedding(idx: Tensor, weight: Tensor, fp32_out: bool = True) -> Tensor:
    """weight[idx] from the fp32 table, written in fp32 or bf16 (the dtype of the residual stream)."""
    w = weight if weight.dtype == torch.float32 else weight.float()
    out, _ = embed_mod.fwd_raw(idx, w.contiguous(), torch.float32 if fp32_out else torch.bfloat16)
    return out


@_fake(embedding)
def _(idx, weight, fp32_out=True):
    return weight.new_empty((*idx.shape, weight.shape[1]), dtype=torch.float32 if fp32_out else torch.bfloat16)


@_operator
def embedding_bwd(idx: Tensor, dout: Tensor, vocab: int) -> Tensor:
    """fp32 [vocab, D] with dout's rows added at idx (rows that repeat are summed)."""
    flat = idx.reshape(-1)
    flat = (flat if flat.dtype == torch.int64 else flat.long()).contiguous()
    dW = torch.zeros((vocab, dout.shape[-1]), dtype=torch.float32, device=dout.device)
    embed_mod.bwd_raw(flat, dout.contiguous(), dW)
    return dW


@_fake(embedding_bwd)
def _(idx, dout, vocab):
    return dout.new_empty((vocab, dout.shape[-1]), dtype=torch.float32)


def _emb_setup(ctx, inputs, output):
    idx, weight, _ = inputs
    ctx.save_for_backward(idx)
    ctx.vocab, ctx.w_dtype = weight.shape[0], weight.dtype


def _emb_backward(ctx, dout):
    (idx,) = ctx.saved_tensors
    return None, _from_formula(embedding_bwd, idx, dout, ctx.vocab).to(ctx.w_dtype), None


_autograd(embedding, _emb_backward, setup_context=_emb_setup)


# ----------------------------------------------------------------------------- fused linear + cross-entropy
@_operator
def linear_ce(x2: Tensor, weight: Tensor, targets: Tensor, chunk_rows: int) -> tuple[Tensor, Tensor, Tensor]:
    """Mean cross-entropy of x2 @ weight^T against targets, and the gradients of that mean with respect to x2 (16-bit)
    and weight (fp32), all produced in the same pass (the logits exist one row chunk at a time, in 16 bits)."""
    w16 = _w16(weight, x2.dtype)
    tg = (targets if targets.dtype == torch.int64 else targets.long()).contiguous()
    dW = torch.empty(weight.shape, dtype=torch.float32, device=x2.device)
    loss_sum, dx = ce_mod.linear_ce_fwd(x2, w16.contiguous(), tg, chunk_rows, dW)
    return loss_sum / x2.shape[0], dx, dW


@_fake(linear_ce)
def _(x2, weight, targets, chunk_rows):
    return x2.new_empty((), dtype=torch.float32), torch.empty_like(x2), weight.new_empty(weight.shape, dtype=torch.float32)


@_operator
def scaled(t: Tensor, scalar: Tensor) -> Tensor:
    """t * scalar for a 0-dim fp32 scalar on the device."""
    return ce_mod.scale(t, scalar)


@_fake(scaled)
def _(t, scalar):
    return torch.empty_like(t, memory_format=torch.contiguous_format)


def _scaled_setup(ctx, inputs, output):
    ctx.save_for_backward(*inputs)


def _scaled_backward(ctx, g):
    t, scalar = ctx.saved_tensors
    return scaled(g.contiguous(), scalar), (g.float() * t.float()).sum().to(scalar.dtype).reshape(scalar.shape)


_autograd(scaled, _scaled_backward, setup_context=_scaled_setup)


def _lce_setup(ctx, inputs, output):
    ctx.save_for_backward(output[1], output[2])
    ctx.w_dtype = inputs[1].dtype
    ctx.set_materialize_grads(False)


def _lce_backward(ctx, dloss, _ddx, _ddw):
    dx, dW = ctx.saved_tensors
    if dloss is None:
        return None, None, None, None
    times = scaled if unpack_dual(dloss).tangent is None else ce_mod.times_upstream  # (`scaled` has no forward-mode formula)
    return times(dx, dloss), times(dW, dloss).to(ctx.w_dtype), None, None


_autograd(linear_ce, _lce_backward, setup_context=_lce_setup)


@_operator
def linear_ce_loss(x2: Tensor, weight: Tensor, targets: Tensor, chunk_rows: int) -> Tensor:
    """The loss of ``linear_ce`` alone: no gradients, one product instead of three, no logits in memory."""
    tg = (targets if targets.dtype == torch.int64 else targets.long()).contiguous()
    return ce_mod.linear_ce_loss(x2, _w16(weight, x2.dtype).contiguous(), tg, chunk_rows) / x2.shape[0]


@_fake(linear_ce_loss)
def _(x2, weight, targets, chunk_rows):
    return x2.new_empty((), dtype=torch.float32)


def linear_cross_entropy(x: Tensor, weight: Tensor, targets: Tensor, chunk_rows: int | None = None) -> Tensor:
    """x: [N, D]; weight: [V, D] (fp32 master or 16-bit); targets: [N] -> scalar mean loss (fp32)."""
    dt = gemm_mod.compute_dtype()
    x2 = x if x.dtype == dt else x.to(dt)
    if not (torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad)):
        if not torch.compiler.is_compiling() and not gemm_mod.no_backward(x, weight):
            raise NotImplementedError("linear_cross_entropy has no forward-mode derivative")  # as with gradients
        return linear_ce_loss(x2.contiguous(), weight, targets, chunk_rows or ce_mod.DEFAULT_CHUNK_ROWS)
    loss, _, _ = linear_ce(x2.contiguous(), weight, targets, chunk_rows or ce_mod.DEFAULT_CHUNK_ROWS)
    return loss


# ----------------------------------------------------------------------------- fused clip + AdamW on flat buffers
@torch.library.custom_op(f"{NS}::adamw_step", mutates_args=("p", "g", "m", "v", "shadow"), device_types="cuda")
def adamw_step(p: Tensor, g: Tensor, m: Tensor, v: Tensor, shadow: Tensor | None, decay_flags: Tensor, grad_norm_sq: Tensor | None,
               lr: float, beta1: float, beta2: float, eps: float, weight_decay: float, step: int, max_norm: float,
               zero_grad: bool) -> None:
    """One launch: clip by the global norm (grad_norm_sq on the device, max_norm <= 0 = no clipping), AdamW on the fp32
    master weights and moments, 16-bit shadow written, gradient zeroed. decay_flags: one byte per 256 elements."""
    adamw_mod.adamw_flat(p, g, m, v, shadow, decay_flags, lr=lr, beta1=beta1, beta2=beta2, eps=eps, weight_decay=weight_decay,
                         step=step, grad_norm_sq=grad_norm_sq if max_norm > 0 else None, max_norm=max_norm if max_norm > 0 else None,
                         zero_grad=zero_grad)


@adamw_step.register_fake
def _(p, g, m, v, shadow, decay_flags, grad_norm_sq, lr, beta1, beta2, eps, weight_decay, step, max_norm, zero_grad):
    return None


# ----------------------------------------------------------------------------- SwiGLU on separate gate / up tensors
@_operator
def swiglu_gu(g: Tensor, u: Tensor) -> Tensor:
    g2, u2 = swiglu_act._rows(g), swiglu_act._rows(u)
    out = torch.empty((g2.shape[0], g2.shape[1]), dtype=g.dtype, device=g.device)
    swiglu_act.fwd_raw(g2, u2, out)
    return out.view(g.shape)


@_fake(swiglu_gu)
def _(g, u):
    return torch.empty_like(g, memory_format=torch.contiguous_format)


@_operator
def swiglu_gu_bwd(dy: Tensor, g: Tensor, u: Tensor) -> tuple[Tensor, Tensor]:
    g2, u2, dy2 = swiglu_act._rows(g), swiglu_act._rows(u), swiglu_act._rows(dy)
    dg = torch.empty((g2.shape[0], g2.shape[1]), dtype=g.dtype, device=g.device)
    du = torch.empty_like(dg)
    swiglu_act.bwd_raw(dy2, g2, u2, dg, du)
    return dg.view(g.shape), du.view(g.shape)


@_fake(swiglu_gu_bwd)
def _(dy, g, u):
    return torch.empty_like(g, memory_format=torch.contiguous_format), torch.empty_like(g, memory_format=torch.contiguous_format)


_autograd(swiglu_gu, lambda ctx, dy: _from_formula(swiglu_gu_bwd, dy.contiguous(), *ctx.saved_tensors),
                            setup_context=lambda ctx, inputs, output: ctx.save_for_backward(*inputs))


# ----------------------------------------------------------------------------- FlashAttention on separate (B, H, T, hd) tensors
def _bthd(t: Tensor) -> Tensor:
    """(B, heads, T, hd) -> the kernel's [B, T, heads, hd] view; copied only when strides / alignment rule it out."""
    t = t.transpose(1, 2)
    ok = t.stride(-1) == 1 and all((s * 2) % 16 == 0 for s in t.stride()[:-1]) and t.data_ptr() % 16 == 0
    return t if ok else t.contiguous()


@_operator
def flash_attn(q: Tensor, k: Tensor, v: Tensor) -> tuple[Tensor, Tensor]:
    """Causal GQA attention on bf16 q (B, H, T, hd), k / v (B, KVH, T, hd) -> (o (B, H, T, hd), lse (B, H, T))."""
    qt, kt, vt = _bthd(q), _bthd(k), _bthd(v)
    B, T, H, hd = qt.shape
    o = torch.empty((B, T, H, hd), dtype=q.dtype, device=q.device)
    lse = attention.fwd_raw(qt, kt, vt, o, 1.0 / math.sqrt(hd))
    return o.transpose(1, 2), lse


@_fake(flash_attn)
def _(q, k, v):
    B, H, T, hd = q.shape
    return q.new_empty((B, T, H, hd)).transpose(1, 2), q.new_empty((B, H, T), dtype=torch.float32)


@_operator
def flash_attn_bwd(do: Tensor, q: Tensor, k: Tensor, v: Tensor, o: Tensor, lse: Tensor) -> tuple[Tensor, Tensor, Tensor]:
    qt, kt, vt, ot, dot = _bthd(q), _bthd(k), _bthd(v), _bthd(o), _bthd(do)
    hd = qt.shape[-1]
    dq = torch.empty(qt.shape, dtype=q.dtype, device=q.device)
    dk = torch.empty(kt.shape, dtype=q.dtype, device=q.device)
    dv = torch.empty(vt.shape, dtype=q.dtype, device=q.device)
    attention.bwd_raw(qt, kt, vt, ot, lse, dot, dq, dk, dv, 1.0 / math.sqrt(hd))
    return dq.transpose(1, 2), dk.transpose(1, 2), dv.transpose(1, 2)


@_fake(flash_attn_bwd)
def _(do, q, k, v, o, lse):
    mk = lambda t: t.new_empty((t.shape[0], t.shape[2], t.shape[1], t.shape[3])).transpose(1, 2)
    return mk(q), mk(k), mk(v)


def _fl_setup(ctx, inputs, output):
    ctx.save_for_backward(*inputs, *output)


def _fl_backward(ctx, do, _dlse):
    q, k, v, o, lse = ctx.saved_tensors
    return _from_formula(flash_attn_bwd, do.to(q.dtype), q, k, v, o, lse)


_autograd(flash_attn, _fl_backward, setup_context=_fl_setup)


# ----------------------------------------------------------------------------- operators without a derivative
# PyTorch lets an operator that has no formula through with a warning and drops its share of the derivative: a gradient of a
# gradient (create_graph=True) would come back with its second-order part missing. These refuse instead. The formula costs a call
# about 6 us on the host, which the derivative formulas above do not pay (_from_formula).
def _refuse(op):
    def backward(ctx, *grads):
        raise RuntimeError(f"Trying to backward through {op.name()}, which has no derivative formula")

    return backward


for _op in list(_NO_FORMULA.values()):
    _autograd(_op, _refuse(_op))

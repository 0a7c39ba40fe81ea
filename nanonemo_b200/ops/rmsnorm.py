"""Fused residual-add + RMSNorm (csrc/elementwise.cu): ``add_rms_norm(x, delta, w, eps) -> (y, h)``.

``h = x + delta`` is rounded to the dtype of the residual stream before normalising, ``y`` takes the
autocast dtype when autocast is on (else x's dtype), statistics are fp32 — the contract of the
reference operator (nanonemo/kernels/cuda/rmsnorm.py:1-69, rmsnorm.cu:64-167), with bf16 supported.
Backward returns the same tensor for ``dx`` and ``ddelta`` when their dtypes match, and a second
16-bit copy (written by the same kernel) when the residual stream is fp32 and delta is 16-bit.
"""

import torch

from nanonemo_b200.ops import _lib


def _y_dtype(x: torch.Tensor, delta) -> torch.dtype:
    if torch.is_autocast_enabled("cuda"):
        return torch.get_autocast_dtype("cuda")
    return delta.dtype if delta is not None else x.dtype


def fwd(x, delta, weight, eps, y_dtype):
    """Raw launcher. x: (..., N) residual dtype; delta same shape or None. Returns (y, h, rstd)."""
    return _lib.native().rms_fwd(x, delta, weight, eps, y_dtype)


def bwd(dy, h, rstd, weight, dres, delta_dtype, dw_out=None, accumulate=False):
    """Raw launcher. Returns (dx [residual dtype], ddelta [delta dtype or None], dw fp32 [N])."""
    return _lib.native().rms_bwd(dy, h, rstd, weight, dres, delta_dtype, dw_out, accumulate)


class _AddRMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, weight, eps):
        y_dtype = _y_dtype(x, delta)
        if delta is not None and delta.dtype != y_dtype:
            delta = delta.to(y_dtype)
        if x.dtype not in (torch.float32, y_dtype):
            x = x.float()
        y, h, rstd = fwd(x, delta, weight, eps, y_dtype)
        ctx.save_for_backward(h, rstd, weight)
        ctx.delta_dtype = delta.dtype if delta is not None else None
        ctx.mark_non_differentiable(rstd)
        return y, h, rstd

    @staticmethod
    def backward(ctx, dy, dh, _drstd):
        h, rstd, weight = ctx.saved_tensors
        if dy is None:
            dy = torch.zeros(h.shape, dtype=_y_dtype(h, None) if ctx.delta_dtype is None else ctx.delta_dtype, device=h.device)
        main = getattr(weight, "_main_grad", None)
        if main is not None and main.dtype == torch.float32:
            dx, ddelta, _ = bwd(dy, h, rstd, weight, dh, ctx.delta_dtype, dw_out=main, accumulate=True)
            cb = getattr(weight, "_grad_ready_cb", None)
            if cb is not None:
                cb(weight, True)
            dw = None
        else:
            dx, ddelta, dw = bwd(dy, h, rstd, weight, dh, ctx.delta_dtype)
            dw = dw.to(weight.dtype)
        return dx, ddelta, dw, None


def add_rms_norm(x, delta, weight, eps):
    out = _lib.operator_call("add_rms_norm", x, delta, weight, eps)
    if out is not NotImplemented:
        return out
    y, h, _ = _AddRMSNorm.apply(x, delta, weight, eps)
    return y, h

"""Raw launchers of the SwiGLU activation ``silu(g) * u`` (csrc/elementwise.cu). Backward recomputes the sigmoid from
the saved g and u (reference: nanonemo/kernels/triton/swiglu.py:19-66); gate and up may be the two halves of the fused
gate||up GEMM output (independent row strides). The differentiable operators are registered in ``ops/library.py``
(``swiglu`` on the packed projection, ``swiglu_gu`` on separate tensors)."""

from nanonemo_b200.ops import _lib


def _rows(t):
    t2 = t.reshape(-1, t.shape[-1])
    return t2 if t2.stride(-1) == 1 else t2.contiguous()


def fwd_raw(g2, u2, out2):
    _lib.native().swiglu_fwd(g2, u2, out2)


def bwd_raw(dy2, g2, u2, dg2, du2):
    _lib.native().swiglu_bwd(dy2, g2, u2, dg2, du2)

"""Raw launcher of the fused rotate-half RoPE on Q and K (csrc/elementwise.cu: rope_packed_kernel).

The kernel works on rows of a packed projection: the first ``n_rot_heads`` heads of every row are rotated, the
remaining ``n_copy_cols`` columns copied through (or left alone when input and output are the same buffer and
``n_copy_cols`` is 0). The inverse (backward) is the same kernel with the sine negated, so only the tables are saved
(as in the reference, nanonemo/kernels/triton/rope.py:44-45,87-90). The differentiable operators built on it are
registered in ``ops/library.py`` (``rope_qkv``, ``rope_rows``).
"""

import torch

from nanonemo_b200.ops import _lib


def rope_packed_raw(x2, out2, cos, sin, T, n_rot_heads, hd, n_copy_cols, sign):
    _lib.native().rope_packed(x2, out2, cos, sin, T, n_rot_heads, hd, n_copy_cols, sign)


def _tables(cos, sin, T):
    cos, sin = cos[:T], sin[:T]
    if cos.dtype != torch.float32:
        cos, sin = cos.float(), sin.float()
    return cos.contiguous(), sin.contiguous()

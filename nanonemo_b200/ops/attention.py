"""Causal grouped-query FlashAttention on tcgen05/TMEM (csrc/flash_fwd.cu, csrc/flash_bwd.cu).

Raw launches (through csrc/binding.cpp); the differentiable operators are there and in ``ops/library.py``: ``flash_attn(q, k, v)`` takes
(B, H, T, hd) / (B, KVH, T, hd) tensors with any strides whose last dim is contiguous (transposed views of a
(B, T, H, hd) projection are the common case) and returns (B, H, T, hd); ``flash_attn_packed(qkv, H, KVH, hd)`` reads
the three operands straight out of the packed (B, T, (H + 2 KVH) hd) projection and writes (B, T, H hd), and its
backward writes dQ, dK, dV into one packed gradient tensor, so no split / transpose / concat kernels run around attention.
Operands are bf16 or fp16 (one dtype for all of them; scores, softmax and every accumulator are fp32 either way).
Query head h reads KV head h // (H // KVH) directly (as the reference kernel does,
nanonemo/kernels/cuda/flash_attn.cu:59,72-74). The log-sum-exp per row is saved for backward.
"""

from nanonemo_b200.ops import _lib


def fwd_raw(q, k, v, o, scale):
    """q, o: [B, T, H, hd] views; k, v: [B, T, KVH, hd] views (any strides, contiguous last dim). Returns the log-sum-exp of the rows."""
    return _lib.native().flash_fwd(q, k, v, o, scale)


def bwd_raw(q, k, v, o, lse, do, dq, dk, dv, scale, rope_cos=None, rope_sin=None, in_order=False):
    """With `rope_cos` / `rope_sin` (fp32 [T, hd / 2], head_dim 64 only) dQ and dK are returned through the inverse RoPE,
    i.e. as gradients of the projection BEFORE the rotation that produced q and k. `in_order`: dK and dV are one sum in the order of
    the queries, whatever the size of the call (small calls otherwise add up the parts of two or four CTAs)."""
    _lib.native().flash_bwd(q, k, v, o, lse, do, dq, dk, dv, scale, rope_cos, rope_sin, in_order)

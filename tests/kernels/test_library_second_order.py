"""Derivatives of derivatives through the registered operators, on meta tensors: the operators' formulas run, their kernels do not."""

import pytest
import torch

from nanonemo_b200.ops import library as L

BF = torch.bfloat16


def _t(*shape, dtype=torch.float32):
    return torch.empty(*shape, dtype=dtype, device="meta", requires_grad=True)


def _ids(n):
    return torch.zeros(n, dtype=torch.long, device="meta")


FORWARD = {  # operator -> (its first result, the inputs to differentiate by)
    "add_rms_norm": lambda x=_t(8, 64), w=_t(64): (L.add_rms_norm(x, None, w, 1e-5, 0)[0], [x, w]),
    "swiglu": lambda gu=_t(8, 64): (L.swiglu(gu), [gu]),
    "swiglu_gu": lambda g=_t(8, 64), u=_t(8, 64): (L.swiglu_gu(g, u), [g, u]),
    "flash_attn_packed": lambda qkv=_t(1, 128, 192, dtype=BF): (L.flash_attn_packed(qkv, 1, 1, 64)[0], [qkv]),
    "flash_attn": lambda q=_t(1, 1, 128, 64, dtype=BF), k=_t(1, 1, 128, 64, dtype=BF): (L.flash_attn(q, k, k)[0], [q, k]),
    "embedding": lambda w=_t(32, 64): (L.embedding(_ids(8), w, True), [w]),
}

BACKWARD = {  # operators without a formula, called on their own
    "add_rms_norm_bwd": lambda x=_t(8, 64): L.add_rms_norm_bwd(x, None, x, _t(8), _t(64), 0),
    "swiglu_bwd": lambda gu=_t(8, 64): L.swiglu_bwd(_t(8, 32), gu),
    "swiglu_gu_bwd": lambda g=_t(8, 64): L.swiglu_gu_bwd(g, g, g),
    "flash_attn_packed_bwd": lambda o=_t(1, 128, 64, dtype=BF): L.flash_attn_packed_bwd(o, _t(1, 128, 192, dtype=BF), o, _t(1, 1, 128), 1, 1, 64),
    "flash_attn_bwd": lambda q=_t(1, 1, 128, 64, dtype=BF): L.flash_attn_bwd(q, q, q, q, q, _t(1, 1, 128)),
    "embedding_bwd": lambda d=_t(8, 64): L.embedding_bwd(_ids(8), d, 32),
    "linear_ce_loss": lambda x=_t(128, 64, dtype=BF): L.linear_ce_loss(x, _t(64, 64, dtype=BF), _ids(128), 128),
}


@pytest.mark.parametrize("name", FORWARD)
def test_second_derivatives_are_refused(name):
    """The backward kernels have no derivative of their own: a gradient that is to be differentiated again must not leave them out."""
    y, inputs = FORWARD[name]()
    dy = torch.empty(y.shape, dtype=y.dtype, device="meta", requires_grad=True)
    grads = torch.autograd.grad(y, inputs, dy, create_graph=True)
    with pytest.raises(RuntimeError, match="no derivative formula"):
        torch.autograd.grad(sum(g.float().sum() for g in grads), [*inputs, dy], allow_unused=True)


@pytest.mark.parametrize("name", FORWARD)
def test_first_derivatives_stay(name):
    y, inputs = FORWARD[name]()
    for g, t in zip(torch.autograd.grad(y, inputs, torch.empty_like(y)), inputs):
        assert g.shape == t.shape and g.dtype == t.dtype and not g.requires_grad


@pytest.mark.parametrize("name", FORWARD)
def test_gradients_of_several_upstream_gradients_at_once(name):
    y, inputs = FORWARD[name]()
    for g, t in zip(torch.autograd.grad(y, inputs, y.new_empty((3, *y.shape)), is_grads_batched=True), inputs):
        assert g.shape == (3, *t.shape)


@pytest.mark.parametrize("name", BACKWARD)
def test_an_operator_without_a_formula_stops_a_backward_pass(name):
    out = BACKWARD[name]()
    out = out[0] if isinstance(out, tuple) else out
    with pytest.raises(RuntimeError, match="no derivative formula"):
        out.float().sum().backward()


def test_every_operator_has_a_formula_or_refuses():
    assert not L._NO_FORMULA


def test_linear_in_the_upstream_gradient_stays_differentiable():
    """RoPE is linear and the fused head scales stored gradients: both are differentiable in the upstream gradient."""
    cos, qkv, x, w = torch.empty(128, 32, device="meta"), _t(1, 128, 192, dtype=BF), _t(128, 64, dtype=BF), _t(64, 64, dtype=BF)
    for y, inputs in ((L.rope_qkv(qkv, cos, cos, 1, 1, 64), [qkv]), (L.linear_ce(x, w, _ids(128), 128)[0], [x, w])):
        dy = torch.empty(y.shape, dtype=y.dtype, device="meta", requires_grad=True)
        grads = torch.autograd.grad(y, inputs, dy, create_graph=True)
        assert torch.autograd.grad(sum(g.float().sum() for g in grads), dy)[0].shape == dy.shape

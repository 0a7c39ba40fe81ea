"""The fused head makes its gradients in the forward pass, for an upstream gradient of one; its backward multiplies them by the real
one. That product has to keep what hangs on the upstream gradient: its history, its tangent, its batch. On CPU, with the
kernels replaced by plain arithmetic and the raw launch by one that, like it, sees values only. Factors are powers of two, so that the
products of the 16-bit gradients are exact."""

import pytest
import torch
from torch.autograd import forward_ad

from nanonemo_b200.ops import library, linear_ce

N, D, V = 6, 4, 10


def _grads(x, w, targets):
    """(sum of row losses, d mean / dx, d mean / dw)."""
    logits = x.float() @ w.float().t()
    p = logits.softmax(-1)
    p[torch.arange(len(targets)), targets] -= 1
    p /= len(targets)
    return torch.nn.functional.cross_entropy(logits, targets, reduction="sum"), (p @ w.float()).to(x.dtype), p.t() @ x.float()


def _values(t, scalar, out=None):
    if not torch._C._has_storage(scalar):
        raise RuntimeError("no data pointer")
    with torch.no_grad():
        got = (forward_ad.unpack_dual(t.float()).primal * forward_ad.unpack_dual(scalar).primal.detach()).to(t.dtype)
        return got if out is None else out.add_(got)


class _Tp:
    world = 1
    all_gather = staticmethod(lambda t: t)


@pytest.fixture(params=["engine", "vocab_parallel"])
def head(request, monkeypatch):
    monkeypatch.setattr(linear_ce, "scale", _values)

    def fwd(x, w, targets, chunk_rows, dW):
        loss, dx, dw = _grads(x, w, targets)
        dW.copy_(dw)
        return loss, dx

    def gemm(a, b, out=None, a_mn=False, b_mn=False, accumulate=False, bn=0):
        out.copy_((a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t()))

    def ce_inplace(logits, targets, loss_rows, scale, v0, v_total, all_gather, world):
        loss_rows.copy_(torch.nn.functional.cross_entropy(logits.float(), targets, reduction="none"))
        p = logits.float().softmax(-1)
        p[torch.arange(len(targets)), targets] -= 1
        logits.copy_(p * scale)

    monkeypatch.setattr(linear_ce, "linear_ce_fwd", fwd)
    monkeypatch.setattr(linear_ce, "gemm", gemm)
    monkeypatch.setattr(linear_ce, "vocab_parallel_ce_inplace", ce_inplace)
    monkeypatch.setattr(linear_ce, "_sm_count", lambda device: 148)
    if request.param == "engine":
        return linear_ce.linear_cross_entropy
    return lambda x, w, t: linear_ce.vocab_parallel_linear_cross_entropy(x, w, t, _Tp, 0)


def _inputs():
    torch.manual_seed(0)
    return torch.randn(N, D, requires_grad=True), torch.randn(V, D, requires_grad=True), torch.randint(0, V, (N,))


def test_gradients_depend_on_the_upstream_factor(head):
    x, w, t = _inputs()
    c = torch.tensor(0.5, requires_grad=True)
    unit = torch.autograd.grad(head(x, w, t), (x, w))
    grads = torch.autograd.grad(head(x, w, t) * c, (x, w), create_graph=True)
    for g, u in zip(grads, unit):
        torch.testing.assert_close(g.detach(), u * 0.5, rtol=1e-6, atol=0)
        torch.testing.assert_close(torch.autograd.grad(g.sum(), c, retain_graph=True)[0], u.sum(), rtol=1e-5, atol=1e-6)


def test_gradients_of_several_upstream_gradients_at_once(head):
    x, w, t = _inputs()
    unit = torch.autograd.grad(head(x, w, t), (x, w))
    c = torch.tensor([1.0, -2.0, 0.25])
    for g, u in zip(torch.autograd.grad(head(x, w, t), (x, w), c, is_grads_batched=True), unit):
        torch.testing.assert_close(g, c.view(3, 1, 1) * u, rtol=1e-6, atol=0)


def test_gradients_carry_the_tangent_of_the_upstream_factor(head):
    x, w, t = _inputs()
    unit = torch.autograd.grad(head(x, w, t), (x, w))
    with forward_ad.dual_level():
        c = forward_ad.make_dual(torch.tensor(0.5), torch.tensor(2.0))
        for g, u in zip(torch.autograd.grad(head(x, w, t) * c, (x, w)), unit):
            torch.testing.assert_close(forward_ad.unpack_dual(g).tangent, 2 * u, rtol=1e-6, atol=0)


def test_the_registered_head_carries_the_tangent_too():
    x, w = (torch.empty(s, dtype=torch.bfloat16, device="meta", requires_grad=True) for s in ((128, 64), (64, 64)))
    with forward_ad.dual_level():
        c = forward_ad.make_dual(torch.empty((), device="meta"), torch.empty((), device="meta"))
        loss = library.linear_cross_entropy(x, w, torch.zeros(128, dtype=torch.long, device="meta"))
        for g, t in zip(torch.autograd.grad(loss * c, (x, w)), (x, w)):
            tangent = forward_ad.unpack_dual(g).tangent
            assert tangent is not None and tangent.shape == t.shape


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("requires_grad", [False, True])
def test_the_registered_head_refuses_tangents_of_its_inputs(which, requires_grad):
    inputs = [torch.empty(s, dtype=torch.bfloat16, device="meta") for s in ((128, 64), (64, 64))]
    targets = torch.zeros(128, dtype=torch.long, device="meta")
    assert library.linear_cross_entropy(*inputs, targets).shape == ()
    with forward_ad.dual_level():
        inputs[which] = forward_ad.make_dual(inputs[which].requires_grad_(requires_grad), torch.empty_like(inputs[which]))
        with pytest.raises(NotImplementedError):
            library.linear_cross_entropy(*inputs, targets)


def test_a_gradient_store_is_added_to(head):
    x, w, t = _inputs()
    unit = torch.autograd.grad(head(x, w, t), (x, w))
    w._main_grad = torch.ones(V, D)
    (head(x, w, t) * 0.5).backward()
    torch.testing.assert_close(w._main_grad, 1 + 0.5 * unit[1])
    assert w.grad is None


@pytest.fixture
def launched(monkeypatch):
    """The arguments of the raw launches: (source, destination, elements, accumulate)."""
    got = []

    def call(name, src, scalar, dst, n, dtype, accumulate, stream):
        assert name == "nnb_scale" and src % 16 == 0 and dst % 16 == 0
        got.append((src, dst, n, accumulate))

    monkeypatch.setattr(linear_ce._lib, "call", call)
    monkeypatch.setattr(linear_ce._lib, "stream_ptr", lambda: 0)
    return got


def test_scale_launches_on_dense_aligned_memory_only(launched):
    s, base = torch.tensor(0.5), torch.randn(12, 8)
    dense = base[:4]
    assert linear_ce.scale(dense, s).shape == (4, 8)
    assert launched.pop()[::2] == (dense.data_ptr(), 32)
    assert linear_ce.scale(dense, s, out=base[4:8]) is not None
    assert launched.pop() == (dense.data_ptr(), base[4:8].data_ptr(), 32, 1)
    offset = base.view(-1)[1:33]  # contiguous, four bytes past a vector: copied (`call` checks the addresses)
    linear_ce.scale(offset, s)
    assert launched.pop()[0] != offset.data_ptr()
    for t, out in ((dense, torch.zeros(4, 16)[:, :8]), (dense, torch.zeros(8, 4).t()), (offset, torch.zeros(33)[1:]),
                   (dense, torch.zeros(4, 8, dtype=torch.float64))):
        assert linear_ce.scale(t, s, out=out) is out and not launched
        torch.testing.assert_close(out.float(), t * 0.5)


@pytest.mark.parametrize("out", [torch.zeros(4, 9), torch.zeros(3, 8), torch.zeros(8)])
def test_scale_refuses_what_does_not_fit(launched, out):
    with pytest.raises(RuntimeError):
        linear_ce.scale(torch.randn(4, 8), torch.tensor(0.5), out=out)
    assert not launched


def test_scale_takes_one_value_on_the_same_device(launched):
    for scalar in (torch.ones(2), torch.ones((), device="meta")):
        with pytest.raises(ValueError):
            linear_ce.scale(torch.randn(4, 8), scalar)
    assert not launched


@pytest.mark.parametrize("rows,width,hint", [(256, 768, 128), (3072, 768, 128), (3073, 768, 0), (1152, 2048, 128), (1153, 2048, 0), (16384, 64, 128),
                                             (32768, 768, 0)])
def test_the_input_gradient_takes_narrow_tiles_while_one_wave_holds_them(monkeypatch, rows, width, hint):
    hints = []

    def gemm(a, b, out=None, a_mn=False, b_mn=False, accumulate=False, bn=0):
        if b_mn and not a_mn:
            hints.append(bn)

    monkeypatch.setattr(linear_ce, "gemm", gemm)
    monkeypatch.setattr(linear_ce, "gemm_ce_stats", lambda *a: None)
    monkeypatch.setattr(linear_ce, "ce_inplace", lambda *a: None)
    monkeypatch.setattr(linear_ce, "vocab_parallel_ce_inplace", lambda *a: None)
    monkeypatch.setattr(linear_ce, "_sm_count", lambda device: 148)
    x, w = (torch.empty(n, width, dtype=torch.bfloat16, device="meta", requires_grad=True) for n in (rows, 512))
    targets = torch.empty(rows, dtype=torch.long, device="meta")
    linear_ce.linear_cross_entropy(x, w, targets)
    linear_ce.vocab_parallel_linear_cross_entropy(x, w, targets, _Tp, 0)
    assert hints == [hint, hint]

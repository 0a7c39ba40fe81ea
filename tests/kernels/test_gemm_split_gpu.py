"""The head's input gradient of few rows: sums over parts of the vocabulary, added up in a fixed order."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,width,vocab", [(1, 128, 4096), (128, 768, 50304), (255, 512, 4104), (257, 1000, 8192), (777, 768, 32000), (4096, 768, 50304), (2049, 264, 16384)])
def test_parts_of_the_vocabulary_add_up_to_the_gradient(rows, width, vocab, dtype):
    from nanonemo_b200.ops import linear_ce
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(rows)
    g, w = torch.randn(rows, vocab, device=DEV).to(dtype), (torch.randn(vocab, width, device=DEV) * 0.02).to(dtype)
    assert linear_ce._dx_splits(rows, width, vocab) > 1
    got = [torch.full((rows, width), float("nan"), device=DEV, dtype=dtype) for _ in range(3)]
    for out, in_order in zip(got, (False, False, True)):
        linear_ce._input_gradient(g, w, out, in_order)
    check_status()
    assert torch.equal(got[0], got[1])  # a fixed order
    ref = g.double() @ w.double()
    off = [((t.double() - ref).norm() / ref.norm()).item() for t in (got[0], got[2])]
    # the result is rounded once, to 8 or 11 bits: 2^-9 or 2^-12 relative at most, and parts are no less exact than one sum (1 % for chance)
    assert off[0] <= (2**-9 if dtype == torch.bfloat16 else 2**-12) and off[0] <= 1.01 * off[1]


@pytest.mark.parametrize("engine", [True, False])
def test_one_sum_where_it_is_asked_for(monkeypatch, engine):
    """`in_order` (block-scaled models): the gradient of a row does not depend on how many rows there are."""
    from nanonemo_b200 import ops

    torch.manual_seed(3)
    x, w, t = torch.randn(300, 256, device=DEV).bfloat16(), torch.randn(8192, 256, device=DEV) * 0.02, torch.randint(0, 8192, (300,), device=DEV)
    if engine:
        w._main_grad, w._shadow = torch.zeros_like(w), w.bfloat16()

    def dx(rows, in_order):
        xr = x[:rows].clone().requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = ops.linear_cross_entropy(xr, w.requires_grad_(), t[:rows], in_order=in_order) * rows / 512  # (a power of two: no other rounding)
        return torch.autograd.grad(loss, xr)[0]

    a, b = dx(256, True), dx(128, True)
    torch.testing.assert_close(a[:128].float(), b.float(), rtol=2**-6, atol=0)  # softmax gradients scaled by 1 / rows before they are rounded
    assert not torch.equal(dx(256, False), dx(256, True))

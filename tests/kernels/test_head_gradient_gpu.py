"""The fused head's input gradient is one sum over the vocabulary, whatever the number of rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,width,vocab", [(4096, 768, 50304), (2048, 2048, 32000), (1000, 264, 8192)])
def test_rows_do_not_depend_on_how_they_are_cut_into_chunks(rows, width, vocab, dtype):
    """A chunk's rows are one product; few rows take other tiles than many, and add up the same products in the same order: equal bits."""
    from nanonemo_b200.ops.gemm import check_status
    from nanonemo_b200.ops.linear_ce import linear_ce_fwd

    torch.manual_seed(rows)
    x, w = torch.randn(rows, width, device=DEV).to(dtype), (torch.randn(vocab, width, device=DEV) * 0.02).to(dtype)
    t = torch.randint(0, vocab, (rows,), device=DEV)
    dW = torch.empty(vocab, width, device=DEV)
    got = {n: linear_ce_fwd(x, w, t, n, dW)[1] for n in (rows, rows // 2, 256)}  # (below 256 rows the softmax is summed in another order)
    check_status()
    last = rows % 256
    for n in (rows // 2, 256):
        assert torch.equal(got[n][: rows - last], got[rows][: rows - last])
    if dtype == torch.bfloat16:  # (in fp16 the gradients of a mean over thousands of rows are below its smallest normal number)
        p = (x.double() @ w.double().t()).softmax(-1)
        p[torch.arange(rows, device=DEV), t] -= 1
        ref = (p / rows) @ w.double()
        # logits, their gradients and the result are rounded to 16 bits once each, half of 2^-8 at most
        assert (got[rows].double() - ref).norm() <= 1.5 * 2**-8 * ref.norm()

"""Products of few rows (csrc/gemm_rows.cu): the same bits as the persistent kernels, from 16-bit and from fp32 weights."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
# rows and sizes at the edges of tiles (128 rows, 32 / 64 / 128 columns, 64 or 128 of K a stage) and of the rule that picks them
SIZES = [(1, 8, 8), (17, 40, 72), (127, 264, 136), (128, 768, 2048), (129, 4096, 768), (201, 1280, 768), (255, 1000, 520), (300, 104, 64), (896, 1280, 768), (897, 1280, 768),
         (2048, 768, 1024), (2100, 1104, 200),
         # an A of less than 128 KB and one of as much, in front of weights of 2^23 and 2^24 elements and a few more; wide weights
         (3, 2048, 4096), (3, 2048, 4104), (15, 4096, 4096), (16, 4096, 4096), (9, 4104, 2040), (31, 8192, 2048), (1, 9480, 1024), (64, 16384, 2048), (64, 16392, 2048)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_products_are_those_of_the_persistent_kernels(M, N, K, dtype):
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device=DEV).to(dtype), (torch.randn(N, K, device=DEV) * 0.05).to(dtype)
    for operand, mn in ((w, False), (w.t().contiguous(), True)):
        out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
        gemm(x, operand, b_mn=mn, out=out)
        check_status()
        assert torch.equal(out, gemm(x, operand, b_mn=mn, bn=128))  # (a tile width asked for: the persistent kernel)


@pytest.mark.parametrize("first,stride", [(0, 264), (8, 264)])
def test_strided_rows(first, stride):
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(0)
    x, w = (torch.randn(n, stride, device=DEV).bfloat16()[:, first : first + 200] for n in (150, 304))
    wide = torch.zeros(150, 400, device=DEV, dtype=torch.bfloat16)
    gemm(x, w, out=wide[:, 48:352])
    check_status()
    assert torch.equal(wide[:, 48:352], gemm(x.contiguous(), w.contiguous(), bn=128))
    assert not wide[:, :48].any() and not wide[:, 352:].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,T", [(1, 1), (64, 16), (130, 65), (201, 201), (512, 512)])
@pytest.mark.parametrize("hd,H,KVH", [(64, 12, 4), (128, 6, 2)])
def test_rope_and_swiglu_from_fp32_weights_are_the_unfused_operators(rows, T, hd, H, KVH, dtype):
    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache
    from nanonemo_b200.ops import _lib
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(rows + hd)
    n, B = _lib.native(), rows // T
    x = torch.randn(B, T, 768, device=DEV)
    wq, gu, down = (torch.randn(*s, device=DEV) * 0.05 for s in (((H + 2 * KVH) * hd, 768), (4096, 768), (768, 2048)))
    cos, sin = rope_cache(hd, 512, device=DEV)
    x2 = x.to(dtype).view(-1, 768)
    with torch.no_grad(), torch.autocast("cuda", dtype=dtype):
        y, z = ops.qkv_rope_attention(x, wq, cos, sin, H, KVH, hd), ops.mlp_swiglu(x, gu, down)
        check_status()
        qkv = gemm(x2, wq.to(dtype), bn=128)
        n.rope_packed(qkv, qkv, cos[:T].contiguous(), sin[:T].contiguous(), T, H + KVH, hd, 0, 1.0)
        heads = [t.transpose(1, 2) for t in qkv.view(B, T, -1, hd).split((H, KVH, KVH), dim=2)]
        assert torch.equal(y, ops.flash_attn(*heads).transpose(1, 2).reshape(B, T, -1))
        p, act = gemm(x2, gu.to(dtype), bn=128), torch.empty(B * T, 2048, device=DEV, dtype=dtype)
        n.swiglu_fwd(p[:, :2048], p[:, 2048:], act)
        assert torch.equal(z.view(-1, 768), gemm(act, down.to(dtype), bn=128))


@pytest.mark.parametrize("n_out,n_in", [(776, 520), (1032, 520), (8, 8), (40, 72), (136, 64), (4104, 1032)])  # (the input gradient's K: up to 1024 straight from fp32)
@pytest.mark.parametrize("rows", [1, 33, 201, 512, 4100])
def test_linear_from_its_fp32_weight_and_its_gradients(rows, n_out, n_in):
    """With and without gradients, few rows and many: the product of the cast weight; gradients as from the cast weight, too."""
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import gemm

    torch.manual_seed(rows)
    x, w = torch.randn(rows, n_in, device=DEV).bfloat16().requires_grad_(), (torch.randn(n_out, n_in, device=DEV) * 0.05).requires_grad_()
    y = ops.linear(x, w, impl="sm100")
    w16 = w.detach().bfloat16()
    assert torch.equal(y, gemm(x.detach(), w16, bn=128))
    with torch.no_grad():
        assert torch.equal(y, ops.linear(x, w, impl="sm100"))
    dy = torch.randn_like(y)
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    assert torch.equal(dx, gemm(dy, w16, b_mn=True, bn=128))
    ref = dy.double().t() @ x.detach().double()
    assert (dw.double() - ref).norm() <= 1e-5 * ref.norm()

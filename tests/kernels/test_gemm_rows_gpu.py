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


def _code(dtype):
    return {torch.bfloat16: 1, torch.float16: 2}[dtype]


def _launch(name, *args):
    """0: launched; 1: declined."""
    from nanonemo_b200.ops import _lib
    from nanonemo_b200.ops.gemm import status_tensor

    return _lib.call_rc(name, *(a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args), status_tensor(torch.device(DEV, 0)).data_ptr(), _lib.stream_ptr())


def _tables(T, hd):
    from nanonemo_b200.models.layers import rope_cache

    return tuple(t.contiguous() for t in rope_cache(hd, T, device=DEV))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (129, 136, 72), (300, 1280, 768)])
def test_every_tile_is_served_by_its_kernel(M, N, K, dtype):
    """The launchers asked for each tile and layout, so that no other route can answer."""
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(M)
    x, w = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV) * 0.05
    w16, ref = w.to(dtype), gemm(x, w.to(dtype), bn=128)
    for mn in (0, 1):
        for operand, name, tiles in ((w16, "nnb_gemm_rows", (32, 64)), (w, "nnb_gemm_rows_f32w", ((),))):
            stored = operand.t().contiguous() if mn else operand
            for g in tiles:
                out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
                assert _launch(name, x, stored, out, M, N, K, K, N if mn else K, N, mn, _code(dtype), *((g,) if g else ())) == 0
                check_status()
                assert torch.equal(out, ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,KVH,hd", [(1, 1, 1, 1, 64), (2, 65, 4, 1, 64), (3, 100, 3, 3, 128), (7, 37, 6, 2, 128)])
def test_rope_epilogue_is_the_product_and_the_rotation(B, T, H, KVH, hd, dtype):
    """16-bit and fp32 weights, each tile, the same bits as the two kernels."""
    from nanonemo_b200.ops import _lib
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(T)
    M, N, K, rot = B * T, (H + 2 * KVH) * hd, 328, (H + KVH) * hd
    x, w, (cos, sin) = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV) * 0.05, _tables(T, hd)
    ref = gemm(x, w.to(dtype), bn=128)
    _lib.native().rope_packed(ref, ref, cos, sin, T, H + KVH, hd, 0, 1.0)
    for operand, f32w, tiles in ((w.to(dtype), 0, (32, 64) if hd == 128 else (32,)), (w, 1, (16,))):
        for g in tiles:
            out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
            assert _launch("nnb_gemm_rows_rope", x, operand, out, cos, sin, M, N, K, K, K, N, T, rot, hd, _code(dtype), f32w, g) == 0
            check_status()
            assert torch.equal(out, ref)


@pytest.mark.parametrize("M,F", [(1, 16), (130, 176), (200, 2048), (512, 768)])  # (the last two: more 16-feature tiles than SMs, so 32 features)
def test_swiglu_epilogue_is_the_product_and_the_activation(M, F):
    from nanonemo_b200.ops import _lib
    from nanonemo_b200.ops.gemm import check_status, gemm

    torch.manual_seed(M)
    x, w = torch.randn(M, 520, device=DEV).bfloat16(), torch.randn(2 * F, 520, device=DEV) * 0.05
    p, ref, out = gemm(x, w.bfloat16(), bn=128), *(torch.full((M, F), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(2))
    _lib.native().swiglu_fwd(p[:, :F], p[:, F:], ref)
    assert _launch("nnb_gemm_rows_f32w_swiglu", x, w, out, M, F, 520, 520, 520, F, 1) == 0
    check_status()
    assert torch.equal(out, ref)


def test_operands_that_are_not_aligned_are_declined():
    M, N, K, hd = 66, 128, 72, 64
    base, wide, w32 = torch.randn(M * 80 + 8, device=DEV).bfloat16(), torch.randn(N * 80 + 8, device=DEV).bfloat16(), torch.randn(N * 136, device=DEV)
    x, w, f, (cos, sin) = base[: M * K], wide[: N * K], w32[: N * K], _tables(M, hd)
    odd = torch.zeros(cos.numel() + 1, device=DEV)[1:]
    out = torch.full((M * 136,), float("nan"), device=DEV, dtype=torch.bfloat16)  # (room for each call, should it be served after all)

    def plain(a=x, b=w, d=out, lda=K, ldw=K, ldd=N):
        return _launch("nnb_gemm_rows", a, b, d, M, N, K, lda, ldw, ldd, 0, 1, 32)

    def rope(a=x, b=w, c=cos, s=sin, f32w=0, ldw=K):
        return _launch("nnb_gemm_rows_rope", a, b, out, c, s, M, N, K, K, ldw, N, M, N, hd, 1, f32w, 32)

    assert [plain(a=base[1:]), plain(b=wide[4:]), plain(d=out[1:]), plain(lda=76), plain(ldw=74), plain(ldd=132)] == [1] * 6
    assert [rope(a=base[1:]), rope(b=wide[2:]), rope(c=odd), rope(s=odd), rope(ldw=74), rope(b=w32[1:], f32w=1), rope(b=f, f32w=1, ldw=74)] == [1] * 7
    for mn in (0, 1):
        assert [_launch("nnb_gemm_rows_f32w", x, b, out, M, N, K, K, ldw, N, mn, 1) for b, ldw in ((w32[1:], N if mn else K), (f, 130))] == [1] * 2
    assert _launch("nnb_gemm_rows_f32w_swiglu", x, w32[1:], out, M, N // 2, K, K, K, N // 2, 1) == 1
    assert _launch("nnb_gemm_rows_f32w_swiglu", x, f, out, M, 56, K, K, K, 56, 1) == 1  # (features in tiles of 16)
    assert _launch("nnb_gemm_rows_f32w", x, f, out, M, N, K, K, K, N, 0, 1) == 0
    torch.cuda.synchronize()
    assert out.isnan().sum() == out.numel() - M * N  # nothing else was launched


def test_what_the_rule_does_not_serve_is_declined():
    from nanonemo_b200.ops import _lib

    lib = _lib.lib()
    assert lib.nnb_gemm_rows_f32w_serves(200, 768, 768, 0) == 1 and lib.nnb_gemm_rows_f32w_serves(200, 768, 768, 2) == 1
    M, N, K = 600, 64, 1032
    x, w, out = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(K, N, device=DEV), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    assert lib.nnb_gemm_rows_f32w_serves(M, N, K, 2) == 0
    assert _launch("nnb_gemm_rows_f32w", x, w, out, M, N, K, K, N, N, 1, 1) == 1

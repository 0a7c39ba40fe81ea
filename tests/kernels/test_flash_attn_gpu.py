"""FlashAttention (tcgen05) against PyTorch attention in fp32: MHA / GQA, odd T, hd 64 / 128."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ref(q, k, v):
    group = q.shape[1] // k.shape[1]
    qf, kf, vf = q.float(), k.float().repeat_interleave(group, 1), v.float().repeat_interleave(group, 1)
    T = q.shape[2]
    s = qf @ kf.transpose(-1, -2) / q.shape[-1] ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(T, T, dtype=torch.bool, device=q.device), 1), float("-inf"))
    return torch.softmax(s, -1) @ vf


@pytest.mark.parametrize("B,H,KVH,T,hd", [(1, 1, 1, 128, 64), (2, 4, 2, 256, 64), (1, 12, 4, 1024, 64), (2, 3, 1, 200, 64),
                                          (1, 2, 2, 37, 64), (1, 4, 1, 384, 128), (2, 2, 2, 100, 128), (1, 2, 1, 640, 64)])
def test_forward_matches_reference(B, H, KVH, T, hd):
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(T + hd)
    q = torch.randn(B, H, T, hd, device=DEV).bfloat16()
    k = torch.randn(B, KVH, T, hd, device=DEV).bfloat16()
    v = torch.randn(B, KVH, T, hd, device=DEV).bfloat16()
    out = ops.flash_attn(q, k, v)
    check_status()
    assert out.shape == (B, H, T, hd)
    torch.testing.assert_close(out.float(), _ref(q, k, v), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T", [(74, 64), (75, 65), (300, 1), (150, 17), (101, 129), (40, 300), (20, 1024)])
def test_forward_of_a_grid_in_several_waves_is_that_of_its_sequences(B, T, hd):
    """Blocks that are running take over blocks that have not started: each sequence comes out as in a call of its own (one wave), bit for bit."""
    from nanonemo_b200.ops.attention import fwd_raw
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(B + T)
    H, KVH = 4, 2
    q, k, v = (torch.randn(B, T, h, hd, device=DEV).bfloat16() for h in (H, KVH, KVH))
    o = torch.full_like(q, float("nan"))
    lse = fwd_raw(q, k, v, o, hd**-0.5)
    check_status()
    for b in sorted({0, 1, B // 3, B // 2, B - 2, B - 1}):
        alone = torch.full_like(o[b : b + 1], float("nan"))
        lse_alone = fwd_raw(q[b : b + 1], k[b : b + 1], v[b : b + 1], alone, hd**-0.5)
        assert torch.equal(o[b : b + 1], alone) and torch.equal(lse[b : b + 1], lse_alone)
    assert torch.isfinite(o).all() and torch.isfinite(lse).all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T", [(75, 64), (74, 65), (160, 1), (90, 17), (50, 129), (27, 300), (10, 1024)])
def test_backward_of_a_grid_in_several_waves_is_that_of_its_sequences(B, T, hd):
    """dK and dV of a sequence, summed in the order of its queries, are the same bits in a large call and alone; dQ is reduce-added in the order of
    arrival, fp32 sums rounded once to 16 bits: at most two neighbouring values apart."""
    from nanonemo_b200.ops.attention import bwd_raw, fwd_raw
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(B + T)
    H, KVH = 4, 2
    q, k, v, do = (torch.randn(B, T, h, hd, device=DEV).bfloat16() for h in (H, KVH, KVH, H))
    o = torch.empty_like(q)
    lse = fwd_raw(q, k, v, o, hd**-0.5)
    got = [torch.full_like(t, float("nan")) for t in (q, k, v)]
    bwd_raw(q, k, v, o, lse, do, *got, hd**-0.5, in_order=True)
    check_status()
    for b in sorted({0, 1, B // 3, B // 2, B - 2, B - 1}):
        at = slice(b, b + 1)
        alone = [torch.full_like(t[at], float("nan")) for t in (q, k, v)]
        bwd_raw(q[at], k[at], v[at], o[at], lse[at].contiguous(), do[at], *alone, hd**-0.5, in_order=True)
        assert torch.equal(got[1][at], alone[1]) and torch.equal(got[2][at], alone[2])
        torch.testing.assert_close(got[0][at].float(), alone[0].float(), rtol=2**-7, atol=1e-5)
    assert all(torch.isfinite(t).all() for t in got)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T", [(75, 65), (150, 1), (38, 129), (25, 300), (10, 1000)])
def test_packed_backward_with_inverse_rope_of_a_grid_in_several_waves(B, T, dtype):
    """What a training step calls: gradients of the packed projection before its rotation. Key tiles follow one another in a CTA, each with rotations of its
    own: dK and dV of a sequence are the bits of a call of its own, and the rotated gradients of the same call without tables."""
    from nanonemo_b200.models.layers import rope_cache
    from nanonemo_b200.ops import rope
    from nanonemo_b200.ops.attention import bwd_raw, fwd_raw
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(B + T)
    H, KVH, hd = 4, 2, 64
    heads, cols = (H, KVH, KVH), (H + 2 * KVH) * hd
    cos, sin = (t.contiguous() for t in rope_cache(hd, T, device=DEV))
    qkv, do = torch.randn(B, T, cols, device=DEV).to(dtype), torch.randn(B, T, H, hd, device=DEV).to(dtype)

    def split(t):
        return t.view(t.shape[0], T, -1, hd).split(heads, dim=2)

    def backward(b0, b1, **tables):
        at = slice(b0, b1)
        o, g = torch.empty_like(do[at]), torch.full_like(qkv[at], float("nan"))
        lse = fwd_raw(*split(qkv[at]), o, hd**-0.5)
        bwd_raw(*split(qkv[at]), o, lse, do[at], *split(g), hd**-0.5, in_order=True, **tables)
        check_status()
        return g

    tables = dict(rope_cos=cos, rope_sin=sin)
    got, plain = backward(0, B, **tables), backward(0, B)
    kv = H * hd
    for b in sorted({0, 1, B // 3, B // 2, B - 2, B - 1}):
        alone = backward(b, b + 1, **tables)
        assert torch.equal(got[b : b + 1, :, kv:], alone[:, :, kv:])
        torch.testing.assert_close(got[b : b + 1, :, :kv].float(), alone[:, :, :kv].float(), rtol=2**-7, atol=1e-5)  # (dQ: added in the order of arrival)
    assert torch.equal(got[:, :, kv + KVH * hd :], plain[:, :, kv + KVH * hd :])  # dV is not rotated
    ref = torch.empty_like(plain)
    rope.rope_packed_raw(plain.view(B * T, cols), ref.view(B * T, cols), cos, sin, T, H + KVH, hd, KVH * hd, -1.0)
    # rounded once, against once before and once after the rotation: half a unit of either partner, and half a unit of each result (dQ: its sums differ, too)
    unit = 2**-8 if dtype == torch.bfloat16 else 2**-11
    pair = plain.float().view(B * T, -1, 2, hd // 2).abs().sum(2, keepdim=True).expand(-1, -1, 2, -1).reshape(B, T, cols)
    off = (got.float() - ref.float()).abs()
    assert (off[:, :, kv:] <= (unit * (pair + ref.float().abs()) + 1e-6)[:, :, kv:]).all()
    assert (off[:, :, :kv] <= (2 * unit * (pair + ref.float().abs()) + 1e-5)[:, :, :kv]).all()


def test_future_keys_do_not_leak():
    from nanonemo_b200 import ops

    torch.manual_seed(0)
    q = torch.randn(1, 2, 256, 64, device=DEV).bfloat16()
    k = torch.randn(1, 2, 256, 64, device=DEV).bfloat16()
    v = torch.randn(1, 2, 256, 64, device=DEV).bfloat16()
    a = ops.flash_attn(q, k, v)
    k2, v2 = k.clone(), v.clone()
    k2[:, :, 150:] = 100.0
    v2[:, :, 150:] = -100.0
    b = ops.flash_attn(q, k2, v2)
    assert torch.equal(a[:, :, :150], b[:, :, :150])  # bitwise: positions before 150 never read later keys


def test_packed_forward_and_backward():
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(1)
    B, T, H, KVH, hd = 2, 384, 6, 2, 64
    qkv = torch.randn(B, T, (H + 2 * KVH) * hd, device=DEV).bfloat16().requires_grad_()
    out = ops.attention_packed(qkv, H, KVH, hd, impl="sm100")
    ref_in = qkv.detach().float().requires_grad_()
    ref = ops.attention_packed(ref_in, H, KVH, hd, impl="torch")
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)
    g = torch.randn_like(ref)
    out.backward(g.bfloat16())
    ref.backward(g)
    check_status()
    torch.testing.assert_close(qkv.grad.float(), ref_in.grad, rtol=5e-2, atol=5e-2)


@pytest.mark.parametrize("B,H,KVH,T,hd", [(1, 2, 1, 256, 64), (2, 6, 2, 512, 64), (1, 3, 3, 200, 64), (1, 4, 2, 1024, 64),
                                          (1, 1, 1, 128, 128), (1, 2, 1, 256, 128), (2, 4, 2, 512, 128), (1, 3, 3, 200, 128),
                                          (1, 4, 1, 1024, 128), (1, 2, 2, 37, 128)])
def test_backward_matches_reference(B, H, KVH, T, hd):
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(2)
    q = torch.randn(B, H, T, hd, device=DEV).bfloat16().requires_grad_()
    k = torch.randn(B, KVH, T, hd, device=DEV).bfloat16().requires_grad_()
    v = torch.randn(B, KVH, T, hd, device=DEV).bfloat16().requires_grad_()
    out = ops.flash_attn(q, k, v)
    g = torch.randn(B, H, T, hd, device=DEV)
    out.backward(g.bfloat16())
    check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    _ref(qr, kr, vr).backward(g.bfloat16().float())
    for got, want, name in ((q.grad, qr.grad, "dq"), (k.grad, kr.grad, "dk"), (v.grad, vr.grad, "dv")):
        err = (got.float() - want).abs().max().item()
        assert err <= 3e-2 * want.abs().max().item() + 2e-2, f"{name}: max err {err}"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,H,KVH,T", [(1, 1, 1, 1), (2, 2, 2, 2), (1, 3, 1, 63), (1, 2, 1, 65), (2, 5, 1, 127), (1, 3, 3, 129), (1, 7, 1, 257),
                                       (3, 2, 1, 385), (1, 12, 1, 640)])
def test_forward_and_backward_at_the_edges_of_the_pipelines(B, H, KVH, T, hd):
    """One visit, two, as many as the rings have stages and one more; one row, and one row or key past a tile; many query heads per
    KV head. 16-bit operands: each of P, dS and the outputs is rounded to 8 bits (2^-9 each), so 1 % in the 2-norm."""
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(T)
    q, k, v = (torch.randn(B, h, T, hd, device=DEV).bfloat16().requires_grad_() for h in (H, KVH, KVH))
    g = torch.randn(B, H, T, hd, device=DEV).bfloat16()
    out = ops.flash_attn(q, k, v)
    grads = torch.autograd.grad(out, (q, k, v), g)
    check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = _ref(qr, kr, vr)
    # one key: dS is zero up to the rounding of P and O, so dQ and dK are measured against dV's size
    refs = torch.autograd.grad(ref, (qr, kr, vr), g.float())
    floor = refs[2].norm() * 1e-3
    for got, want in zip((out, *grads), (ref, *refs)):
        assert (got.float() - want).norm() <= 1e-2 * want.norm() + floor


@pytest.mark.parametrize("B,H,KVH,T,hd", [(2, 4, 2, 256, 64), (1, 3, 1, 200, 64), (1, 4, 1, 384, 128), (1, 2, 2, 37, 128)])
def test_fp16_operands_run_natively(B, H, KVH, T, hd):
    """fp16 q / k / v go to the tensor cores as fp16 (no bf16 detour): forward and the three gradients against the fp32
    reference, with the tighter tolerance the 10-bit mantissa allows."""
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(3)
    q = torch.randn(B, H, T, hd, device=DEV).half().requires_grad_()
    k = torch.randn(B, KVH, T, hd, device=DEV).half().requires_grad_()
    v = torch.randn(B, KVH, T, hd, device=DEV).half().requires_grad_()
    out = ops.flash_attn(q, k, v)
    assert out.dtype == torch.float16
    g = torch.randn(B, H, T, hd, device=DEV).half()
    out.backward(g)
    check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = _ref(qr, kr, vr)
    ref.backward(g.float())
    torch.testing.assert_close(out.float(), ref, rtol=4e-3, atol=4e-3)
    for got, want, name in ((q.grad, qr.grad, "dq"), (k.grad, kr.grad, "dk"), (v.grad, vr.grad, "dv")):
        assert got.dtype == torch.float16
        err = (got.float() - want).abs().max().item()
        assert err <= 6e-3 * want.abs().max().item() + 4e-3, f"{name}: max err {err}"


def test_mixed_operand_dtypes_are_refused():
    from nanonemo_b200.ops import attention

    q = torch.randn(1, 128, 1, 64, device=DEV).half()
    k = torch.randn(1, 128, 1, 64, device=DEV).bfloat16()
    with pytest.raises(TypeError):
        attention.fwd_raw(q, k, k, torch.empty_like(q), 0.125)


@pytest.mark.parametrize("B,T,H,KVH", [(1, 128, 1, 1), (1, 1, 3, 3), (1, 300, 2, 2), (2, 333, 12, 4), (1, 1000, 6, 1), (40, 130, 8, 4), (3, 1153, 5, 5)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hd", [64, 128])
def test_backward_whose_key_tiles_are_shared_by_several_ctas(B, T, H, KVH, dtype, hd):
    """One, two and four CTAs a key tile, some of them without a visit: dK and dV are those of fp32 math to the rounding of 16-bit
    probabilities, the same in every run, and nothing beyond the last key is written."""
    from nanonemo_b200.ops import attention
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(T + H)
    q, k, v, do = (torch.randn(B, T, n, hd, device="cuda").to(dtype) for n in (H, KVH, KVH, H))
    o, scale = torch.empty_like(q), hd ** -0.5
    lse = attention.fwd_raw(q, k, v, o, scale)
    got = []
    for _ in range(2):
        pad = torch.full((B, T + 1, KVH, 2, hd), 7.0, device="cuda", dtype=dtype)  # dK and dV interleaved, a row more than they need
        dq, dk, dv = torch.empty_like(q), pad[:, :T, :, 0], pad[:, :T, :, 1]
        attention.bwd_raw(q, k, v, o, lse, do, dq, dk, dv, scale)
        check_status()
        assert (pad[:, T] == 7).all()
        got.append((dq, dk.clone(), dv.clone()))
    assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][2], got[1][2])
    qf, kf, vf = (t.float().transpose(1, 2).requires_grad_() for t in (q, k, v))
    group = H // KVH
    s = (qf @ kf.repeat_interleave(group, 1).transpose(-1, -2)) * scale
    p = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf")).softmax(-1)
    refs = torch.autograd.grad(p @ vf.repeat_interleave(group, 1), (qf, kf, vf), do.float().transpose(1, 2))
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11  # P, dS, O and the results are each rounded to half of this at most
    for g, r in zip(got[0], refs):
        r = r.transpose(1, 2)
        size = max(r.norm().item(), 1e-3 * r.numel() ** 0.5)  # (one query: its gradients vanish, dP and D cancel to their roundings)
        assert (g.float() - r).norm().item() <= 2 * eps * size


@pytest.mark.parametrize("B,T,H,KVH,hd", [(4, 1001, 12, 4, 64), (4, 513, 16, 4, 128)])
def test_backward_whose_key_tiles_are_shared_by_two_ctas(B, T, H, KVH, hd):
    """Odd T: the last tile ends inside a warp of the exchange."""
    from nanonemo_b200.ops import _lib

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _lib.lib().nnb_flash_bwd_split(T, 128 if hd == 64 else 64, ctypes.c_longlong(B * KVH), H // KVH, sms) == 2
    test_backward_whose_key_tiles_are_shared_by_several_ctas(B, T, H, KVH, torch.bfloat16, hd)


@pytest.mark.parametrize("B,T,hd", [(32, 255, 128), (32, 256, 128), (64, 255, 64), (64, 256, 64)])
def test_backward_on_both_sides_of_the_size_from_which_its_pre_pass_is_launched_in_order(B, T, hd):
    test_backward_whose_key_tiles_are_shared_by_several_ctas(B, T, 16, 4, torch.float16, hd)


@pytest.mark.parametrize("H,KVH,T,hd", [(12, 4, 333, 64), (6, 1, 1000, 64), (16, 4, 333, 128)])
@pytest.mark.parametrize("direct_route", [False, True])
def test_packed_attention_in_order_sums_a_sequence_the_same_way_in_calls_of_any_size(monkeypatch, H, KVH, T, hd, direct_route):
    """dK and dV of one sequence alone, where key tiles would be shared, against the same sequence in a batch that fills the GPU."""
    from nanonemo_b200 import ops
    from nanonemo_b200.ops import _lib, direct

    monkeypatch.setattr(direct, "ENABLED", direct_route)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = -(-2 * sms // (KVH * -(-T // 128)))
    split = lambda b: _lib.lib().nnb_flash_bwd_split(T, 128 if hd == 64 else 64, ctypes.c_longlong(b * KVH), H // KVH, sms)  # noqa: E731
    assert split(1) > 1 == split(B)
    torch.manual_seed(T)
    qkv, do = torch.randn(B, T, (H + 2 * KVH) * hd, device=DEV).bfloat16(), torch.randn(B, T, H * hd, device=DEV).bfloat16()

    def grad(b, in_order):
        x = qkv[:b].clone().requires_grad_()
        (g,) = torch.autograd.grad(ops.attention_packed(x, H, KVH, hd, impl="sm100", in_order=in_order), x, do[:b])
        return g[0, :, H * hd:]

    full, alone, shared = grad(B, True), grad(1, True), grad(1, False)
    assert torch.equal(alone, full)
    assert (shared.float() - full.float()).norm() <= 2 ** -8 * full.float().norm()  # (two roundings to 16 bits of the same sums)

"""MXFP8 quantiser kernels and the fp8 linear: block-scale rules, round trip, and loss tracking vs bf16."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_quantise_matches_reference_rules():
    from nanonemo_b200 import fp8

    torch.manual_seed(0)
    x = (torch.randn(64, 256, device="cuda") * torch.logspace(-3, 2, 256, device="cuda")).bfloat16()
    q, s = fp8.quantize(x)
    assert q.shape == (64, 256) and s.shape == (64, 8)
    blocks = x.float().view(64, 8, 32)
    amax = blocks.abs().amax(-1)
    expect = (torch.floor(torch.log2(amax)) - 8 + 127).clamp(0, 254)
    assert torch.equal(s.float(), expect)
    deq = fp8.dequantize(q, s)
    torch.testing.assert_close(deq, fp8.fake_quant(x).float(), rtol=0, atol=0)
    rel = (deq - x.float()).abs() / amax.repeat_interleave(32, 1)
    # e4m3: 3 mantissa bits (half an ulp of the top binade = 1/16 of the block maximum) and, per the OCP MX rule
    # scale = 2^(floor(log2 amax) - 8), block maxima that land in (448, 512) saturate to 448 (at most 1/8 off)
    assert rel.max() < 0.15 and rel.mean() < 0.01


def test_fp8_linear_tracks_bf16():
    from nanonemo_b200 import fp8
    from nanonemo_b200.ops.gemm import linear_sm100

    torch.manual_seed(1)
    x = torch.randn(256, 768, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(1280, 768, device="cuda") * 0.02).requires_grad_()
    g = torch.randn(256, 1280, device="cuda", dtype=torch.bfloat16)
    with fp8.fp8_context("delayed")():
        y8 = fp8.linear_mxfp8(x, w)
    y8.backward(g)
    gx8, gw8 = x.grad.clone(), w.grad.clone()
    x.grad = w.grad = None
    y16 = linear_sm100(x, w)
    y16.backward(g)
    for a, b in ((y8, y16), (gx8, x.grad), (gw8, w.grad)):
        err = (a.float() - b.float()).norm() / b.float().norm()
        assert err < 6e-2, err
    assert fp8.linear_mxfp8(x, w).sub(y16).abs().max() == 0  # outside the context: the plain 16-bit GEMM


def test_fp8_precision_trains(tmp_path):
    from nanonemo_b200.models.config import ModelConfig
    from nanonemo_b200.train.config import TrainConfig
    from nanonemo_b200.train.trainer import train

    losses = {}
    for prec, lin in (("bf16", "sm100"), ("fp8", "mxfp8")):
        mc = ModelConfig.sm100(n_layers=2, d_model=256, n_heads=4, n_kv_heads=2, d_ff=512, max_seq_len=256, linear_impl=lin)
        tc = TrainConfig(data_dir="synthetic", out_dir=str(tmp_path / prec), seq_len=256, micro_batch=8, global_batch_tokens=2048,
                         total_tokens=2048 * 10, peak_lr=1e-3, precision=prec, eval_every=100, eval_batches=1)
        losses[prec] = [r["loss"] for r in train(mc, tc, device="cuda:0") if "loss" in r]
    assert losses["fp8"] == pytest.approx(losses["bf16"], abs=2e-2)


def _dequant_chunked(q, sf):
    from nanonemo_b200 import fp8

    return fp8.dequantize(q, fp8.scales_to_plain(sf, q.shape[0], q.shape[1]).contiguous())


def test_tile_quantiser_matches_the_plain_quantiser_both_ways():
    from nanonemo_b200 import fp8

    torch.manual_seed(2)
    x = (torch.randn(384, 256, device="cuda") * torch.logspace(-2, 2, 256, device="cuda")).bfloat16()
    q, sf, qt, sft = fp8.quantize_mx(x, True, True)
    q_ref, s_ref = fp8.quantize(x)
    assert torch.equal(q, q_ref) and torch.equal(fp8.scales_to_plain(sf, 384, 256), s_ref)
    qt_ref, st_ref = fp8.quantize(x.t().contiguous())
    assert torch.equal(qt, qt_ref) and torch.equal(fp8.scales_to_plain(sft, 256, 384), st_ref)
    only_t = fp8.quantize_mx(x, False, True)
    assert only_t[0] is None and torch.equal(only_t[2], qt_ref)


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 384, 512), (1024, 2304, 768), (512, 768, 2048)])
def test_block_scaled_gemm_matches_fp32_product_of_the_quantised_values(M, N, K):
    """The tensor-core path must multiply exactly the MXFP8 values: compare with an fp32 matmul of the dequantised operands."""
    from nanonemo_b200 import fp8
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(M + N + K)
    # per-column magnitudes spread over several binades so that a wrong scale (row, k-block or byte) cannot go unnoticed
    a = (torch.randn(M, K, device="cuda") * torch.logspace(-2, 1, K, device="cuda")[torch.randperm(K, device="cuda")]).bfloat16()
    b = (torch.randn(N, K, device="cuda") * torch.logspace(-1, 1, N, device="cuda").unsqueeze(1)).bfloat16()
    aq, asf, _, _ = fp8.quantize_mx(a)
    bq, bsf, _, _ = fp8.quantize_mx(b)
    want = _dequant_chunked(aq, asf) @ _dequant_chunked(bq, bsf).t()
    got32 = fp8.gemm_mxfp8(aq, asf, bq, bsf, out_dtype=torch.float32)
    got16 = fp8.gemm_mxfp8(aq, asf, bq, bsf)
    check_status()
    scale = want.abs().max().item()
    assert (got32 - want).abs().max().item() <= 2e-5 * scale * (K / 128) ** 0.5 + 1e-6
    assert (got16.float() - want).abs().max().item() <= 1e-2 * scale
    acc = torch.ones(M, N, device="cuda")
    fp8.gemm_mxfp8(aq, asf, bq, bsf, out=acc, accumulate=True, k_splits=min(2, K // 128))
    check_status()
    assert (acc - 1.0 - want).abs().max().item() <= 2e-5 * scale * (K / 128) ** 0.5 + 1e-5


@pytest.mark.parametrize("M,N,K,bound", [(2048, 2048, 8192, 2e-7), (1280, 768, 8192, 1.2e-7), (2048, 5632, 4224, 1.2e-7)])
@pytest.mark.parametrize("accumulate", [True, False])
def test_block_scaled_fp32_products_keep_their_accumulation_chains_short(M, N, K, bound, accumulate):
    """One chain over K = 8192 is 4.7e-7 off the product of the quantised values (2-norm, 64 bits), chains of 16 k-blocks 1.1e-7; the
    fp32 sums add less than 1e-7. K = 4224 leaves a shorter last chain."""
    from nanonemo_b200 import fp8
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(M + K)
    a, b = (torch.randn(r, K, device="cuda", dtype=torch.bfloat16) for r in (M, N))
    (aq, asf, _, _), (bq, bsf, _, _) = fp8.quantize_mx(a), fp8.quantize_mx(b)
    out = torch.zeros(M, N, device="cuda")
    fp8.gemm_mxfp8(aq, asf, bq, bsf, out=out, accumulate=accumulate)
    check_status()
    ref = _dequant_chunked(aq, asf).double() @ _dequant_chunked(bq, bsf).double().t()
    assert (out.double() - ref).norm() <= bound * ref.norm()


def test_fp8_linear_tensor_core_path_equals_the_emulation(monkeypatch):
    from nanonemo_b200 import fp8

    torch.manual_seed(3)
    x = torch.randn(512, 768, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(1280, 768, device="cuda") * 0.02).requires_grad_()
    g = torch.randn(512, 1280, device="cuda", dtype=torch.bfloat16)
    out = {}
    for emulate in ("0", "1"):
        monkeypatch.setenv("NANONEMO_FP8_EMULATE", emulate)
        x.grad = w.grad = None
        with fp8.fp8_context("mxfp8")():
            y = fp8.linear_mxfp8(x, w)
        y.backward(g)
        out[emulate] = (y.detach().float(), x.grad.float().clone(), w.grad.float().clone())
    for real, emu in zip(out["0"], out["1"]):
        # same quantised values; only the accumulation order and the output rounding differ
        assert (real - emu).abs().max().item() <= 1e-2 * emu.abs().max().item()


def test_attention_of_a_block_scaled_model_sums_its_gradients_in_order(monkeypatch):
    from nanonemo_b200 import ops
    from nanonemo_b200.models.config import ModelConfig
    from nanonemo_b200.models.layers import Attention, rope_cache

    seen, real = [], ops.attention_packed
    monkeypatch.setattr(ops, "attention_packed", lambda *a, **k: seen.append(k["in_order"]) or real(*a, **k))
    cos, sin = rope_cache(64, 128, device="cuda")
    for impl, fuse in (("mxfp8", True), ("sm100", False)):
        cfg = ModelConfig.sm100(n_layers=1, d_model=256, n_heads=4, n_kv_heads=2, d_ff=512, max_seq_len=128, linear_impl=impl, fuse_epilogues=fuse)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            Attention(cfg).cuda()(torch.randn(1, 128, 256, device="cuda"), cos, sin)
    assert seen == [True, False]


@pytest.mark.parametrize("batch,seq", [(1, 256), (8, 1024)])
def test_gradients_of_an_fp8_step_are_those_of_the_bf16_engine_to_the_operands_rounding(batch, seq):
    """First moments after one step. A block-scaled product is within 6e-2 of the 16-bit one (test_fp8_linear_tracks_bf16); the gradient of
    a weight has at most the 8 linears of two layers forward and 8 backward before it, whose roundings are independent."""
    from nanonemo_b200 import parallel
    from nanonemo_b200.models.config import ModelConfig
    from nanonemo_b200.train.config import TrainConfig
    from nanonemo_b200.train.optim import build_optimizer
    from nanonemo_b200.train.trainer import build_parallel, train_step

    g = torch.Generator(device="cuda").manual_seed(0)
    window = torch.randint(0, 500, (batch, seq + 1), generator=g, device="cuda")

    class Source:
        micro_step = 0

        def next_batch(self):
            self.micro_step += 1
            return window[:, :-1], window[:, 1:]

    moments = []
    for precision, linear in (("bf16", "sm100"), ("fp8", "mxfp8")):
        mc = ModelConfig.sm100(n_layers=2, d_model=256, n_heads=4, n_kv_heads=2, d_ff=512, max_seq_len=seq, vocab_size=512, linear_impl=linear)
        tc = TrainConfig(data_dir="synthetic", seq_len=seq, micro_batch=batch, precision=precision, global_batch_tokens=batch * seq)
        torch.manual_seed(0)
        with torch.device("cuda"):
            strategy = build_parallel(mc, tc, parallel.Dist(device="cuda:0"))
        opt = build_optimizer(strategy.model, 1e-4, 0.1, store=strategy.store)
        train_step(strategy, opt, Source(), 1, 1e9, torch.bfloat16, None, host_sync=False)
        moments.append(strategy.store.exp_avg.clone())
    off = (moments[1] - moments[0]).norm() / moments[0].norm()
    assert 0 < off <= 6e-2 * 16 ** 0.5


@pytest.mark.parametrize("M,F", [(128, 128), (384, 640), (256, 2048)])
def test_activation_in_the_quantiser_gives_the_bytes_of_activation_and_quantiser(M, F):
    from nanonemo_b200 import fp8
    from nanonemo_b200.ops import _lib, swiglu_act

    torch.manual_seed(0)
    wide = torch.randn(M, 2 * F + 8, device="cuda").bfloat16() * torch.logspace(-3, 2, M, device="cuda").bfloat16()[:, None]
    wide[0, :32], wide[1, 5], wide[2, F + 7] = 0.0, 3e38, float("inf")
    gu, dact = wide[:, : 2 * F], torch.randn(M, F, device="cuda").bfloat16()  # (rows further apart than they are long)
    act, dgu = torch.empty(M, F, device="cuda", dtype=torch.bfloat16), torch.empty(M, 2 * F, device="cuda", dtype=torch.bfloat16)
    swiglu_act.fwd_raw(gu[:, :F], gu[:, F:], act)
    swiglu_act.bwd_raw(dact, gu[:, :F], gu[:, F:], dgu[:, :F], dgu[:, F:])
    for row, col in ((True, True), (True, False), (False, True)):
        for got, want in ((_lib.native().swiglu_mx(gu, row, col), fp8.quantize_mx(act, row, col)), (_lib.native().swiglu_bwd_mx(dact, gu, row, col), fp8.quantize_mx(dgu, row, col))):
            for a, b in zip(got, want):
                assert (a is None and b is None) or torch.equal(a, b)


@pytest.mark.parametrize("trained", ["xgd", "x", "g", "d", "xd", ""])  # the input, the gate and up projection, the down projection
def test_block_scaled_mlp_in_one_node_is_that_of_its_linears(trained):
    from nanonemo_b200 import fp8
    from nanonemo_b200.models.config import ModelConfig
    from nanonemo_b200.models.layers import MLP

    torch.manual_seed(0)
    mlp = MLP(ModelConfig.sm100(n_layers=1, vocab_size=512, linear_impl="mxfp8")).to("cuda")
    told = []
    for w, name in ((mlp.w_gu.weight, "g"), (mlp.w_down.weight, "d")):
        w.requires_grad_(name in trained)
        w._shadow, w._main_grad = w.detach().bfloat16(), torch.zeros_like(w)
        w._grad_ready_cb = lambda p, direct, name=name: told.append(name)
    x0, dy = torch.randn(2, 128, mlp.w_gu.in_features, device="cuda").bfloat16(), torch.randn(2, 128, mlp.w_gu.in_features, device="cuda").bfloat16()

    def run():
        x = x0.clone().requires_grad_("x" in trained)
        for w in (mlp.w_gu.weight, mlp.w_down.weight):
            w._main_grad.zero_()
        told.clear()
        with fp8.fp8_context()():
            y = mlp(x)
        if trained:
            y.backward(dy)
        return [y.detach(), x.grad, mlp.w_gu.weight._main_grad.clone(), mlp.w_down.weight._main_grad.clone()], list(told), type(y.grad_fn).__name__

    one, told_one, node = run()
    hook = mlp.w_down.register_forward_hook(lambda *a: None)  # somebody watches the linears
    two, told_two, node_two = run()
    hook.remove()
    assert told_one == told_two and (not trained or ("MLP" in node and "MLP" not in node_two))
    for a, b in zip(one, two):
        assert (a is None and b is None) or torch.equal(a, b)

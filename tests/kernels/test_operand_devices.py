"""A kernel that gets a host address faults, and the process loses its context: such operands are refused before a launch."""

import pytest
import torch

from nanonemo_b200.csrc import build
from nanonemo_b200.ops import _lib

BF = torch.bfloat16


@pytest.fixture(scope="module")
def native():
    if not (build.LIB.exists() and build.NATIVE.exists()):
        pytest.skip("kernel library not built")
    return _lib.native()


def test_raw_launches_refuse_host_tensors(native):
    x, w, f = torch.ones(256, 128, dtype=BF), torch.ones(256, 128, dtype=BF), torch.ones(256, 128)
    q = torch.ones(1, 64, 2, 64, dtype=BF)
    u8 = torch.ones(128, 128, dtype=torch.uint8)
    calls = {
        "gemm": lambda: native.gemm(x, w, False, False, None, None, False, 0, 0, 0), "gemm_swiglu": lambda: native.gemm_swiglu(x, w),
        "gemm_swiglu_act": lambda: native.gemm_swiglu_act(x, w), "gemm_swiglu_bwd": lambda: native.gemm_swiglu_bwd(x, w, x), "gemm_rope": lambda: native.gemm_rope(x, w, f, f, 256, 128, 64),
        "rope_packed": lambda: native.rope_packed(x, x, f, f, 256, 2, 64, 0, 1.0), "swiglu_fwd": lambda: native.swiglu_fwd(x, x, x), "swiglu_bwd": lambda: native.swiglu_bwd(x, x, x, x, x),
        "rms_fwd": lambda: native.rms_fwd(x, None, f[0], 1e-5, BF), "rms_bwd": lambda: native.rms_bwd(x, f, f[:, 0], f[0], None, None, None, False),
        "flash_fwd": lambda: native.flash_fwd(q, q, q, q, 0.125), "flash_bwd": lambda: native.flash_bwd(q, q, q, q, f, q, q, q, q, 0.125, None, None, False),
        "quantize_mx": lambda: native.quantize_mx(x, True, True), "gemm_mxfp8": lambda: native.gemm_mxfp8(u8, u8, u8, u8, None, BF, False, 0),
    }
    for name, call in calls.items():
        with pytest.raises(AssertionError, match="cannot reach"):
            pytest.fail(f"{name}: {call()}")


def test_head_and_embedding_refuse_host_tensors():
    from nanonemo_b200.ops import embed, linear_ce

    x, w, t = torch.ones(256, 128, dtype=BF), torch.ones(512, 128, dtype=BF), torch.zeros(256, dtype=torch.long)
    for call in (lambda: linear_ce.linear_ce_fwd(x, w, t, 256, torch.empty(512, 128)), lambda: linear_ce.linear_ce_loss(x, w, t, 256),
                 lambda: embed.fwd_raw(t, w.float(), torch.float32), lambda: embed.bwd_raw(t, x, torch.zeros(512, 128))):
        with pytest.raises(AssertionError, match="cannot reach"):
            call()


@pytest.mark.gpu
def test_operators_refuse_a_weight_on_the_host():
    from nanonemo_b200 import ops

    x, w = torch.randn(300, 128, device="cuda"), torch.randn(256, 128)
    calls = [lambda: ops.linear(x, w, impl="sm100"), lambda: ops.add_rms_norm(x, None, torch.ones(128), 1e-5, impl="sm100"), lambda: ops.mlp_swiglu(x, w, torch.randn(128, 128)),
             lambda: ops.linear_cross_entropy(x, w, torch.zeros(300, dtype=torch.long, device="cuda")),
             lambda: ops.linear_cross_entropy(x, w.cuda(), torch.zeros(300, dtype=torch.long)),
             lambda: ops.flash_attn(torch.randn(1, 2, 64, 64, device="cuda").to(BF), torch.randn(1, 2, 64, 64).to(BF), torch.randn(1, 2, 64, 64).to(BF))]
    for call in calls:
        with pytest.raises((AssertionError, RuntimeError, ValueError)):
            call()
    torch.cuda.synchronize()  # nothing was launched that could have faulted
    assert ops.linear(x, w.cuda(), impl="sm100").isfinite().all()

"""Kernels that may start before their predecessor has finished (csrc/common.cuh: nnb_launch): chains of small dependent calls give what
they give when the device is idle between any two, launched eagerly and replayed from a graph."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _chain(rows, sync):
    """Every operator reads what the one before has just written, and several write over memory that was freed a moment ago."""
    from nanonemo_b200.ops import attention, embed, linear_ce, rmsnorm, rope, swiglu_act
    from nanonemo_b200.ops.gemm import gemm, gemm_rope, gemm_swiglu, gemm_swiglu_bwd

    g = torch.Generator(device=DEV).manual_seed(rows)

    def rnd(*shape, dt=torch.bfloat16, k=0.1):
        return (torch.randn(*shape, generator=g, device=DEV) * k).to(dt)

    def then(value):
        sync()
        return value

    d, F, H, hd, T = 128, 256, 2, 64, rows
    table, w, wq, wgu, wd = rnd(512, d, dt=torch.float32), 1 + rnd(d, dt=torch.float32), rnd(4 * hd, d), rnd(2 * F, d), rnd(d, F)
    cos, sin = rnd(T, hd // 2, dt=torch.float32, k=1.0), rnd(T, hd // 2, dt=torch.float32, k=1.0)
    idx = torch.randint(0, 512, (rows,), generator=g, device=DEV)
    half = torch.full((), 0.5, device=DEV)

    def run():
        out = []
        x, _ = then(embed.fwd_raw(idx, table, torch.float32))
        for _ in range(4):
            y, h, rstd = then(rmsnorm.fwd(x, None, w, 1e-5, torch.bfloat16))
            qkv = then(gemm_rope(y, wq, cos, sin, T, 3 * hd, hd))
            if qkv is None:
                qkv = then(gemm(y, wq))
                then(rope.rope_packed_raw(qkv, qkv, cos, sin, T, 3, hd, 0, 1.0))
            q, k, v = (qkv[:, a * hd:b * hd].view(1, T, b - a, hd) for a, b in ((0, 2), (2, 3), (3, 4)))
            o = torch.empty(1, T, H, hd, dtype=torch.bfloat16, device=DEV)
            lse = then(attention.fwd_raw(q, k, v, o, 0.125))
            do, dqkv = then(o * 1), torch.empty_like(qkv)
            then(attention.bwd_raw(q, k, v, o, lse, do, *(dqkv[:, a * hd:b * hd].view(1, T, b - a, hd) for a, b in ((0, 2), (2, 3), (3, 4))), 0.125))
            del do
            fused = then(gemm_swiglu(o.view(T, d), wgu))
            if fused is None:
                gu, act = then(gemm(o.view(T, d), wgu)), torch.empty(T, F, dtype=torch.bfloat16, device=DEV)
                then(swiglu_act.fwd_raw(gu[:, :F], gu[:, F:], act))
            else:
                gu, act = fused
            down = then(gemm(act, wd))
            dgu = then(gemm_swiglu_bwd(down, wd, gu))
            dw = then(gemm(down, act, a_mn=True, b_mn=True, out_dtype=torch.float32))
            dx, dd, dn = then(rmsnorm.bwd(down, h, rstd, w, x, torch.bfloat16))
            scaled = then(linear_ce.scale(dx, half))
            x = then(x + down.float())
            out += [t for t in (y, o, gu, act, down, dgu, dw, dx, dd, dn, scaled, dqkv[:, 2 * hd:]) if t is not None]
        return out

    return run


def _same(got, ref):
    assert len(got) == len(ref)
    for a, b in zip(got, ref):  # (weight gradients may be cut into splits that are added in any order)
        assert torch.equal(a, b) if a.dtype != torch.float32 else torch.allclose(a, b, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rows", [64, 200, 512, 9600])  # (the last one: the projection by the CTA-pair kernel)
def test_dependent_kernels_see_what_their_predecessors_wrote(rows):
    ref = _chain(rows, torch.cuda.synchronize)()
    run = _chain(rows, lambda: None)
    for _ in range(20):
        _same(run(), ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        run()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            got = run()
    for _ in range(10):
        graph.replay()
    torch.cuda.synchronize()
    _same(got, ref)


def test_two_streams_with_events_between_them():
    """Work of another stream that an event orders before a kernel, and after one."""
    from nanonemo_b200.ops.gemm import gemm

    a, b = torch.randn(512, 256, device=DEV).bfloat16(), torch.randn(256, 256, device=DEV).bfloat16()
    ref = gemm(gemm(a, b), b)
    side = torch.cuda.Stream()
    for _ in range(50):
        x = gemm(a, b)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            y = x * 1
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(gemm(y, b), ref)
        torch.cuda.synchronize()  # (before the allocator hands x or y to the other stream)

"""The native operators against the registered operators and Python autograd functions that served every call before them: the same
results over the forms a call can have, and everything that is not a plain call (modes, transforms, tangents) still goes there."""

import math

import pytest
import torch
from torch.autograd import forward_ad

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture
def python_route(monkeypatch):
    """Run a function with the native operators switched off."""
    from nanonemo_b200.ops import _lib

    def run(fn):
        with monkeypatch.context() as m:
            m.setattr(_lib, "operator_call", lambda *a: NotImplemented)
            return fn()

    return run


def _native(name, *args):
    from nanonemo_b200.ops import _lib

    out = _lib.operator_call(name, *args)
    assert out is not NotImplemented, f"{name} did not take a plain call"
    return out


def _run(fn, leaves, grads):
    out = fn()
    out = out if isinstance(out, tuple) else (out,)
    pairs = [(o, g) for o, g in zip(out, grads) if g is not None and o.requires_grad]
    got = torch.autograd.grad([o for o, _ in pairs], leaves, [g for _, g in pairs], allow_unused=True) if pairs else ()
    return (*[o.detach() for o in out], *got)


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.dtype == y.dtype and x.shape == y.shape and x.device == y.device
            assert torch.equal(x, y)  # the same launches: bitwise


def _rand(*shape, dtype=torch.float32, grad=True):
    return (torch.randn(*shape, device=DEV) * 0.5).to(dtype).requires_grad_(grad)


@pytest.mark.parametrize("amp", [None, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("x_shape", [(7, 64), (300, 64), (2, 65, 64), (5, 3, 1, 64)])
@pytest.mark.parametrize("x_dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float32)])
def test_linear(python_route, amp, x_shape, x_dtype, w_dtype):
    from nanonemo_b200 import ops

    torch.manual_seed(0)
    x, w = _rand(*x_shape, dtype=x_dtype), _rand(136, 64, dtype=w_dtype)
    dy = torch.randn(*x_shape[:-1], 272, device=DEV)[..., ::2]  # strided upstream gradient
    with torch.autocast("cuda", dtype=amp or torch.bfloat16, enabled=amp is not None):
        _native("linear", x, w)
        fn = lambda: _run(lambda: ops.linear(x, w, impl="sm100"), (x, w), (dy.to(amp or torch.bfloat16),))  # noqa: E731
        _same(fn(), python_route(fn))


def test_linear_on_strided_and_unaligned_inputs(python_route):
    from nanonemo_b200 import ops

    base, w = torch.randn(130, 200, device=DEV).bfloat16(), _rand(72, 64)
    for x in (base[:, :64], base[:, 3:67], base.t()[:64].t(), base[::2, 8:72], torch.randn(64, 130, device=DEV).t(), base[:1, :64].expand(130, 64)):
        x = x.detach().requires_grad_()
        for dy in (torch.randn(x.shape[0], 72, device=DEV).bfloat16(), torch.ones((), device=DEV).bfloat16().expand(x.shape[0], 72),
                   torch.randn(72, x.shape[0], device=DEV).bfloat16().t(), torch.randn(x.shape[0], 80, device=DEV).bfloat16()[:, 3:75]):
            _native("linear", x, w)
            fn = lambda: _run(lambda: ops.linear(x, w, impl="sm100"), (x, w), (dy,))  # noqa: E731, B023
            _same(fn(), python_route(fn))


@pytest.mark.parametrize("with_delta", [False, True])
@pytest.mark.parametrize("x_dtype,d_dtype,amp", [(torch.float32, torch.bfloat16, True), (torch.float32, torch.float32, False), (torch.bfloat16, torch.bfloat16, False),
                                                 (torch.float16, torch.float32, False), (torch.float32, torch.float32, True)])
@pytest.mark.parametrize("use", [(True, True), (True, False), (False, True)])
def test_add_rms_norm(python_route, with_delta, x_dtype, d_dtype, amp, use):
    from nanonemo_b200 import ops

    torch.manual_seed(1)
    x, w = _rand(3, 37, 264, dtype=x_dtype), (1 + 0.1 * torch.randn(264, device=DEV)).requires_grad_()
    delta = _rand(3, 37, 528, dtype=d_dtype, grad=False)[..., ::2].requires_grad_() if with_delta else None
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=amp):
        y, h = _native("add_rms_norm", x, delta, w, 1e-5)
        grads = (torch.randn_like(y) if use[0] else None, torch.randn_like(h).transpose(0, 1).contiguous().transpose(0, 1) if use[1] else None)
        fn = lambda: _run(lambda: ops.add_rms_norm(x, delta, w, 1e-5, impl="sm100"), [t for t in (x, delta, w) if t is not None], grads)  # noqa: E731
        _same(fn(), python_route(fn))


@pytest.mark.parametrize("B,T,H,KVH,hd", [(1, 65, 2, 1, 64), (2, 130, 4, 4, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("layout", ["bthd", "bhtd", "odd"])
def test_flash_attn(python_route, B, T, H, KVH, hd, dtype, layout):
    from nanonemo_b200 import ops

    torch.manual_seed(2)

    def make(heads):
        if layout == "bthd":
            return torch.randn(B, T, heads, hd, device=DEV).to(dtype).transpose(1, 2)
        if layout == "bhtd":
            return torch.randn(B, heads, T, hd, device=DEV).to(dtype)
        return torch.randn(B, T, heads, hd + 4, device=DEV).to(dtype)[..., 3:hd + 3].transpose(1, 2)  # neither aligned nor dense

    q, k, v = (make(n).detach().requires_grad_() for n in (H, KVH, KVH))
    do = make(H)
    _native("flash_attn", q, k, v)
    fn = lambda: _run(lambda: ops.flash_attn(q, k, v), (q, k, v), (do,))  # noqa: E731
    a, b = fn(), python_route(fn)
    _same(a[:1] + a[2:], b[:1] + b[2:])
    # dQ is summed in fp32 by atomic adds in any order, then rounded once
    assert ((a[1].float() - b[1].float()).abs() <= 2 ** -7 * b[1].float().abs() + 1e-4).all()


def _engine(*ws):
    for w in ws:
        w._shadow, w._main_grad = w.detach().bfloat16(), torch.zeros_like(w)
        w._told = []
        w._grad_ready_cb = lambda p, done: p._told.append(done)


@pytest.mark.parametrize("M", [128, 320])
@pytest.mark.parametrize("hd", [64, 128])
def test_engine_nodes_add_into_the_flat_gradient_and_report_it(python_route, M, hd):
    """Both sides of the 256 rows from which the fused GEMM epilogues serve; x in fp32 and bf16."""
    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache

    torch.manual_seed(3)
    d, F, H, KVH = 192, 256, 2, 1
    cos, sin = rope_cache(hd, 1024, device=DEV)
    for dtype in (torch.float32, torch.bfloat16):
        x = _rand(2, M // 2, d, dtype=dtype)
        wq, gu, down, norm = _rand((H + 2 * KVH) * hd, d), _rand(2 * F, d), _rand(d, F), (torch.rand(d, device=DEV) + 0.5).requires_grad_()
        calls = {"qkv": ((wq,), lambda: ops.qkv_rope_attention(x, wq, cos, sin, H, KVH, hd)), "mlp": ((gu, down), lambda: ops.mlp_swiglu(x, gu, down)),  # noqa: B023
                 "linear": ((wq,), lambda: ops.linear(x, wq, impl="sm100")), "norm": ((norm,), lambda: ops.add_rms_norm(x, None, norm, 1e-5, impl="sm100")[0])}  # noqa: B023
        for name, (ws, fn) in calls.items():
            got = []
            for run in (lambda f: f(), python_route):
                _engine(*ws)
                out = run(fn)
                g = torch.linspace(-1, 1, out.numel(), device=DEV).view(out.shape).to(out.dtype)
                dx, *dw = torch.autograd.grad(out, (x, *ws), g, allow_unused=True)
                assert all(t is None for t in dw) and all(w._told == [True] for w in ws), name
                got.append((out.detach(), dx, *(w._main_grad for w in ws)))
            for a, b in zip(*got):  # the weight gradients of these sizes are cut into splits that are added in any order; dQ likewise
                assert a.dtype == b.dtype
                assert (a.float() - b.float()).norm() <= (2 ** -8 if a.dtype != torch.float32 or name == "qkv" else 1e-6) * b.float().norm(), name


def test_engine_nodes_add_their_weight_gradients_whatever_a_backward_pass_asks_for(python_route):
    """autograd.grad of the input alone, and a weight that is not trained."""
    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache

    torch.manual_seed(8)
    cos, sin = rope_cache(64, 1024, device=DEV)
    x = _rand(2, 160, 192, dtype=torch.bfloat16)
    wq, gu, down, norm = _rand(256, 192), _rand(512, 192), _rand(192, 256), torch.ones(192, device=DEV).requires_grad_()
    frozen, frozen_gu = _rand(256, 192, grad=False), _rand(512, 192, grad=False)
    calls = [((wq,), lambda: ops.qkv_rope_attention(x, wq, cos, sin, 2, 1, 64)), ((gu, down), lambda: ops.mlp_swiglu(x, gu, down)), ((wq,), lambda: ops.linear(x, wq, impl="sm100")),
             ((norm,), lambda: ops.add_rms_norm(x, None, norm, 1e-5, impl="sm100")[0]), ((frozen,), lambda: ops.linear(x, frozen, impl="sm100")),
             ((frozen,), lambda: ops.qkv_rope_attention(x, frozen, cos, sin, 2, 1, 64)), ((frozen_gu, down), lambda: ops.mlp_swiglu(x, frozen_gu, down))]
    for ws, fn in calls:
        got = []
        for run in (lambda f: f(), python_route):
            _engine(*ws)
            out = run(fn)
            torch.autograd.grad(out, x, torch.linspace(-1, 1, out.numel(), device=DEV).view(out.shape).to(out.dtype))
            got.append([(w._told, w._main_grad) for w in ws])
        for w, (told, a), (ref_told, b) in zip(ws, *got):
            assert told == ref_told == ([True] if w.requires_grad else [])
            assert (a - b).norm() <= 2 ** -8 * b.norm() and (b.norm() > 0) == w.requires_grad  # (dQ is summed in any order, then rounded)


def test_calls_without_gradients_match_the_registered_operators(python_route):
    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache

    torch.manual_seed(4)
    cos, sin = rope_cache(64, 512, device=DEV)
    for rows in (33, 300):
        x, wq, gu, down = _rand(1, rows, 128, grad=False), _rand(256, 128), _rand(512, 128), _rand(128, 256)
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            fn = lambda: (ops.qkv_rope_attention(x, wq, cos, sin, 2, 1, 64), ops.mlp_swiglu(x, gu, down), ops.linear(x, wq, impl="sm100"),  # noqa: E731, B023
                          *ops.add_rms_norm(x, None, down[:, 0].contiguous(), 1e-5, impl="sm100"))  # noqa: B023
            _same(fn(), python_route(fn))


def _cases():
    from nanonemo_b200 import ops

    torch.manual_seed(5)
    x, w, n = _rand(66, 64, dtype=torch.bfloat16), _rand(72, 64), torch.ones(64, device=DEV).requires_grad_()
    q = _rand(1, 2, 66, 64, dtype=torch.bfloat16)
    return [(lambda a: ops.linear(a, w, impl="sm100"), x), (lambda a: ops.add_rms_norm(a, a.detach(), n, 1e-5, impl="sm100")[0], x), (lambda a: ops.flash_attn(a, a.detach(), a.detach()), q)]


def test_second_derivatives_batched_gradients_and_hooks_behave_as_before(python_route):
    for fn, x in _cases():
        out = fn(x)
        g = torch.randn_like(out)
        plain = torch.autograd.grad(out, x, g)[0]

        def second():  # create_graph=True, and one more derivative: the gradient, or the refusal, of the registered operators
            try:
                (d,) = torch.autograd.grad(fn(x), x, g, create_graph=True)  # noqa: B023
                return d.detach(), torch.autograd.grad(d.float().sum(), x)[0]  # noqa: B023
            except (RuntimeError, AssertionError) as e:
                return type(e)

        a, b = second(), python_route(second)
        assert all(torch.allclose(s.float(), t.float(), rtol=2e-2, atol=1e-3) for s, t in zip(a, b)) if isinstance(b, tuple) else a is b
        batched = torch.autograd.grad(fn(x), x, torch.stack((g, 2 * g)), is_grads_batched=True)[0]
        assert batched.shape == (2, *x.shape) and torch.allclose(batched[0].float(), plain.float(), rtol=2e-2, atol=1e-3)
        # saved tensors pass through hooks, and what was saved is checked for in-place changes
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t.cpu(), lambda t: t.to(DEV)):
            out = fn(x)
        assert packed and torch.allclose(torch.autograd.grad(out, x, g)[0].float(), plain.float(), rtol=2e-2, atol=1e-3)
    from nanonemo_b200 import ops

    y, w = torch.randn(66, 64, device=DEV).bfloat16().requires_grad_(), _rand(72, 64)
    z = y * 1
    out = ops.linear(z, w, impl="sm100")
    with torch.no_grad():
        z.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, w, torch.ones_like(out))


@pytest.mark.parametrize("make", [lambda: _rand(66, 64), lambda: _rand(2, 33, 64, dtype=torch.bfloat16), lambda: _rand(2, 33, 64), lambda: _rand(66, 70, dtype=torch.bfloat16)[:, 3:67],
                                  lambda: _rand(66, 64, dtype=torch.bfloat16)])
def test_second_derivatives_of_a_linear_reach_its_input_or_are_refused_as_before(python_route, make):
    """Also where the input is cast, reshaped or copied first: what the node saves has to lead back to it."""
    from nanonemo_b200 import ops

    x, w = make().detach().requires_grad_(), _rand(72, 64)
    frozen = w.detach()

    def penalty():  # of the weight's gradient, with respect to the input
        (dw,) = torch.autograd.grad(ops.linear(x, w, impl="sm100").float().square().sum(), w, create_graph=True)
        return torch.autograd.grad(dw.float().square().sum(), x)[0]

    def hessian():
        return torch.autograd.functional.hvp(lambda a: ops.linear(a, frozen, impl="sm100").float().sum(), x.detach(), torch.ones_like(x))[1]

    for fn in (penalty, hessian):
        got = []
        for run in (lambda f: f(), python_route):
            try:
                got.append(run(fn))
            except (RuntimeError, AssertionError) as e:
                got.append(type(e))
        a, b = got
        assert torch.allclose(a.float(), b.float(), rtol=2e-2, atol=1e-3) if isinstance(b, torch.Tensor) else a is b


def test_the_trainers_linear_takes_part_in_graphs_of_gradients_as_before(python_route):
    """Weights with and without the engine's buffers, and calls without gradients."""
    from nanonemo_b200.ops.gemm import linear_sm100

    x = _rand(66, 64, dtype=torch.bfloat16)
    for engine in (False, True):
        w = _rand(72, 64)
        if engine:
            _engine(w)

        def first():
            (dx,) = torch.autograd.grad(linear_sm100(x, w).float().sum(), x, create_graph=True)  # noqa: B023
            return dx.detach(), dx.requires_grad

        (a, a_graph), (b, b_graph) = first(), python_route(first)
        assert torch.equal(a, b) and a_graph == b_graph
        with torch.no_grad():
            assert torch.equal(linear_sm100(x, w), python_route(lambda: linear_sm100(x, w)))  # noqa: B023


def test_outputs_may_be_changed_in_place():
    for fn, x in _cases()[:2]:  # (attention keeps its output for the backward)
        fn(x).mul_(2).float().sum().backward()
        assert x.grad is not None


def test_anything_but_a_plain_call_takes_the_other_route(python_route):
    from torch.utils._python_dispatch import TorchDispatchMode

    from nanonemo_b200.ops import _lib

    x, w = _rand(66, 64, dtype=torch.bfloat16), _rand(72, 64)

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    assert _lib.operator_call("linear", x, w) is not NotImplemented
    assert _lib.operator_call("linear", x.cpu(), w.cpu()) is NotImplemented
    assert _lib.operator_call("linear", x.detach().as_subclass(Sub), w) is NotImplemented
    with Mode():
        assert _lib.operator_call("linear", x, w) is NotImplemented
    with torch.device(DEV):
        assert _lib.operator_call("linear", x, w) is NotImplemented
    with forward_ad.dual_level():
        assert _lib.operator_call("linear", forward_ad.make_dual(x.detach(), torch.ones_like(x)), w) is NotImplemented
    seen = []
    torch.func.vmap(lambda a: seen.append(_lib.operator_call("linear", a, w)) or a)(x[None])
    torch.func.grad(lambda a: seen.append(_lib.operator_call("linear", a, w)) or a.float().sum())(x.detach())
    assert seen == [NotImplemented, NotImplemented]
    for fn, x in _cases():  # torch.func.grad through the front end: as the registered operators have it
        f = lambda a: fn(a).float().sum()  # noqa: E731, B023
        try:
            ref = python_route(lambda: torch.func.grad(f)(x.detach()))  # noqa: B023
        except RuntimeError as e:
            with pytest.raises(type(e)):
                torch.func.grad(f)(x.detach())
        else:
            assert torch.allclose(torch.func.grad(f)(x.detach()).float(), ref.float(), rtol=2e-2, atol=1e-3)


def test_wrong_calls_are_refused_with_the_same_errors(python_route):
    from nanonemo_b200 import ops
    from nanonemo_b200.ops.gemm import gemm

    x, w = _rand(66, 64, dtype=torch.bfloat16), _rand(72, 64)
    q = _rand(1, 2, 66, 64, dtype=torch.bfloat16)
    calls = [lambda: ops.linear(x, w[:, :32], impl="sm100"), lambda: ops.linear(x, w[:, :60], impl="sm100"), lambda: ops.flash_attn(q[..., :32], q[..., :32], q[..., :32]),
             lambda: ops.add_rms_norm(x[:, :60], None, w[0, :60], 1e-5, impl="sm100"), lambda: ops.add_rms_norm(x.double(), None, w[0], 1e-5, impl="sm100")]
    for call in calls:
        with pytest.raises(Exception) as ref:
            python_route(call)
        with pytest.raises(ref.type):
            call()
    with pytest.raises(AssertionError):
        gemm(x.detach(), w.detach())  # dtypes differ
    with pytest.raises(AssertionError):
        gemm(x.detach(), x.detach()[:, :32])


def test_launches_are_counted_once():
    from nanonemo_b200 import ops
    from nanonemo_b200.ops import _lib

    x, w = _rand(66, 64, dtype=torch.bfloat16), _rand(72, 64, dtype=torch.bfloat16)
    before = _lib.LAUNCHES
    y = ops.linear(x, w, impl="sm100")
    torch.autograd.grad(y, (x, w), torch.ones_like(y))
    assert _lib.LAUNCHES - before == 3
    assert math.isfinite(y.float().sum().item())


@pytest.mark.parametrize("direct", [True, False])
@pytest.mark.parametrize("rows", [33, 201, 300])
def test_calls_without_gradients_cast_no_more_than_the_registered_operators(python_route, rows, direct):
    """The input, and no fp32 weight that the kernels take as it is; others (here: not at a multiple of 16 bytes) once each, also where the fused kernel does
    not serve the rows and others take over."""
    from torch.profiler import ProfilerActivity, profile

    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache

    cos, sin = rope_cache(64, 512, device=DEV)
    weight = lambda *s: _rand(*s) if direct else _rand(s[0] * s[1] + 1)[1:].view(s)  # noqa: E731
    x, wq, gu, down = _rand(1, rows, 128, grad=False), weight(256, 128), weight(512, 128), weight(128, 256)

    def casts(fn):
        with torch.no_grad():
            fn()
            with profile(activities=[ProfilerActivity.CPU]) as p:
                fn()
        return sum(e.count for e in p.key_averages() if e.key == "aten::_to_copy")

    for fn, weights in ((lambda: ops.mlp_swiglu(x, gu, down), 2), (lambda: ops.qkv_rope_attention(x, wq, cos, sin, 2, 1, 64), 1), (lambda: ops.linear(x, wq, impl="sm100"), 1)):
        assert casts(fn) == 1 + (0 if direct else weights) <= python_route(lambda: casts(fn))  # noqa: B023


def test_the_fused_swiglu_backward_can_be_switched_off_on_the_models_path(monkeypatch):
    from nanonemo_b200 import ops
    from nanonemo_b200.ops import _lib, fused_block

    torch.manual_seed(7)
    x, gu, down = _rand(300, 128), _rand(512, 128), _rand(128, 256)
    launches, got = [], []
    for fused in (True, False):
        monkeypatch.setattr(fused_block, "FUSE_SWIGLU_BWD", fused)
        _engine(gu, down)
        before = _lib.LAUNCHES
        out = ops.mlp_swiglu(x, gu, down)
        (dx,) = torch.autograd.grad(out, x, torch.ones_like(out))
        launches.append(_lib.LAUNCHES - before)
        got.append((out.detach(), dx, gu._main_grad))
    assert launches[1] == launches[0] + 1  # d(act) and the activation's backward apart
    for a, b in zip(*got):  # d(act) is rounded to 16 bits between the two
        assert (a.float() - b.float()).norm() <= 2 ** -7 * b.float().norm()


def test_inference_mode(python_route):
    from nanonemo_b200 import ops
    from nanonemo_b200.models.layers import rope_cache

    torch.manual_seed(6)
    cos, sin = rope_cache(64, 512, device=DEV)
    x, wq, gu, down, n = _rand(1, 300, 128, grad=False), _rand(256, 128), _rand(512, 128), _rand(128, 256), torch.ones(128, device=DEV).requires_grad_()
    q = _rand(1, 2, 66, 64, dtype=torch.bfloat16, grad=False)

    def fn():
        y, h = ops.add_rms_norm(x, x.bfloat16(), n, 1e-5, impl="sm100")
        return (ops.qkv_rope_attention(y, wq, cos, sin, 2, 1, 64), ops.mlp_swiglu(y, gu, down), ops.linear(y, wq, impl="sm100"), y, h, ops.flash_attn(q, q, q))

    with torch.inference_mode(), torch.autocast("cuda", dtype=torch.bfloat16):
        _same(fn(), python_route(fn))


_FIRST_CALLS = """
import torch
from nanonemo_b200 import ops
torch.manual_seed(0)
x, w, n = (torch.randn(*s, device="cuda", requires_grad=True) for s in ((66, 64), (72, 64), (64,)))
q = torch.randn(1, 2, 66, 64, device="cuda").bfloat16().requires_grad_()
for fn, leaf in ((lambda: ops.linear(x, w, impl="sm100"), x), (lambda: ops.add_rms_norm(x, None, n, 1e-5, impl="sm100")[0], x), (lambda: ops.flash_attn(q, q.detach(), q.detach()), q)):
    g = torch.randn_like(fn())
    (plain,) = torch.autograd.grad(fn(), leaf, g)
    (two,) = torch.autograd.grad(fn(), leaf, torch.stack((g, 2 * g)), is_grads_batched=True)
    assert torch.allclose(two[0].float(), plain.float(), rtol=2e-2, atol=1e-3)
for fn, leaf in ((lambda: ops.add_rms_norm(x, None, n, 1e-5, impl="sm100")[0], x), (lambda: ops.flash_attn(q, q.detach(), q.detach()), q)):
    assert torch.autograd.grad(fn().float().sum(), leaf, create_graph=True)[0].requires_grad
"""


def test_backward_nodes_find_the_registered_operators_in_a_new_process():
    """Nothing but `ops` imported and no call made that would have registered them."""
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", _FIRST_CALLS], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, None])
@pytest.mark.parametrize("B,T,head_dim", [(1, 1, 64), (1, 201, 64), (2, 100, 128), (3, 300, 64), (1, 130, 128)])
def test_a_block_without_gradients_is_its_operators_in_one_call(monkeypatch, B, T, head_dim, dtype):
    """The same bits, few rows (one workspace) and many, with and without a pending delta; parts that are watched run one by one."""
    from contextlib import nullcontext

    from torch.profiler import ProfilerActivity, profile

    from nanonemo_b200 import ops
    from nanonemo_b200.models.config import ModelConfig
    from nanonemo_b200.models.layers import Block, rope_cache
    from nanonemo_b200.ops import _lib
    from nanonemo_b200.ops.gemm import check_status

    torch.manual_seed(B * T)
    cfg = ModelConfig.sm100(n_layers=1, d_model=768, n_heads=768 // head_dim, n_kv_heads=2, d_ff=2048, max_seq_len=512, head_dim_override=head_dim)
    block = Block(cfg).to(DEV).eval()
    cos, sin = rope_cache(head_dim, 512, device=DEV)
    x, delta = torch.randn(B, T, 768, device=DEV), torch.randn(B, T, 768, device=DEV).to(dtype or torch.bfloat16)

    def run(d):
        with torch.no_grad(), torch.autocast("cuda", dtype=dtype) if dtype else nullcontext():
            return block(x, cos, sin, d)

    answers, in_one = [], ops.decoder_block
    monkeypatch.setattr(ops, "decoder_block", lambda *a: answers.append(in_one(*a)) or answers[-1])
    for d in (None, delta):
        before = _lib.LAUNCHES
        with profile(activities=[ProfilerActivity.CPU]) as p:
            got = run(d)
        check_status()
        assert _lib.LAUNCHES - before == 7 and len(answers) == 1 and answers.pop() is not NotImplemented
        # few rows with an output in the compute type (without autocast and a delta it is that of x, fp32): one workspace and the two results
        allocated = sum(e.count for e in p.key_averages() if e.key.startswith("aten::empty"))
        assert (allocated == 3) == (B * T <= 201 and (dtype is not None or d is not None)), allocated
        with monkeypatch.context() as m:
            m.setattr(Block, "_one_call", lambda self: False)
            ref = run(d)
        for a, b in zip(got, ref):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    seen = []
    handle = block.attn.wo.register_forward_hook(lambda *a: seen.append(1))
    assert not block._one_call()
    again = run(delta)
    handle.remove()
    assert seen == [1] and all(torch.equal(a, b) for a, b in zip(again, got))

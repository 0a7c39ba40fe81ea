"""The work that a user has this framework do, as cases to time: optimizer steps, validation, scoring, and the
operators called on their own. Inputs come from a seed; ``exact`` gives the same results in plain 64-bit torch.
"""

import math

import torch
import torch.nn.functional as F

from nanonemo_b200 import ops, parallel
from nanonemo_b200.models.config import ModelConfig
from nanonemo_b200.models.model import NanoNemo
from nanonemo_b200.train.config import TrainConfig
from nanonemo_b200.train.optim import build_optimizer
from nanonemo_b200.train.trainer import build_parallel, evaluate, train_step

DEV = "cuda"
VOCAB, TOKENS = 50304, 50257  # padded vocabulary of the model; ids that the tokenizer produces
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
LR, BETAS, EPS, DECAY, CLIP, NORM_EPS, ROPE_BASE = 1e-4, (0.9, 0.95), 1e-8, 0.1, 1.0, 1e-5, 10000.0

# the two model widths of configs/: the 114M model, and the layers of the 1.3B model
WIDTHS = {"114m": dict(d_model=768, n_heads=12, n_kv_heads=4, d_ff=2048, max_seq_len=1024, head_dim_override=64),
          "1p3b": dict(d_model=2048, n_heads=16, n_kv_heads=4, d_ff=5632, max_seq_len=2048, head_dim_override=128)}


def listed():
    return [
        # the step of configs/b200/single.yaml as bench.py runs it: the largest ordinary call, replayed from a CUDA graph
        dict(name="train-114m", kind="train", width="114m", layers=12, batch=32, seq=1024, accum=1, graph=True, precision="bf16"),
        # a small global batch by gradient accumulation, launched eagerly (the default): host and launches count
        dict(name="train-114m-accum", kind="train", width="114m", layers=12, batch=4, seq=1024, accum=2, graph=False, precision="bf16"),
        # 1.3B layers (head_dim 128, seq 2048); four of the 24, which all do the same
        dict(name="train-1p3b-4layers", kind="train", width="1p3b", layers=4, batch=4, seq=2048, accum=1, graph=False, precision="bf16"),
        # `precision: fp8` at the micro-batch of configs/precision
        dict(name="train-114m-fp8", kind="train", width="114m", layers=12, batch=8, seq=1024, accum=1, graph=False, precision="fp8"),
        # validation between training steps: two batches, loss only
        dict(name="validate-114m", kind="validate", width="114m", layers=12, batch=16, seq=1024, batches=2),
        # scoring one short text of odd length with a loaded model: logits, no gradients
        dict(name="score-114m", kind="score", width="114m", layers=12, batch=1, seq=201),
        # attention on its own, forward and backward: long context; wide heads in fp16; a short ragged call
        dict(name="attention-long", kind="attention", batch=8, heads=12, kv_heads=4, seq=4096, head_dim=64, dtype="bf16", backward=True),
        dict(name="attention-wide", kind="attention", batch=8, heads=16, kv_heads=4, seq=2048, head_dim=128, dtype="fp16", backward=True),
        dict(name="attention-ragged", kind="attention", batch=2, heads=12, kv_heads=4, seq=333, head_dim=64, dtype="bf16", backward=True),
        # the fused head and loss in a user's own training loop
        dict(name="head-loss", kind="loss", rows=4096, width_in=768, vocab=VOCAB, dtype="bf16"),
        # residual add + norm, fp32 residual stream, forward and backward
        dict(name="add-norm", kind="norm", rows=16384, width_in=768, dtype="bf16"),
        # a linear layer, odd number of rows, forward and backward, weight in fp32
        dict(name="linear-odd", kind="linear", rows=777, width_in=768, width_out=4096, dtype="fp16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "validate", "score", "attention", "attention", "loss", "norm", "linear"])
    if kind == "train":
        width = rng.choice(["114m", "114m", "1p3b"])
        seq = _log_int(rng, 64, WIDTHS[width]["max_seq_len"])
        precision = rng.choice(["bf16", "bf16", "fp8"]) if width == "114m" else "bf16"
        if precision == "fp8":
            seq = max(128, seq // 128 * 128)  # the block-scaled operands take whole 128-row blocks
        accum = rng.choice([1, 1, 2])
        batch = _log_int(rng, 1, max(1, min(32, (32768 if width == "114m" else 8192) // (seq * accum))))
        return dict(kind=kind, width=width, layers=12 if width == "114m" else 4, batch=batch, seq=seq, accum=accum,
                    graph=precision == "bf16" and rng.random() < 0.5, precision=precision)
    if kind == "validate":
        seq = _log_int(rng, 64, 1024)
        return dict(kind=kind, width="114m", layers=12, batch=_log_int(rng, 1, min(32, 32768 // seq)), seq=seq, batches=rng.choice([1, 2, 3]))
    if kind == "score":
        return dict(kind=kind, width="114m", layers=12, batch=rng.choice([1, 1, 2, 8]), seq=_log_int(rng, 16, 1024))
    if kind == "attention":
        head_dim = rng.choice([64, 128])
        heads, kv_heads = rng.choice([(12, 4), (16, 4), (8, 8), (6, 1)])
        seq = _log_int(rng, 64, 4096)
        batch = _log_int(rng, 1, max(1, min(64, int(8 * (4096 / seq) * 64 / head_dim * 12 / heads))))
        return dict(kind=kind, batch=batch, heads=heads, kv_heads=kv_heads, seq=seq, head_dim=head_dim,
                    dtype=rng.choice(["bf16", "fp16"]), backward=rng.random() < 0.7)
    if kind == "loss":
        return dict(kind=kind, rows=_log_int(rng, 128, 16384), width_in=rng.choice([512, 768, 2048]), vocab=rng.choice([VOCAB, 32000]),
                    dtype=rng.choice(["bf16", "fp16"]))
    if kind == "norm":
        return dict(kind=kind, rows=_log_int(rng, 16, 32768), width_in=rng.choice([512, 768, 1000, 2048]), dtype=rng.choice(["bf16", "fp16", "fp32"]))
    return dict(kind="linear", rows=_log_int(rng, 64, 16384), width_in=rng.choice([512, 768, 2048]), width_out=rng.choice([768, 1280, 4096]),
                dtype=rng.choice(["bf16", "fp16"]))


# ------------------------------------------------------------------------------------------------ inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device=DEV).mul_(std).to(dtype)


def _tokens(g, *shape):
    """Ids whose frequency falls with their rank, as in text: the id's logarithm is uniform."""
    u = torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)
    return (u * math.log(TOKENS)).exp().long().sub_(1).clamp_(0, TOKENS - 1)


def _batches(case, seed):
    g = _rng(seed * 7 + 1)
    windows = [_tokens(g, case["batch"], case["seq"] + 1) for _ in range(case.get("accum", case.get("batches", 1)))]
    return [(w[:, :-1], w[:, 1:]) for w in windows]


def _weights(case, seed):
    """name -> fp32 tensor, in the order of the model's parameters."""
    g, w, c, n = _rng(seed * 7 + 2), {}, WIDTHS[case["width"]], case["layers"]
    d, hd, ff = c["d_model"], c["head_dim_override"], c["d_ff"]
    resid = 0.02 / math.sqrt(2 * n)
    w["tok_emb.weight"] = _normal(g, VOCAB, d, std=0.02)
    for i in range(n):
        p = f"blocks.{i}."
        w[p + "norm_attn.weight"] = 1 + _normal(g, d, std=0.1)
        w[p + "attn.wqkv.weight"] = _normal(g, (c["n_heads"] + 2 * c["n_kv_heads"]) * hd, d, std=0.02)
        w[p + "attn.wo.weight"] = _normal(g, d, c["n_heads"] * hd, std=resid)
        w[p + "norm_mlp.weight"] = 1 + _normal(g, d, std=0.1)
        w[p + "mlp.w_gu.weight"] = _normal(g, 2 * ff, d, std=0.02)
        w[p + "mlp.w_down.weight"] = _normal(g, d, ff, std=resid)
    w["norm_out.weight"] = 1 + _normal(g, d, std=0.1)
    return w


class Source:
    """Batches that are on the GPU already, handed out in turn."""

    def __init__(self, batches):
        self.batches, self.micro_step = batches, 0

    def next_batch(self):
        self.micro_step += 1
        return self.batches[(self.micro_step - 1) % len(self.batches)]


def _trainer(case, seed):
    precision = case.get("precision", "bf16")
    model_cfg = ModelConfig.sm100(n_layers=case["layers"], vocab_size=VOCAB, linear_impl="mxfp8" if precision == "fp8" else "sm100",
                                  **WIDTHS[case["width"]])
    cfg = TrainConfig(data_dir="synthetic", seq_len=case["seq"], micro_batch=case["batch"], precision=precision,
                      global_batch_tokens=case["batch"] * case["seq"] * case.get("accum", 1), cuda_graph=case.get("graph", False))
    with torch.device(DEV):
        strategy = build_parallel(model_cfg, cfg, parallel.Dist(device="cuda:0"))
    opt = build_optimizer(strategy.model, LR, DECAY, betas=BETAS, eps=EPS, store=strategy.store)
    for name, value in _weights(case, seed).items():
        strategy.restore_tensor(opt, "model", name, value)
    strategy.finish_restore(opt, 0)
    return strategy, opt


def _op_inputs(case, seed):
    g, k, dt = _rng(seed * 7 + 3), case["kind"], DTYPES[case["dtype"]]
    if k == "attention":
        B, T, H, KVH, hd = (case[n] for n in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        # what projections hand over: (B, T, heads, hd) in memory, seen as (B, heads, T, hd)
        q, key, v, do = (_normal(g, B, T, h, hd, dtype=dt).transpose(1, 2) for h in (H, KVH, KVH, H))
        return q, key, v, do
    rows, n = case["rows"], case["width_in"]
    if k == "norm":
        return (_normal(g, rows, n), _normal(g, rows, n, std=0.5, dtype=dt), 1 + _normal(g, n, std=0.1), _normal(g, rows, n, dtype=dt),
                _normal(g, rows, n))
    x = _normal(g, rows, n, dtype=dt)
    if k == "loss":
        return x, _normal(g, case["vocab"], n, std=0.02), _tokens(g, rows).clamp_(max=case["vocab"] - 1)
    return x, _normal(g, case["width_out"], n, std=0.02), _normal(g, rows, case["width_out"], dtype=dt)


def prepare(case, seed):
    k = case["kind"]
    if k in ("train", "validate"):
        strategy, opt = _trainer(case, seed)
        return dict(case=case, strategy=strategy, opt=opt, source=Source(_batches(case, seed)))
    if k == "score":
        with torch.device(DEV):
            model = NanoNemo(ModelConfig.sm100(n_layers=case["layers"], vocab_size=VOCAB, **WIDTHS[case["width"]]))
        model.load_state_dict(_weights(case, seed), strict=False)
        return dict(case=case, model=model.eval(), idx=_batches(case, seed)[0][0])
    t = _op_inputs(case, seed)
    leaves = {"attention": t[:3], "norm": t[:3], "loss": t[:2], "linear": t[:2]}[k]
    if case.get("backward", True):
        for x in leaves:
            x.requires_grad_(True)
    return dict(case=case, t=t, leaves=leaves)


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "train":
        st = state["strategy"]
        out = train_step(st, state["opt"], state["source"], case["accum"], CLIP, torch.bfloat16, None, host_sync=False)
        return dict(loss=out[0], norm=out[1], weights=st.store.master, exp_avg=st.store.exp_avg, exp_avg_sq=st.store.exp_avg_sq)
    if k == "validate":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return evaluate(state["strategy"].model, state["source"], case["batches"])
    if k == "score":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return state["model"](state["idx"])[0]
    t, leaves, dt = state["t"], state["leaves"], DTYPES[case["dtype"]]
    if k == "attention":
        o = ops.flash_attn(*t[:3])
        return (o, *torch.autograd.grad(o, leaves, t[3])) if case["backward"] else (o,)
    if k == "norm":
        y, h = ops.add_rms_norm(t[0], t[1], t[2], NORM_EPS, impl="sm100")
        return (y, h, *torch.autograd.grad((y, h), leaves, (t[3], t[4])))
    with torch.autocast("cuda", dtype=dt):
        if k == "loss":
            loss = ops.linear_cross_entropy(*t)
            return (loss, *torch.autograd.grad(loss, leaves))
        y = ops.linear(t[0], t[1], impl="sm100")
    return (y, *torch.autograd.grad(y, leaves, t[2]))


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _model_size(case):
    c = WIDTHS[case["width"]]
    d, hd = c["d_model"], c["head_dim_override"]
    matmul = case["layers"] * ((c["n_heads"] + 2 * c["n_kv_heads"]) * hd * d + d * c["n_heads"] * hd + 3 * d * c["d_ff"]) + VOCAB * d
    attention = case["layers"] * 2 * c["n_heads"] * hd * case["seq"]  # multiply-adds of the causal half, per token, times two
    return matmul, matmul + (2 * case["layers"] + 1) * d, attention


def work(case):
    k = case["kind"]
    if k in ("train", "validate", "score"):
        matmul, params, attention = _model_size(case)
        tokens = case["batch"] * case["seq"] * case.get("accum", case.get("batches", 1))
        flops = tokens * (2 * matmul + attention)
        if k == "train":  # weights and both moments are read and written; inputs and targets read
            return dict(bytes=24 * params + 16 * tokens, flops=3 * flops)
        if k == "validate":  # the 16-bit weights
            return dict(bytes=2 * params + 16 * tokens, flops=flops)
        return dict(bytes=4 * params + 8 * tokens + 2 * tokens * VOCAB, flops=flops)  # the fp32 weights; the logits
    size = 4 if case["dtype"] == "fp32" else 2
    if k == "attention":
        B, T, H, KVH, hd = (case[n] for n in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        elements, flops = 2 * H + 2 * KVH, 2 * B * H * T * T * hd
        if case["backward"]:  # dO read, dQ, dK, dV written; four more products
            elements, flops = elements + 2 * H + 2 * KVH, 3 * flops
        return dict(bytes=size * B * T * hd * elements, flops=flops)
    rows, n = case["rows"], case["width_in"]
    if k == "norm":  # x, delta, dy, dh in; y, h, dx, ddelta out; the 32-bit ones are the residual stream
        return dict(bytes=rows * n * (4 * 4 + 4 * size) + 8 * n, flops=14 * rows * n)
    wide = case["vocab"] if k == "loss" else case["width_out"]
    moved = 2 * size * rows * n + 8 * wide * n  # x, dx; the fp32 weight and its gradient
    return dict(bytes=moved + (8 * rows if k == "loss" else 2 * size * rows * wide), flops=6 * rows * n * wide)


def tolerance(case):
    """About four times what a pass is off the 64-bit result at these precisions."""
    k = case["kind"]
    if k == "train":  # fp8: 8-bit operands, whose rounding goes over to another value now and then
        return {"rel": 0.1} if case["precision"] == "fp8" else {"rel": 0.04}
    if k == "validate":
        return {"rel": 1e-4}
    if k == "score":
        return {"rel": 0.04}
    return {"rel": {"bf16": 0.01, "fp16": 0.0015, "fp32": 1e-6}[case["dtype"]]}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + NORM_EPS) * w


def _attention64(q, k, v):
    """(B, H, T, hd), a few heads at a time where the score matrix would be large."""
    group, T = q.shape[1] // k.shape[1], q.shape[2]
    k, v = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1)
    s = (q @ k.transpose(-1, -2)) / math.sqrt(q.shape[-1])
    return s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), float("-inf")).softmax(-1) @ v


def _rope64(x):
    half, T = x.shape[-1] // 2, x.shape[-2]
    inv = ROPE_BASE ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    a = torch.outer(torch.arange(T, device=x.device, dtype=torch.float64), inv)
    x1, x2 = x[..., :half], x[..., half:]
    return torch.cat((x1 * a.cos() - x2 * a.sin(), x1 * a.sin() + x2 * a.cos()), -1)


def _logits64(w, case, idx):
    c = WIDTHS[case["width"]]
    H, KVH, hd = c["n_heads"], c["n_kv_heads"], c["head_dim_override"]
    B, T = idx.shape
    heads = lambda t, n: t.view(B, T, n, hd).transpose(1, 2)  # noqa: E731
    x = w["tok_emb.weight"][idx]
    for i in range(case["layers"]):
        p = f"blocks.{i}."
        q, k, v = (_norm64(x, w[p + "norm_attn.weight"]) @ w[p + "attn.wqkv.weight"].T).split((H * hd, KVH * hd, KVH * hd), -1)
        a = _attention64(_rope64(heads(q, H)), _rope64(heads(k, KVH)), heads(v, KVH))
        x = x + a.transpose(1, 2).reshape(B, T, H * hd) @ w[p + "attn.wo.weight"].T
        gate, up = (_norm64(x, w[p + "norm_mlp.weight"]) @ w[p + "mlp.w_gu.weight"].T).chunk(2, -1)
        x = x + (F.silu(gate) * up) @ w[p + "mlp.w_down.weight"].T
    return _norm64(x, w["norm_out.weight"]) @ w["tok_emb.weight"].T


def _slices(case, batches):
    """The batches in pieces of whole sequences that fit in memory in 64 bits."""
    rows = max(1, (4096 if case["width"] == "114m" else 2048) // case["seq"])
    return [(x[i:i + rows], y[i:i + rows]) for x, y in batches for i in range(0, x.shape[0], rows)]


def _exact_model(case, seed):
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    batches = _batches(case, seed)
    if case["kind"] == "score":
        return torch.cat([_logits64(w, case, x) for x, _ in _slices(case, batches)])
    total = sum(y.numel() for _, y in batches)
    grads = case["kind"] == "train" and case["precision"] != "fp8"
    loss = 0.0
    for t in w.values():
        t.requires_grad_(grads)
    for x, y in _slices(case, batches):
        part = F.cross_entropy(_logits64(w, case, x).flatten(0, 1), y.reshape(-1), reduction="sum") / total
        if grads:
            part.backward()
        loss += part.item()
    if case["kind"] == "validate":
        return loss
    if not grads:  # no 64-bit value belongs to a gradient of 8-bit operands
        return dict(loss=loss, norm=None, weights=None, exp_avg=None, exp_avg_sq=None)
    norm = torch.sqrt(sum(t.grad.square().sum() for t in w.values()))
    coef = (CLIP / (norm + 1e-6)).clamp(max=1.0)
    p, m, v = [], [], []
    for name, t in w.items():
        g, t = t.grad * coef, t.detach()
        m.append(((1 - BETAS[0]) * g).reshape(-1))
        v.append(((1 - BETAS[1]) * g * g).reshape(-1))
        decay = DECAY if t.dim() == 2 and name != "tok_emb.weight" else 0.0
        p.append((t * (1 - LR * decay) - LR * g / (g.abs() + EPS)).reshape(-1))
    return dict(loss=loss, norm=norm, weights=torch.cat(p), exp_avg=torch.cat(m), exp_avg_sq=torch.cat(v))


def exact(case, seed):
    if case["kind"] in ("train", "validate", "score"):
        with torch.set_grad_enabled(case["kind"] == "train"):
            return _exact_model(case, seed)
    k = case["kind"]
    t = [x.double() if x.is_floating_point() else x for x in _op_inputs(case, seed)]
    if k == "attention":
        # one KV head and its query heads of one sequence at a time: the score matrices stay small
        group, parts = case["heads"] // case["kv_heads"], []
        o, *grads = [torch.empty_like(x) for x in (t[0], *t[:3])]
        for b in range(case["batch"]):
            for h in range(case["kv_heads"]):
                qs, ks = (slice(b, b + 1), slice(h * group, (h + 1) * group)), (slice(b, b + 1), slice(h, h + 1))
                parts = [t[0][qs].clone().requires_grad_(), t[1][ks].clone().requires_grad_(), t[2][ks].clone().requires_grad_()]
                with torch.enable_grad():
                    out = _attention64(*parts)
                o[qs] = out.detach()
                if case["backward"]:
                    for dst, at, g in zip(grads, (qs, ks, ks), torch.autograd.grad(out, parts, t[3][qs])):
                        dst[at] = g
        return (o, *grads) if case["backward"] else (o,)
    with torch.enable_grad():
        if k == "norm":
            leaves = [x.requires_grad_() for x in t[:3]]
            h = t[0] + t[1]
            y = _norm64(h, t[2])
            return (y.detach(), h.detach(), *torch.autograd.grad((y, h), leaves, (t[3], t[4])))
        leaves = [x.requires_grad_() for x in t[:2]]
        if k == "loss":
            loss = F.cross_entropy(t[0] @ t[1].T, t[2])
            return (loss.detach(), *torch.autograd.grad(loss, leaves))
        y = t[0] @ t[1].T
        return (y.detach(), *torch.autograd.grad(y, leaves, t[2]))

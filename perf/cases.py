"""Workloads of this framework for timing and for comparing results: training and evaluation passes of its models, and the
operators and the optimizer step that they are made of, each called as a user's program calls it.

A case is a dict of plain values with a ``kind``:

* ``gpt`` / ``llama``: forward, loss and backward of a model through ``OptimManager`` (or an evaluation pass without
  gradients), returning loss, logits and every parameter gradient;
* ``attention``, ``linear``, ``norm``, ``loss``: one operator, forward and backward;
* ``adam``: overflow check, gradient clipping and the optimizer step over the shards of a model.
"""
import math
import os
import socket

import torch
import torch.nn.functional as F

import bmtrain_b200 as bmt
from bmtrain_b200.ops import attention as attention_op
from bmtrain_b200.ops import gemm as gemm_op
from bmtrain_b200.ops import norm as norm_op

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
FP16_SCALE = 4096.0   # loss scale of fp16 training cases; bf16 trains unscaled


# ------------------------------------------------------------------------------------------------------------- cases
def listed():
    gpt = dict(kind="gpt", activation="relu", dtype="fp16", dense_mask=True, train=True)
    return [
        # smallest model of the configurations: launches and latency, not bandwidth, decide
        dict(gpt, name="gpt d256 x2 256 tokens", layers=2, vocab=10240, heads=4, dim_head=64, dim_ff=1024, batch=2, seq=128),
        # the benchmark model (half its layers): forward + backward with recomputation
        dict(gpt, name="gpt d2560 x4 1024 tokens", layers=4, vocab=10240, heads=32, dim_head=80, dim_ff=8192, batch=2, seq=512),
        # evaluation of the benchmark model on a ragged batch
        dict(gpt, name="gpt d2560 x4 eval 3x437", layers=4, vocab=10240, heads=32, dim_head=80, dim_ff=8192, batch=3, seq=437,
             dtype="bf16", train=False),
        # block and vocabulary of the larger GPT configuration: GELU, head dim 128, 2048 tokens a sequence, causal flag
        dict(gpt, name="gpt d4096 gelu 2x2048", layers=1, vocab=50304, heads=32, dim_head=128, dim_ff=16384, batch=2, seq=2048,
             activation="gelu", dtype="bf16", dense_mask=False),
        # 13B-shaped decoder layer at its training length
        dict(kind="llama", name="llama d5120 1x4096", layers=1, vocab=32000, heads=40, kv_heads=40, dim_head=128, dim_ff=13824,
             batch=1, seq=4096, dtype="bf16", train=True),
        # 70B-shaped decoder layer, grouped-query attention
        dict(kind="llama", name="llama d8192 gqa 1x2048", layers=1, vocab=32000, heads=64, kv_heads=8, dim_head=128, dim_ff=28672,
             batch=1, seq=2048, dtype="bf16", train=True),
        # padded batch of uneven lengths, head dim of the benchmark model
        dict(kind="attention", name="attention 4x1000 h32 d80 lens", batch=4, seq=1000, heads=32, kv_heads=32, dim_head=80,
             causal=False, lens=True, dtype="fp16"),
        # long causal sequences
        dict(kind="attention", name="attention 2x4096 h20 d128", batch=2, seq=4096, heads=20, kv_heads=20, dim_head=128,
             causal=True, lens=False, dtype="bf16"),
        # one projection on an odd number of tokens
        dict(kind="linear", name="linear 777x2560x7680", tokens=777, dim_in=2560, dim_out=7680, bias=True, dtype="fp16"),
        # loss on the logits of a large vocabulary, a few tokens ignored
        dict(kind="loss", name="loss 4096x50304", tokens=4096, vocab=50304, dtype="bf16"),
        # optimizer step of the benchmark model's shards (half its layers)
        dict(kind="adam", name="adam 4 blocks d2560", layers=4, dim=2560, dim_ff=8192, vocab=10240, dtype="fp16"),
        # the norm of a 13B-shaped layer
        dict(kind="norm", name="rms norm 16384x5120", rows=16384, dim=5120, rms=True, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gpt", "gpt", "gpt", "llama", "llama", "attention", "attention", "linear", "linear", "norm", "loss", "adam"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("gpt", "llama"):
        dim_head = rng.choice([64, 80, 128] if kind == "gpt" else [64, 128])
        hidden = _log(rng, 256, 5120)
        kv = max(1, hidden // dim_head)
        group = rng.choice([1, 1, 4, 8]) if kind == "llama" else 1
        kv = max(1, kv // group)
        heads = kv * group
        dim = heads * dim_head
        ff = max(256, int(dim * rng.choice([2.7, 3.2, 4.0])) // 64 * 64)
        seq = _log(rng, 64, 2048)
        batch = max(1, min(8, _log(rng, 256, 3000) // seq))
        layers = rng.choice([1, 2, 3]) if dim <= 2560 else 1
        vocab = rng.choice([10240, 32000, 50304] if dim >= 1024 else [10240, 10007])
        case = dict(kind=kind, layers=layers, vocab=vocab, heads=heads, dim_head=dim_head, dim_ff=ff, batch=batch, seq=seq,
                    dtype=dtype, train=rng.random() < 0.8)
        if kind == "gpt":
            case.update(activation=rng.choice(["relu", "gelu"]), dense_mask=rng.random() < 0.6)
        else:
            case.update(kv_heads=kv)
        return case
    if kind == "attention":
        seq = _log(rng, 64, 4096)
        group = rng.choice([1, 1, 4, 8])
        kv = rng.choice([1, 2, 4]) if group > 1 else rng.choice([4, 12, 20, 32])
        tokens = _log(rng, 512, 8192)
        return dict(kind=kind, batch=max(1, tokens // seq), seq=seq, heads=kv * group, kv_heads=kv,
                    dim_head=rng.choice([32, 64, 80, 96, 128]), causal=rng.random() < 0.6, lens=rng.random() < 0.4, dtype=dtype)
    if kind == "linear":
        def dim():
            n = _log(rng, 256, 10240)
            return n if rng.random() < 0.15 else max(64, n // 64 * 64) if rng.random() < 0.7 else max(8, n // 8 * 8)
        return dict(kind=kind, tokens=_log(rng, 16, 8192), dim_in=dim(), dim_out=dim(), bias=rng.random() < 0.6, dtype=dtype)
    if kind == "norm":
        return dict(kind=kind, rows=_log(rng, 128, 32768), dim=max(64, _log(rng, 256, 8192) // 8 * 8), rms=rng.random() < 0.5,
                    dtype=dtype)
    if kind == "loss":
        vocab = rng.choice([10240, 32000, 50304, 50257])
        return dict(kind=kind, tokens=_log(rng, 64, 4000), vocab=vocab, dtype=dtype)
    dim = max(256, _log(rng, 256, 2560) // 64 * 64)
    return dict(kind="adam", layers=rng.choice([1, 2, 3]), dim=dim, dim_ff=4 * dim, vocab=10240, dtype=dtype)


# ------------------------------------------------------------------------------------------------------------ inputs
def _start():
    """World-size-1 runtime on the GPU."""
    if not bmt.is_initialized():
        with socket.socket() as s:
            s.bind(("127.0.0.1", 0))
            port = s.getsockname()[1]
        os.environ.update(RANK="0", WORLD_SIZE="1", LOCAL_RANK="0", LOCAL_WORLD_SIZE="1", MASTER_ADDR="127.0.0.1",
                          MASTER_PORT=str(port))
        bmt.init_distributed(seed=0, verbose=False)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen, shape, dtype, std=1.0, mean=0.0):
    return torch.randn(*shape, generator=gen, dtype=dtype, device="cuda").mul_(std).add_(mean)


def _model_shapes(c):
    """Parameter names and shapes of a model case, in checkpoint order."""
    d, inner, ff = c["heads"] * c["dim_head"], c["heads"] * c["dim_head"], c["dim_ff"]
    shapes = {"word_emb.weight": (c["vocab"], d)}
    if c["kind"] == "gpt":
        shapes["pos_emb.weight"] = (c["seq"], d)
    else:
        shapes["lm_head.weight"] = (c["vocab"], d)
    for i in range(c["layers"]):
        p = "transformers.%d." % i
        if c["kind"] == "gpt":
            shapes.update({p + "ln_attn.weight": (d,), p + "ln_attn.bias": (d,),
                           p + "attn.project_qkv.weight": (3 * inner, d), p + "attn.project_qkv.bias": (3 * inner,),
                           p + "attn.project_out.weight": (d, inner), p + "attn.project_out.bias": (d,),
                           p + "ln_ff.weight": (d,), p + "ln_ff.bias": (d,),
                           p + "ff.w_in.weight": (ff, d), p + "ff.w_in.bias": (ff,),
                           p + "ff.w_out.weight": (d, ff), p + "ff.w_out.bias": (d,)})
        else:
            qkv = (c["heads"] + 2 * c["kv_heads"]) * c["dim_head"]
            shapes.update({p + "ln_attn.weight": (d,), p + "attn.project_qkv.weight": (qkv, d),
                           p + "attn.project_out.weight": (d, inner), p + "ln_ff.weight": (d,),
                           p + "ff.w_gate_up.weight": (2 * ff, d), p + "ff.w_out.weight": (d, ff)})
    shapes["layernorm.weight"] = (d,)
    if c["kind"] == "gpt":
        shapes["layernorm.bias"] = (d,)
    return shapes


def _weights(c, gen):
    """Matrices N(0, 0.02), norm weights around one, biases around zero, in the case's data type."""
    dt, out = DTYPES[c["dtype"]], {}
    for name, shape in _model_shapes(c).items():
        norm_weight = len(shape) == 1 and name.endswith("weight")
        out[name] = _randn(gen, shape, dt, 0.02, 1.0 if norm_weight else 0.0)
    return out


def _tokens(c, gen):
    ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=gen, device="cuda")
    return ids[:, :-1].contiguous(), ids[:, 1:].contiguous()


def _scale(c):
    return FP16_SCALE if c["dtype"] == "fp16" else None


def _lens(c, gen):
    """Key counts spread evenly from a quarter of the length to all of it, in an order of the seed's."""
    lens = torch.linspace(0.25, 1.0, c["batch"]).mul(c["seq"]).long().clamp(min=1).cuda()
    return lens[torch.randperm(c["batch"], generator=gen, device="cuda")]


def _attention_inputs(c, gen):
    dt, b, s, d = DTYPES[c["dtype"]], c["batch"], c["seq"], c["dim_head"]
    q = _randn(gen, (b, s, c["heads"], d), dt)
    k, v = (_randn(gen, (b, s, c["kv_heads"], d), dt) for _ in range(2))
    return q, k, v, _randn(gen, q.shape, dt), _lens(c, gen) if c["lens"] else None


def _linear_inputs(c, gen):
    dt = DTYPES[c["dtype"]]
    x = _randn(gen, (1, c["tokens"], c["dim_in"]), dt)
    w = _randn(gen, (c["dim_out"], c["dim_in"]), dt, 0.02)
    return x, w, _randn(gen, (c["dim_out"],), dt, 0.02) if c["bias"] else None, _randn(gen, (1, c["tokens"], c["dim_out"]), dt)


def _norm_inputs(c, gen):
    dt = DTYPES[c["dtype"]]
    x = _randn(gen, (c["rows"], c["dim"]), dt)
    w = _randn(gen, (c["dim"],), dt, 0.02, 1.0)
    return x, w, None if c["rms"] else _randn(gen, (c["dim"],), dt, 0.02), _randn(gen, x.shape, dt)


def _loss_inputs(c, gen):
    x = _randn(gen, (c["tokens"], c["vocab"]), DTYPES[c["dtype"]], 1.5)
    t = torch.randint(0, c["vocab"], (c["tokens"],), generator=gen, device="cuda")
    t[torch.rand(c["tokens"], generator=gen, device="cuda") < 0.03] = -100
    t[0] = 1
    return x, t


def _adam_inputs(c, gen):
    """Flat shards of the blocks and the tables outside them, and loss-scaled gradients."""
    dt, d, ff = DTYPES[c["dtype"]], c["dim"], c["dim_ff"]
    sizes = [4 * d * d + 2 * d * ff + 9 * d + ff] * c["layers"] + [c["vocab"] * d, 512 * d, d, d]
    params = [_randn(gen, (n,), dt, 0.02) for n in sizes]
    return params, [_randn(gen, (n,), dt, 1e-3 * (_scale(c) or 1.0)) for n in sizes]


def prepare(case, seed):
    _start()
    c, gen = case, _gen(seed)
    if c["kind"] in ("gpt", "llama"):
        dt, d = DTYPES[c["dtype"]], c["heads"] * c["dim_head"]
        weights = _weights(c, gen)
        ids, targets = _tokens(c, gen)
        if c["kind"] == "gpt":
            model = bmt.models.GPT(c["layers"], c["vocab"], d, c["dim_head"], c["heads"], c["dim_ff"], c["seq"], bias=True,
                                   dtype=dt, activation=c["activation"], dense_mask=c["dense_mask"])
            pos = torch.arange(c["seq"], device="cuda")[None].expand(c["batch"], -1).contiguous()
            inputs = (ids, pos, torch.ones_like(ids, dtype=torch.bool))
        else:
            model = bmt.models.Llama(c["layers"], c["vocab"], d, c["heads"], c["dim_ff"], num_kv_heads=c["kv_heads"],
                                     dim_head=c["dim_head"], dtype=dt)
            inputs = (ids,)
        model.load_state_dict(weights)
        state = dict(case=c, model=model, inputs=inputs, targets=targets)
        if c["train"]:
            manager = bmt.optim.OptimManager(loss_scale=_scale(c))
            manager.add_optimizer(bmt.optim.AdamOptimizer(model.parameters(), lr=1e-4))
            state.update(manager=manager, loss=bmt.loss.FusedCrossEntropy(ignore_index=-100))
        return state
    if c["kind"] == "attention":
        q, k, v, go, lens = _attention_inputs(c, gen)
        return dict(case=c, leaves=[t.requires_grad_() for t in (q, k, v)], go=go, lens=lens)
    if c["kind"] in ("linear", "norm"):
        x, w, b, go = (_linear_inputs if c["kind"] == "linear" else _norm_inputs)(c, gen)
        return dict(case=c, leaves=[None if t is None else t.requires_grad_() for t in (x, w, b)], go=go)
    if c["kind"] == "loss":
        x, t = _loss_inputs(c, gen)
        return dict(case=c, x=x.requires_grad_(), targets=t, loss=bmt.loss.FusedCrossEntropy(ignore_index=-100))
    params, grads = _adam_inputs(c, gen)
    params = [torch.nn.Parameter(p) for p in params]
    for p, g in zip(params, grads):
        p.grad = g
    optimizer = bmt.optim.AdamOptimizer(params, lr=1e-3, weight_decay=1e-2)
    manager = bmt.optim.OptimManager(loss_scale=_scale(c))
    manager.add_optimizer(optimizer)
    return dict(case=c, params=params, optimizer=optimizer, manager=manager)


# -------------------------------------------------------------------------------------------------------------- pass
def run(state):
    c = state["case"]
    if c["kind"] in ("gpt", "llama"):
        model = state["model"]
        if not c["train"]:
            with torch.no_grad():
                return {"logits": model(*state["inputs"])}
        manager = state["manager"]
        logits = model(*state["inputs"])
        loss = state["loss"](logits.view(-1, logits.shape[-1]), state["targets"].view(-1))
        manager.zero_grad()
        manager.backward(loss)
        out = {"grad " + n: p.grad.reshape(-1) for n, p in model.named_parameters()}
        out.update(logits=logits, loss=loss)
        return out
    if c["kind"] == "attention":
        q, k, v = state["leaves"]
        o = attention_op.attention(q, k, v, causal=c["causal"], kv_lens=state["lens"])
        return [o, *torch.autograd.grad(o, (q, k, v), state["go"])]
    if c["kind"] == "linear":
        x, w, b = state["leaves"]
        y = gemm_op.linear(x, w, b)
        return [y, *torch.autograd.grad(y, [t for t in (x, w, b) if t is not None], state["go"])]
    if c["kind"] == "norm":
        x, w, b = state["leaves"]
        y = norm_op.rms_norm(x, w) if c["rms"] else norm_op.layer_norm(x, w, b)
        return [y, *torch.autograd.grad(y, [t for t in (x, w, b) if t is not None], state["go"])]
    if c["kind"] == "loss":
        loss = state["loss"](state["x"], state["targets"])
        return [loss, *torch.autograd.grad(loss, (state["x"],))]
    manager, optimizer = state["manager"], state["optimizer"]
    norm = manager.clip_grad_norm(optimizer.param_groups, max_norm=1.0)
    manager.step()
    st = [optimizer.state[p] for p in state["params"]]
    return {"norm": norm, "param": [p.detach() for p in state["params"]], "master": [s["_param_fp32"] for s in st],
            "exp_avg": [s["exp_avg"] for s in st], "exp_avg_sq": [s["exp_avg_sq"] for s in st]}


# -------------------------------------------------------------------------------------------------- work and tolerance
def _sizes(c):
    """(all parameters, parameters that multiply every token) of a model case."""
    shapes = _model_shapes(c)
    total = sum(math.prod(s) for s in shapes.values())
    looked_up = "pos_emb.weight" if c["kind"] == "gpt" else "word_emb.weight"
    return total, sum(math.prod(s) for n, s in shapes.items() if len(s) == 2 and n != looked_up)


def work(case):
    c = case
    if c["kind"] in ("gpt", "llama"):
        total, dense = _sizes(c)
        tokens = c["batch"] * c["seq"]
        scores = 4 * c["layers"] * tokens * c["seq"] * c["heads"] * c["dim_head"] * 0.5
        passes = 3 if c["train"] else 1
        # parameters read, gradients and logits written, token ids in
        return {"bytes": total * 2 * (2 if c["train"] else 1) + tokens * c["vocab"] * 2 + tokens * 16,
                "flops": passes * (2 * dense * tokens + scores)}
    if c["kind"] == "attention":
        rows = c["batch"] * c["seq"] * c["dim_head"] * 2
        share = (0.5 if c["causal"] else 1.0) * (0.625 if c["lens"] else 1.0)
        # q, o, do, dq and k, v, dk, dv
        return {"bytes": rows * 4 * (c["heads"] + c["kv_heads"]),
                "flops": 3 * 4 * c["batch"] * c["heads"] * c["seq"] ** 2 * c["dim_head"] * share}
    if c["kind"] == "linear":
        t, i, o = c["tokens"], c["dim_in"], c["dim_out"]
        return {"bytes": 2 * (2 * t * i + 2 * t * o + 2 * i * o + (2 * o if c["bias"] else 0)), "flops": 3 * 2 * t * i * o}
    if c["kind"] == "norm":
        return {"bytes": 2 * 4 * c["rows"] * c["dim"], "flops": 16 * c["rows"] * c["dim"]}
    if c["kind"] == "loss":
        return {"bytes": 2 * 2 * c["tokens"] * c["vocab"], "flops": 8 * c["tokens"] * c["vocab"]}
    d, ff = c["dim"], c["dim_ff"]
    n = (4 * d * d + 2 * d * ff + 9 * d + ff) * c["layers"] + c["vocab"] * d + 514 * d
    # gradient in and out (clipped); master, half parameter and both moments in and out (half parameter out only)
    per = 2 + 2 + 8 + 2 + 2 * (2 if c["dtype"] == "fp16" else 4) + 8
    return {"bytes": per * n, "flops": 20 * n}


def tolerance(case):
    """About four times the error against 64 bits of an operator; a model's gradients are two to three per cent off it in
    fp16 (ReLU inputs that round to the other side of zero) and one to two in bf16, and bounded at 0.03."""
    half = case["dtype"] == "fp16"
    if case["kind"] in ("gpt", "llama"):
        return {"rel": 0.03}
    if case["kind"] == "adam":
        return {"rel": 0.0015 if half else 0.014}
    return {"rel": 0.0012 if half else 0.01}


# ------------------------------------------------------------------------------------------------------------- exact
def _norm64(x, w, b, eps, rms):
    if rms:
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w
    return F.layer_norm(x, (x.shape[-1],), w, b, eps)


def _attend64(q, k, v, causal, lens=None):
    """softmax(q k^T / sqrt(d)) v over (batch, seq, heads, dim), one batch entry at a time (the scores are large)."""
    group, s = q.shape[2] // k.shape[2], q.shape[1]
    outs = []
    for i in range(q.shape[0]):
        ki, vi = (t[i].repeat_interleave(group, dim=1).transpose(0, 1) for t in (k, v))
        score = q[i].transpose(0, 1) @ ki.transpose(1, 2) / math.sqrt(q.shape[-1])
        keep = torch.ones(s, s, dtype=torch.bool, device=q.device)
        if causal:
            keep = keep.tril()
        if lens is not None:
            keep = keep & (torch.arange(s, device=q.device) < lens[i])[None]
        outs.append((torch.softmax(score.masked_fill(~keep, float("-inf")), -1) @ vi).transpose(0, 1))
    return torch.stack(outs)


def _rope64(x, theta=10000.0):
    s, d = x.shape[1], x.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = torch.outer(torch.arange(s, device=x.device, dtype=torch.float64), inv)
    cos, sin = ang.cos()[None, :, None], ang.sin()[None, :, None]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)


def _model64(c, w, ids):
    b, s, h, dh = c["batch"], c["seq"], c["heads"], c["dim_head"]
    x = F.embedding(ids, w["word_emb.weight"])
    if c["kind"] == "gpt":
        x = x + w["pos_emb.weight"][:s][None]
    for i in range(c["layers"]):
        p = lambda n: w["transformers.%d.%s" % (i, n)]  # noqa: E731
        if c["kind"] == "gpt":
            y = _norm64(x, p("ln_attn.weight"), p("ln_attn.bias"), 1e-5, False)
            qkv = F.linear(y, p("attn.project_qkv.weight"), p("attn.project_qkv.bias")).view(b, s, h, 3, dh)
            o = _attend64(qkv[:, :, :, 0], qkv[:, :, :, 1], qkv[:, :, :, 2], True)
            x = x + F.linear(o.reshape(b, s, h * dh), p("attn.project_out.weight"), p("attn.project_out.bias"))
            y = F.linear(_norm64(x, p("ln_ff.weight"), p("ln_ff.bias"), 1e-5, False), p("ff.w_in.weight"), p("ff.w_in.bias"))
            y = torch.relu(y) if c["activation"] == "relu" else F.gelu(y)
            x = x + F.linear(y, p("ff.w_out.weight"), p("ff.w_out.bias"))
        else:
            hk, g = c["kv_heads"], h // c["kv_heads"]
            y = _norm64(x, p("ln_attn.weight"), None, 1e-5, True)
            qkv = F.linear(y, p("attn.project_qkv.weight")).view(b, s, hk, g + 2, dh)
            q, k, v = _rope64(qkv[:, :, :, :g].reshape(b, s, h, dh)), _rope64(qkv[:, :, :, g]), qkv[:, :, :, g + 1]
            x = x + F.linear(_attend64(q, k, v, True).reshape(b, s, h * dh), p("attn.project_out.weight"))
            gate, up = F.linear(_norm64(x, p("ln_ff.weight"), None, 1e-5, True), p("ff.w_gate_up.weight")).chunk(2, -1)
            x = x + F.linear(F.silu(gate) * up, p("ff.w_out.weight"))
    if c["kind"] == "gpt":
        return F.linear(_norm64(x, w["layernorm.weight"], w["layernorm.bias"], 1e-5, False), w["word_emb.weight"])
    return F.linear(_norm64(x, w["layernorm.weight"], None, 1e-6, True), w["lm_head.weight"])


def exact(case, seed):
    c, gen = case, _gen(seed)
    if c["kind"] in ("gpt", "llama"):
        w = {n: t.double().requires_grad_(c["train"]) for n, t in _weights(c, gen).items()}
        ids, targets = _tokens(c, gen)
        logits = _model64(c, w, ids)
        if not c["train"]:
            return {"logits": logits}
        loss = F.cross_entropy(logits.view(-1, c["vocab"]), targets.view(-1))
        grads = torch.autograd.grad(loss * (_scale(c) or 1.0), list(w.values()))
        out = {"grad " + n: g.reshape(-1) for n, g in zip(w, grads)}
        out.update(logits=logits.detach(), loss=loss.detach())
        return out
    if c["kind"] == "attention":
        q, k, v, go, lens = _attention_inputs(c, gen)
        q, k, v = (t.double().requires_grad_() for t in (q, k, v))
        o = _attend64(q, k, v, c["causal"], lens)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), go.double())]
    if c["kind"] in ("linear", "norm"):
        x, w, b, go = (_linear_inputs if c["kind"] == "linear" else _norm_inputs)(c, gen)
        leaves = [t.double().requires_grad_() for t in (x, w, b) if t is not None]
        x, w, b = (leaves + [None])[:3]
        y = F.linear(x, w, b) if c["kind"] == "linear" else _norm64(x, w, b, 1e-6 if c["rms"] else 1e-5, c["rms"])
        return [y.detach(), *torch.autograd.grad(y, leaves, go.double())]
    if c["kind"] == "loss":
        x, t = _loss_inputs(c, gen)
        x = x.double().requires_grad_()
        loss = F.cross_entropy(x, t, ignore_index=-100)
        return [loss.detach(), *torch.autograd.grad(loss, (x,))]
    params, grads = _adam_inputs(c, gen)
    s, out = _scale(c) or 1.0, {"param": [], "master": [], "exp_avg": [], "exp_avg_sq": []}
    norm = math.sqrt(sum(float(g.double().square().sum()) for g in grads))
    coef = min(1.0, s / (norm + 1e-6))
    for p, g in zip(params, grads):
        g, p = g.double() * coef, p.double()
        true = g / s
        p = p - 1e-3 * (true / (true.abs() + 1e-8) + 1e-2 * p)
        out["param"].append(p)
        out["master"].append(p)
        kept = g if c["dtype"] == "fp16" else true     # fp16 moments are kept in loss-scaled units
        out["exp_avg"].append(0.1 * kept)
        out["exp_avg_sq"].append(0.001 * kept * kept / (s if c["dtype"] == "fp16" else 1.0))
        del g, p, true, kept
    out["norm"] = torch.tensor(norm / s, dtype=torch.float64)
    return out


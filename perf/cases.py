"""The work this framework does for its users, as a list of timed cases.

A case is one call or one short chain of calls of the operator library (``autoparallel_b200.ops``), of the optimizer
(``autoparallel_b200.optim.AdamW``) or of a model planned with ``AutoParallel``, on one GPU, forward and backward the way
a training step runs them.  Sizes are those of the repository's own models (``models/llama3.py``: the 8B and the debug
configuration; ``models/moe.py``: 64 experts, top-8, d 2048, hidden 1408), of its kernel benchmark and of its tests, and
generic ones around them: odd token counts, few rows, narrow projections.

Kinds
  step     a whole planned decoder (AutoParallel, bf16 compute over fp32 parameters): loss and all parameter gradients
  attn     attention half of a decoder block: norm, q / k / v projections, rotary embedding, attention, output projection
  mlp      feed-forward half of a block: norm, two projections, SwiGLU, projection back
  moe      routed-expert region: slots, dispatch into capacity buffers, grouped expert GEMMs, weighted combine
  head     final norm, vocabulary projection and cross-entropy loss
  embed    token embedding and its table gradient
  linear   one projection (``mm_nd``); forward only for inference-sized inputs
  norm     RMSNorm alone
  adamw    one optimizer step over a list of parameters, with the bf16 copy that the next forward reads
"""
from __future__ import annotations

import math

import torch

import autoparallel_b200.ops as K
from autoparallel_b200.ops import library as L

EPS = 1e-5
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
_DT = {"bf16": BF16, "fp32": F32}


# ------------------------------------------------------------------------------------------------ the list
def listed():
    return [
        # the smallest whole call: a debug-sized decoder; latency, launches and host work are what it costs
        {"name": "step_debug", "kind": "step", "dim": 256, "layers": 2, "heads": 8, "kv": 4, "hidden": 512, "vocab": 1024,
         "batch": 2, "seq": 256},
        # one attention layer of the 8B model over one sequence of full length
        {"name": "attn_8b", "kind": "attn", "dim": 4096, "heads": 32, "kv": 8, "batch": 1, "seq": 8192},
        # one feed-forward layer of the 8B model: the bulk of a training step
        {"name": "mlp_8b", "kind": "mlp", "tokens": 8192, "dim": 4096, "hidden": 14336},
        # the shared expert of the MoE model on a short batch with a ragged token count
        {"name": "mlp_ragged", "kind": "mlp", "tokens": 999, "dim": 2048, "hidden": 1408},
        # the routed experts of the MoE model on one rank's 8192 tokens
        {"name": "moe_8k", "kind": "moe", "tokens": 8192, "dim": 2048, "hidden": 1408, "experts": 64, "topk": 8, "blocks": 1,
         "factor": 1.25, "zipf": 0.0},
        # the same experts on few tokens, with skewed routing and the planner's eight dispatch blocks
        {"name": "moe_small", "kind": "moe", "tokens": 1000, "dim": 2048, "hidden": 1408, "experts": 64, "topk": 8, "blocks": 8,
         "factor": 1.25, "zipf": 0.5},
        # vocabulary projection and loss of the 8B model: the largest GEMMs and the largest activations
        {"name": "head_8b", "kind": "head", "tokens": 8192, "dim": 4096, "vocab": 128256},
        # token embedding of the 8B model and the gradient of its table
        {"name": "embed_8b", "kind": "embed", "tokens": 8192, "dim": 4096, "vocab": 128256, "dtype": "bf16"},
        # router projection of an MoE layer: a narrow output, and a weight gradient that contracts over all tokens
        {"name": "linear_router", "kind": "linear", "rows": 8192, "k": 2048, "n": 64, "grad": True},
        # a projection of the 8B model on a handful of rows, forward only (inference)
        {"name": "linear_few_rows", "kind": "linear", "rows": 16, "k": 4096, "n": 4096, "grad": False},
        # RMSNorm of an fp32 model on an odd number of rows
        {"name": "norm_fp32", "kind": "norm", "rows": 2047, "dim": 2048, "dtype": "fp32"},
        # optimizer step over the parameters of one 8B block
        {"name": "adamw_block", "kind": "adamw", "dim": 4096, "kvdim": 1024, "hidden": 14336, "layers": 1},
    ]


def _log_int(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm; odd and ragged values as they come."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_mult(rng, lo, hi, m):
    return max(lo, _log_int(rng, lo, hi) // m * m)


def draw(rng):
    kind = rng.choice(["step", "attn", "mlp", "moe", "head", "embed", "linear", "norm", "adamw"])
    if kind == "step":
        heads = rng.choice([4, 8])
        hd = rng.choice([32, 64])
        return {"kind": kind, "dim": heads * hd, "layers": rng.randint(1, 3), "heads": heads, "kv": heads // rng.choice([1, 2]),
                "hidden": _log_mult(rng, 256, 1024, 64), "vocab": _log_mult(rng, 512, 4096, 64), "batch": rng.randint(1, 4),
                "seq": _log_mult(rng, 64, 256, 32)}
    if kind == "attn":
        dim, heads, kv = rng.choice([(4096, 32, 8), (2048, 16, 4), (1024, 16, 8), (2048, 32, 8)])
        seq = _log_int(rng, 128, 4096)
        return {"kind": kind, "dim": dim, "heads": heads, "kv": kv, "batch": rng.randint(1, max(1, min(8, 8192 // seq))), "seq": seq}
    if kind == "mlp":
        dim, hidden = rng.choice([(4096, 14336), (2048, 1408), (2048, 5632), (1024, 2816), (256, 512)])
        return {"kind": kind, "tokens": _log_int(rng, 64, 8192), "dim": dim, "hidden": hidden}
    if kind == "moe":
        dim, hidden, experts, topk = rng.choice([(2048, 1408, 64, 8), (1024, 704, 32, 4), (2048, 1408, 16, 2), (128, 64, 8, 2)])
        blocks = rng.choice([1, 1, 2, 8])
        return {"kind": kind, "tokens": _log_mult(rng, 128, 8192, blocks), "dim": dim, "hidden": hidden, "experts": experts,
                "topk": topk, "blocks": blocks, "factor": rng.choice([1.0, 1.25, 2.0]), "zipf": rng.choice([0.0, 0.5, 1.0])}
    if kind == "head":
        return {"kind": kind, "tokens": _log_int(rng, 32, 4096), "dim": rng.choice([1024, 2048, 4096]),
                "vocab": rng.choice([128256, 102400, 50264, 32064, _log_mult(rng, 1024, 65536, 8)])}
    if kind == "embed":
        return {"kind": kind, "tokens": _log_int(rng, 16, 16384), "dim": rng.choice([256, 1024, 2048, 4096]),
                "vocab": rng.choice([128256, 102400, 50257, 32000, 1000]), "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "linear":
        return {"kind": kind, "rows": _log_int(rng, 1, 8192), "k": _log_mult(rng, 64, 8192, 8), "n": _log_mult(rng, 8, 8192, 8),
                "grad": rng.random() < 0.5}
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 16384), "dim": rng.choice([256, 768, 1024, 2048, 4096, 5120, 8192]),
                "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    dim = rng.choice([256, 512, 1024, 2048, 4096])
    return {"kind": kind, "dim": dim, "kvdim": dim // 4, "hidden": _log_mult(rng, dim, dim * 7 // 2, 8),
            "layers": rng.randint(1, max(1, min(8, (4096 // dim) ** 2)))}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=BF16):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F32).mul_(std).to(dtype)


def _leaf(t):
    return t.requires_grad_(True)


def _rope_tables(hd, n):
    inv = 1.0 / (500000.0 ** (torch.arange(0, hd, 2, device="cuda", dtype=F32) / hd))
    ang = torch.outer(torch.arange(n, device="cuda", dtype=F32), inv)
    return ang.cos(), ang.sin()


def _zipf_ids(g, n, vocab):
    """Token ids with the skew of text: rank r has weight 1 / r."""
    u = torch.rand(n, generator=g, device="cuda", dtype=F64)
    rank = torch.exp(u * math.log(vocab + 1.0)).floor().long() - 1
    return torch.randperm(vocab, generator=g, device="cuda")[rank.clamp_(0, vocab - 1)]


def _moe_capacity(c):
    return max(1, math.ceil(c["factor"] * (c["tokens"] // c["blocks"]) * c["topk"] / c["experts"]))


def _adamw_shapes(c):
    d, kv, h = c["dim"], c["kvdim"], c["hidden"]
    return [(d, d), (kv, d), (kv, d), (d, d), (h, d), (h, d), (d, h), (d,), (d,)] * c["layers"]


ADAMW = dict(lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
ADAMW_STEP = 100  # steps taken before the timed one


def _step_params(c, seed):
    """Parameters of the decoder by name, fp32."""
    g = _gen(seed)
    d, hd, h = c["dim"], c["dim"] // c["heads"], c["hidden"]
    p = {"tok_embeddings.weight": _randn(g, c["vocab"], d, std=0.02, dtype=F32)}
    for i in range(c["layers"]):
        a, f = f"layers.{i}.attention.", f"layers.{i}.feed_forward."
        p[a + "wq.weight"] = _randn(g, c["heads"] * hd, d, std=0.02, dtype=F32)
        p[a + "wk.weight"] = _randn(g, c["kv"] * hd, d, std=0.02, dtype=F32)
        p[a + "wv.weight"] = _randn(g, c["kv"] * hd, d, std=0.02, dtype=F32)
        p[a + "wo.weight"] = _randn(g, d, c["heads"] * hd, std=0.02, dtype=F32)
        p[f + "w1.weight"] = _randn(g, h, d, std=0.02, dtype=F32)
        p[f + "w3.weight"] = _randn(g, h, d, std=0.02, dtype=F32)
        p[f + "w2.weight"] = _randn(g, d, h, std=0.02, dtype=F32)
        p[f"layers.{i}.attention_norm.weight"] = 1.0 + _randn(g, d, std=0.1, dtype=F32)
        p[f"layers.{i}.ffn_norm.weight"] = 1.0 + _randn(g, d, std=0.1, dtype=F32)
    p["norm.weight"] = 1.0 + _randn(g, d, std=0.1, dtype=F32)
    p["output.weight"] = _randn(g, c["vocab"], d, std=0.02, dtype=F32)
    tok = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g, device="cuda")
    lab = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g, device="cuda")
    return p, tok, lab


def _inputs(c, seed):
    """Tensors of a case by name (``step`` apart), made from the seed alone."""
    g = _gen(seed)
    k = c["kind"]
    if k == "attn":
        d, hd = c["dim"], c["dim"] // c["heads"]
        t = {"x": _randn(g, c["batch"], c["seq"], d), "g": (1.0 + 0.1 * _randn(g, d, dtype=F32)).to(BF16),
             "wq": _randn(g, c["heads"] * hd, d, std=0.02), "wk": _randn(g, c["kv"] * hd, d, std=0.02),
             "wv": _randn(g, c["kv"] * hd, d, std=0.02), "wo": _randn(g, d, c["heads"] * hd, std=0.02),
             "dy": _randn(g, c["batch"], c["seq"], d)}
        t["cos"], t["sin"] = _rope_tables(hd, c["seq"])
    elif k == "mlp":
        n, d, h = c["tokens"], c["dim"], c["hidden"]
        t = {"x": _randn(g, 1, n, d), "g": (1.0 + 0.1 * _randn(g, d, dtype=F32)).to(BF16), "w1": _randn(g, h, d, std=0.02),
             "w3": _randn(g, h, d, std=0.02), "w2": _randn(g, d, h, std=0.02), "dy": _randn(g, 1, n, d)}
    elif k == "moe":
        n, d, h, e = c["tokens"], c["dim"], c["hidden"], c["experts"]
        scores = torch.randn(n, e, generator=g, device="cuda")
        if c["zipf"]:
            scores = scores - c["zipf"] * torch.log(torch.arange(1, e + 1, device="cuda", dtype=F32))
        w, idx = torch.topk(torch.softmax(scores, -1), c["topk"], dim=-1)
        t = {"idx": idx, "gate": (w / w.sum(-1, keepdim=True)).to(BF16), "x": _randn(g, n, d), "w1": _randn(g, e, d, h, std=0.02),
             "w3": _randn(g, e, d, h, std=0.02), "w2": _randn(g, e, h, d, std=0.02), "dy": _randn(g, n, d)}
    elif k == "head":
        t = {"x": _randn(g, 1, c["tokens"], c["dim"]), "g": (1.0 + 0.1 * _randn(g, c["dim"], dtype=F32)).to(BF16),
             "w": _randn(g, c["vocab"], c["dim"], std=0.02), "labels": _zipf_ids(g, c["tokens"], c["vocab"]).view(1, -1)}
    elif k == "embed":
        dt = _DT[c["dtype"]]
        t = {"w": _randn(g, c["vocab"], c["dim"], std=0.02, dtype=dt), "ids": _zipf_ids(g, c["tokens"], c["vocab"]).view(1, -1),
             "dy": _randn(g, 1, c["tokens"], c["dim"], dtype=dt)}
    elif k == "linear":
        t = {"x": _randn(g, c["rows"], c["k"]), "w": _randn(g, c["n"], c["k"], std=0.02)}
        if c["grad"]:
            t["dy"] = _randn(g, c["rows"], c["n"])
    elif k == "norm":
        dt = _DT[c["dtype"]]
        t = {"x": _randn(g, c["rows"], c["dim"], dtype=dt), "g": (1.0 + 0.1 * _randn(g, c["dim"], dtype=F32)).to(dt),
             "dy": _randn(g, c["rows"], c["dim"], dtype=dt)}
    else:
        t = {"p": [], "grad": [], "m": [], "v": []}
        for s in _adamw_shapes(c):
            t["p"].append(_randn(g, *s, std=0.02, dtype=F32))
            t["grad"].append(_randn(g, *s, std=1e-3, dtype=F32))
            t["m"].append(_randn(g, *s, std=3e-4, dtype=F32))
            t["v"].append(_randn(g, *s, std=1e-3, dtype=F32).square_())
    return t


_DIFF = {"attn": ("x", "g", "wq", "wk", "wv", "wo"), "mlp": ("x", "g", "w1", "w3", "w2"), "moe": ("x", "gate", "w1", "w3", "w2"),
         "head": ("x", "g", "w"), "embed": ("w",), "linear": ("x", "w"), "norm": ("x", "g")}


def _prepare_step(c, seed):
    import torch.distributed as dist
    from torch.distributed.device_mesh import init_device_mesh
    from torch.distributed.tensor.placement_types import Shard

    from autoparallel_b200 import AutoParallel, ForwardInputs
    from autoparallel_b200.models.llama3 import LlamaConfig, Transformer
    from autoparallel_b200.parallel.frontend.mp_cast import MPPolicy

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    mesh = init_device_mesh("cuda", (1,), mesh_dim_names=("dp",))
    cfg = LlamaConfig(dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"], n_kv_heads=c["kv"], ffn_hidden=c["hidden"],
                      vocab_size=c["vocab"], max_seq_len=c["seq"])
    with torch.device("meta"):
        model = Transformer(cfg)

    def input_fn():
        ids = (c["batch"], c["seq"])
        return ForwardInputs((torch.randint(0, c["vocab"], ids),), {"labels": torch.randint(0, c["vocab"], ids)})

    with AutoParallel(model, input_fn, mesh, MPPolicy(BF16, F32)) as ap:
        ap.add_parameter_memory_constraint()
        ap.add_input_constraints([(Shard(0),)] * 2)
        ap.optimize_placement()
        pm = ap.apply_placement()
    pm.to_empty(device="cuda")
    pm.init_weights(seed=0)
    values, tok, lab = _step_params(c, seed)
    params = dict(pm.named_parameters())
    with torch.no_grad():
        for name, v in values.items():
            params[name].to_local().copy_(v)
    return {"case": c, "model": pm, "params": [params[n] for n in values], "tok": tok, "lab": lab}


def prepare(case, seed):
    c = case
    if c["kind"] == "step":
        return _prepare_step(c, seed)
    t = _inputs(c, seed)
    if c["kind"] == "adamw":
        from autoparallel_b200.optim import AdamW

        params = [torch.nn.Parameter(p) for p in t["p"]]
        opt = AdamW(params, emit_bf16=True, **ADAMW)
        for p, gr, m, v in zip(params, t["grad"], t["m"], t["v"]):
            p.grad = gr
            opt.state[p] = {"step": torch.tensor(float(ADAMW_STEP)), "exp_avg": m, "exp_avg_sq": v}
        return {"case": c, "opt": opt, "params": params}
    state = {"case": c, **t}
    if c.get("grad", True):
        for n in _DIFF[c["kind"]]:
            state[n] = _leaf(state[n])
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _linear(x, w):
    return K.ops.mm_nd(x, w, True, x.dtype)


def _attn_layer(s):
    c, x = s["case"], s["x"]
    b, n, d = x.shape
    hd = d // c["heads"]
    h = K.rms_norm(x, s["g"], EPS)
    q = K.rope(_linear(h, s["wq"]).view(b, n, c["heads"], hd), s["cos"], s["sin"])
    k = K.rope(_linear(h, s["wk"]).view(b, n, c["kv"], hd), s["cos"], s["sin"])
    v = _linear(h, s["wv"]).view(b, n, c["kv"], hd)
    return x + _linear(K.attention(q, k, v, causal=True).view(b, n, d), s["wo"])


def _mlp_layer(s):
    h = K.rms_norm(s["x"], s["g"], EPS)
    return s["x"] + _linear(K.swiglu(_linear(h, s["w1"]), _linear(h, s["w3"])), s["w2"])


def _moe_layer(s):
    c = s["case"]
    e, nb, cap, d = c["experts"], c["blocks"], _moe_capacity(c), c["dim"]
    slot = K.moe_slots(s["idx"], e, cap, nb)
    h = K.moe_dispatch(s["x"], slot, e, cap, nb).view(e, nb * cap, d)
    y = K.grouped_mm(K.swiglu(K.grouped_mm(h, s["w1"]), K.grouped_mm(h, s["w3"])), s["w2"])
    return K.moe_combine(y.view(e, nb, cap, d), slot, s["gate"])


def run(state):
    s, c = state, state["case"]
    k = c["kind"]
    if k == "step":
        s["model"].zero_grad(set_to_none=True)
        loss = s["model"](s["tok"], labels=s["lab"])
        loss.backward()
        return [loss.detach()] + [p.grad.to_local() for p in s["params"]]
    if k == "adamw":
        s["opt"].step()
        st = s["opt"].state
        return ([p.detach() for p in s["params"]] + [st[p]["exp_avg"] for p in s["params"]] + [st[p]["exp_avg_sq"] for p in s["params"]]
                + [K.dtype_cast(p.detach(), BF16) for p in s["params"]])
    if k == "head":
        loss = K.cross_entropy(_linear(K.rms_norm(s["x"], s["g"], EPS), s["w"]), s["labels"])
        return [loss.detach(), *torch.autograd.grad(loss, [s[n] for n in _DIFF[k]])]
    if k == "linear" and not c["grad"]:
        return [_linear(s["x"], s["w"])]
    if k == "attn":
        y = _attn_layer(s)
    elif k == "mlp":
        y = _mlp_layer(s)
    elif k == "moe":
        y = _moe_layer(s)
    elif k == "embed":
        y = L.embedding(s["w"], s["ids"])
    elif k == "linear":
        y = _linear(s["x"], s["w"])
    else:
        y = K.rms_norm(s["x"], s["g"], EPS)
    return [y.detach(), *torch.autograd.grad(y, [s[n] for n in _DIFF[k]], s["dy"])]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c = case
    k = c["kind"]
    if k == "step":
        d, hd, h, v, n = c["dim"], c["dim"] // c["heads"], c["hidden"], c["vocab"], c["batch"] * c["seq"]
        dense = c["layers"] * (2 * d * c["heads"] * hd + 2 * d * c["kv"] * hd + 3 * d * h) + v * d
        attn = c["layers"] * c["batch"] * c["heads"] * 7 * c["seq"] ** 2 * hd  # causal: half of 4 + 10 per score
        params = dense + v * d + (2 * c["layers"] + 1) * d
        return {"bytes": 8 * params + 16 * n, "flops": 6 * dense * n + attn}
    if k == "attn":
        d, hd, n = c["dim"], c["dim"] // c["heads"], c["batch"] * c["seq"]
        w = 2 * d * c["heads"] * hd + 2 * d * c["kv"] * hd
        return {"bytes": 2 * (4 * n * d + 2 * w + 2 * d) + 4 * c["seq"] * hd,
                "flops": 6 * n * w + c["batch"] * c["heads"] * 7 * c["seq"] ** 2 * hd}
    if k == "mlp":
        n, d, h = c["tokens"], c["dim"], c["hidden"]
        return {"bytes": 2 * (4 * n * d + 6 * d * h + 2 * d), "flops": 18 * n * d * h}
    if k == "moe":
        n, d, h, e = c["tokens"], c["dim"], c["hidden"], c["experts"]
        rows = min(n * c["topk"], e * c["blocks"] * _moe_capacity(c))  # assignments that can be kept
        return {"bytes": 2 * (4 * n * d + 6 * e * d * h) + n * c["topk"] * 12, "flops": 18 * rows * d * h}
    if k == "head":
        n, d, v = c["tokens"], c["dim"], c["vocab"]
        return {"bytes": 2 * (2 * n * d + 2 * v * d + 2 * d) + 8 * n, "flops": 6 * n * d * v}
    if k == "embed":
        b = 2 if c["dtype"] == "bf16" else 4
        return {"bytes": b * (3 * c["tokens"] * c["dim"] + c["vocab"] * c["dim"]) + 8 * c["tokens"], "flops": c["tokens"] * c["dim"]}
    if k == "linear":
        r, kk, n = c["rows"], c["k"], c["n"]
        if not c["grad"]:
            return {"bytes": 2 * (r * kk + n * kk + r * n), "flops": 2 * r * kk * n}
        return {"bytes": 2 * (2 * r * kk + 2 * n * kk + 2 * r * n), "flops": 6 * r * kk * n}
    if k == "norm":
        b = 2 if c["dtype"] == "bf16" else 4
        return {"bytes": b * (4 * c["rows"] * c["dim"] + 2 * c["dim"]), "flops": 12 * c["rows"] * c["dim"]}
    n = sum(math.prod(s) for s in _adamw_shapes(c))
    return {"bytes": 30 * n, "flops": 15 * n}


def tolerance(case):
    k = case["kind"]
    if k in ("embed", "norm"):
        # sums in fp32, one rounding into the result's type
        return {"rel": 7e-3 if case["dtype"] == "bf16" else 1e-5}
    return {"rel": {"step": 4e-2, "attn": 3e-2, "mlp": 2e-2, "moe": 2e-2, "head": 1e-2, "linear": 7e-3, "adamw": 1e-4}[k]}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _norm64(x, g):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * g


def _rope64(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    co, si = cos[None, :, None, :], sin[None, :, None, :]
    return torch.stack((a * co - b * si, a * si + b * co), -1).reshape(x.shape)


class _Attention64(torch.autograd.Function):
    """Causal attention, one head at a time, so that one score matrix is in memory at once."""

    @staticmethod
    def _probs(q, k):
        s = (q @ k.t()) * q.shape[-1] ** -0.5
        return torch.softmax(s.masked_fill_(torch.ones_like(s, dtype=torch.bool).triu_(1), -math.inf), -1)

    @staticmethod
    def forward(ctx, q, k, v):
        ctx.save_for_backward(q, k, v)
        rep = q.shape[2] // k.shape[2]
        o = torch.empty_like(q)
        for b in range(q.shape[0]):
            for h in range(q.shape[2]):
                o[b, :, h] = _Attention64._probs(q[b, :, h], k[b, :, h // rep]) @ v[b, :, h // rep]
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        rep, scale = q.shape[2] // k.shape[2], q.shape[-1] ** -0.5
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for b in range(q.shape[0]):
            for h in range(q.shape[2]):
                j = h // rep
                p = _Attention64._probs(q[b, :, h], k[b, :, j])
                dv[b, :, j] += p.t() @ do[b, :, h]
                dp = do[b, :, h] @ v[b, :, j].t()
                ds = p * (dp - (p * dp).sum(-1, keepdim=True)) * scale
                dq[b, :, h] = ds @ k[b, :, j]
                dk[b, :, j] += ds.t() @ q[b, :, h]
        return dq, dk, dv


def _attn64(x, g, wq, wk, wv, wo, cos, sin, heads, kv):
    b, n, d = x.shape
    hd = d // heads
    h = _norm64(x, g)
    q = _rope64((h @ wq.t()).view(b, n, heads, hd), cos, sin)
    k = _rope64((h @ wk.t()).view(b, n, kv, hd), cos, sin)
    return x + _Attention64.apply(q, k, (h @ wv.t()).view(b, n, kv, hd)).reshape(b, n, d) @ wo.t()


def _mlp64(x, g, w1, w3, w2):
    h = _norm64(x, g)
    return x + (torch.nn.functional.silu(h @ w1.t()) * (h @ w3.t())) @ w2.t()


def _moe64(c, t):
    n, d, e, k, nb, cap = c["tokens"], c["dim"], c["experts"], c["topk"], c["blocks"], _moe_capacity(c)
    idx = t["idx"].view(nb, -1)
    order = torch.argsort(idx, dim=1, stable=True)
    first = torch.searchsorted(torch.gather(idx, 1, order).contiguous(), torch.arange(e, device="cuda").expand(nb, e).contiguous())
    rank = torch.empty_like(idx).scatter_(1, order, torch.arange(idx.shape[1], device="cuda").expand_as(idx)) - torch.gather(first, 1, idx)
    keep = (rank < cap).reshape(-1)  # arrival rank inside (block, expert), token-major
    tok = torch.arange(n, device="cuda").repeat_interleave(k)[keep]
    exp, wgt = t["idx"].reshape(-1)[keep], t["gate"].reshape(-1)[keep]
    out = torch.zeros_like(t["x"])
    for j in range(e):
        m = exp == j
        rows = t["x"][tok[m]]
        y = (torch.nn.functional.silu(rows @ t["w1"][j]) * (rows @ t["w3"][j])) @ t["w2"][j]
        out = out.index_add(0, tok[m], y * wgt[m].unsqueeze(1))
    return out


def _xent64(logits, labels):
    return torch.nn.functional.cross_entropy(logits.reshape(-1, logits.shape[-1]), labels.reshape(-1))


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "step":
        values, tok, lab = _step_params(c, seed)
        p = {n: v.double().requires_grad_(True) for n, v in values.items()}
        cos, sin = (t.double() for t in _rope_tables(c["dim"] // c["heads"], c["seq"]))
        h = p["tok_embeddings.weight"][tok]
        for i in range(c["layers"]):
            a, f = f"layers.{i}.attention.", f"layers.{i}.feed_forward."
            h = _attn64(h, p[f"layers.{i}.attention_norm.weight"], p[a + "wq.weight"], p[a + "wk.weight"], p[a + "wv.weight"],
                        p[a + "wo.weight"], cos, sin, c["heads"], c["kv"])
            h = _mlp64(h, p[f"layers.{i}.ffn_norm.weight"], p[f + "w1.weight"], p[f + "w3.weight"], p[f + "w2.weight"])
        loss = _xent64(_norm64(h, p["norm.weight"]) @ p["output.weight"].t(), lab)
        return [loss.detach(), *torch.autograd.grad(loss, list(p.values()))]
    t = _inputs(c, seed)
    if k == "adamw":
        b1, b2 = ADAMW["betas"]
        step = ADAMW_STEP + 1
        out = [[], [], [], []]
        for p, g, m, v in zip(t["p"], t["grad"], t["m"], t["v"]):
            p, g, m, v = p.double(), g.double(), m.double(), v.double()
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p * (1 - ADAMW["lr"] * ADAMW["weight_decay"])
            p = p - ADAMW["lr"] * (m / (1 - b1**step)) / ((v / (1 - b2**step)).sqrt() + ADAMW["eps"])
            for o, val in zip(out, (p, m, v, p)):
                o.append(val)
        return sum(out, [])
    if k == "embed":
        dw = torch.zeros(c["vocab"], c["dim"], device="cuda", dtype=F64)
        dw.index_add_(0, t["ids"].reshape(-1), t["dy"].reshape(-1, c["dim"]).double())
        return [t["w"][t["ids"]].double(), dw]
    grad = c.get("grad", True)
    for n, v in t.items():
        if v.is_floating_point():
            t[n] = v.double()
    if grad:
        for n in _DIFF[k]:
            t[n] = _leaf(t[n])
    if k == "head":
        loss = _xent64(_norm64(t["x"], t["g"]) @ t["w"].t(), t["labels"])
        return [loss.detach(), *torch.autograd.grad(loss, [t[n] for n in _DIFF[k]])]
    if k == "attn":
        y = _attn64(t["x"], t["g"], t["wq"], t["wk"], t["wv"], t["wo"], t["cos"], t["sin"], c["heads"], c["kv"])
    elif k == "mlp":
        y = _mlp64(t["x"], t["g"], t["w1"], t["w3"], t["w2"])
    elif k == "moe":
        y = _moe64(c, t)
    elif k == "linear":
        y = t["x"] @ t["w"].t()
    else:
        y = _norm64(t["x"], t["g"])
    if not grad:
        return [y]
    return [y.detach(), *torch.autograd.grad(y, [t[n] for n in _DIFF[k]], t["dy"])]

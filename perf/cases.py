"""Workloads on one GPU whose speed matters to a user of this library, with their sizes, inputs,
lower bounds of work and tolerances.

    mlp_step      one training step (forward, loss, backward, SGD) of the SwiGLU MLP stack
    mlp_forward   the forward pass alone: evaluation, or a batch of tokens being decoded
    moe_step      one training step of the mixture-of-experts layer
    moe_forward   its forward pass alone on a small batch
    gemm          one matrix product in any operand layout, rounded, accumulated or kept in float32
    sgd           the optimizer update of one flat parameter bucket

A case is a dict of plain values; ``kind`` is one of the above and the rest are its sizes.
"""
import math

import torch

from megray_b200.models import MoEConfig, MoELayer, TPMLPConfig, TPMLPStack
from megray_b200.ops import EPI_ACCUM, EPI_STORE, EPI_STORE_F32, gemm, sgd_step

_EPILOGUES = {"store": EPI_STORE, "accum": EPI_ACCUM, "f32": EPI_STORE_F32}


def listed():
    return [
        # The smallest training step of the test suite: every kernel is tiny, launches count.
        {"name": "mlp_step_tiny", "kind": "mlp_step", "d_model": 256, "ffn": 512, "tokens": 256, "layers": 2},
        # A mid-sized model on one GPU: many products of tens of microseconds each.
        {"name": "mlp_step_medium", "kind": "mlp_step", "d_model": 2048, "ffn": 7168, "tokens": 4096, "layers": 4},
        # One rank's matrix products of the benchmark model sharded over 8 GPUs (ffn 28672 / 8).
        {"name": "mlp_step_eighth", "kind": "mlp_step", "d_model": 8192, "ffn": 3584, "tokens": 32768, "layers": 4},
        # The benchmark model itself on one GPU (bench.py).
        {"name": "mlp_step_full", "kind": "mlp_step", "d_model": 8192, "ffn": 28672, "tokens": 32768, "layers": 4},
        # The benchmark model with one small batch of tokens, as in decoding: bound by reading the weights.
        {"name": "mlp_forward_decode", "kind": "mlp_forward", "d_model": 8192, "ffn": 28672, "tokens": 128, "layers": 4},
        # The benchmark model on one sequence of 4096 tokens (evaluation, prefill).
        {"name": "mlp_forward_prefill", "kind": "mlp_forward", "d_model": 8192, "ffn": 28672, "tokens": 4096, "layers": 4},
        # The test suite's MoE layer: 1000 tokens, ragged expert segments.
        {"name": "moe_step_tiny", "kind": "moe_step", "experts": 8, "hidden": 256, "ffn": 384, "tokens": 1000},
        # One rank's share of the benchmark MoE layer on 8 GPUs: 8 experts, 16384 tokens.
        {"name": "moe_step_eighth", "kind": "moe_step", "experts": 8, "hidden": 4096, "ffn": 14336, "tokens": 16384},
        # One rank's share on 4 GPUs (16 experts) with a small batch: a few rows per expert.
        {"name": "moe_forward_decode", "kind": "moe_forward", "experts": 16, "hidden": 4096, "ffn": 14336, "tokens": 250},
        # A small ragged product of the test suite (every dimension off the tile).
        {"name": "gemm_small", "kind": "gemm", "m": 300, "n": 264, "k": 200, "a_mn": False, "b_mn": False,
         "epilogue": "store"},
        # An ordinary ragged product with both operands stored transposed, as a weight gradient is.
        {"name": "gemm_ragged", "kind": "gemm", "m": 1544, "n": 3080, "k": 5000, "a_mn": True, "b_mn": True,
         "epilogue": "store"},
        # The parameters of the data-parallel ResNet-50 as one bucket, SGD with momentum.
        {"name": "sgd_resnet50", "kind": "sgd", "n": 25557032, "momentum": 0.9, "weight_decay": 1e-4},
    ]


# ----------------------------------------------------------------------------------- drawn cases

def _log(rng, lo, hi, step):
    """A multiple of ``step`` between ``lo`` and ``hi``, uniform in its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    """One more case of the same ranges, never more work than the largest listed one."""
    kind = rng.choice(["mlp_step", "mlp_step", "mlp_forward", "moe_step", "moe_forward", "gemm", "gemm", "gemm", "sgd"])
    if kind in ("mlp_step", "mlp_forward"):
        d, f = _log(rng, 256, 8192, 256), _log(rng, 256, 28672, 128)
        t, n = _log(rng, 128, 32768, 128), rng.randint(1, 4)
        return {"kind": kind, "d_model": d, "ffn": f, "tokens": t, "layers": n}
    if kind in ("moe_step", "moe_forward"):
        h, f = _log(rng, 256, 4096, 256), _log(rng, 128, 14336, 128)
        e = rng.choice([4, 8, 16])
        t = _log(rng, 200, 16384, 1) if kind == "moe_step" else _log(rng, 16, 4096, 1)
        return {"kind": kind, "experts": e, "hidden": h, "ffn": f, "tokens": t}
    if kind == "gemm":
        a_mn, b_mn = rng.random() < 0.5, rng.random() < 0.5
        m = _log(rng, 64, 16384, 8 if a_mn else 1)
        return {"kind": kind, "m": m, "n": _log(rng, 64, 16384, 8), "k": _log(rng, 64, 16384, 8), "a_mn": a_mn,
                "b_mn": b_mn, "epilogue": rng.choice(["store", "store", "accum", "f32"])}
    return {"kind": kind, "n": _log(rng, 10_000, 250_000_000, 1), "momentum": rng.choice([0.0, 0.9]),
            "weight_decay": rng.choice([0.0, 1e-4])}


# ------------------------------------------------------------------------------- inputs and runs

def _randn(gen, *shape, dtype=torch.bfloat16, scale=1.0):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0, scale, generator=gen)


def prepare(case, seed):
    """Weights N(0, 0.02), tokens and router logits N(0, 1), all from ``seed``."""
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("mlp_step", "mlp_forward"):
        cfg = TPMLPConfig(d_model=case["d_model"], ffn=case["ffn"], layers=case["layers"], tokens=case["tokens"],
                          seed=seed % 100003)
        return {"kind": kind, "model": TPMLPStack(cfg), "x": _randn(gen, cfg.tokens, cfg.d_model)}
    if kind in ("moe_step", "moe_forward"):
        cfg = MoEConfig(experts=case["experts"], hidden=case["hidden"], ffn=case["ffn"], tokens=case["tokens"],
                        seed=seed % 100003)
        return {"kind": kind, "model": MoELayer(cfg), "x": _randn(gen, cfg.tokens, cfg.hidden),
                "logits": _randn(gen, cfg.tokens, cfg.experts, dtype=torch.float32)}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        s = {"kind": kind, "a": _randn(gen, *((k, m) if case["a_mn"] else (m, k))),
             "b": _randn(gen, *((k, n) if case["b_mn"] else (n, k)), scale=0.02),
             "kw": {"a_mn": case["a_mn"], "b_mn": case["b_mn"], "epilogue": _EPILOGUES[case["epilogue"]]}}
        s["out"] = _randn(gen, m, n) if case["epilogue"] == "accum" else None
        return s
    n = case["n"]
    return {"kind": kind, "w": _randn(gen, n, scale=0.02), "g": _randn(gen, n, scale=0.01),
            "m": _randn(gen, n, dtype=torch.float32, scale=0.01) if case["momentum"] else None,
            "hyper": {"lr": 0.1, "momentum": case["momentum"], "weight_decay": case["weight_decay"]}}


def run(state):
    kind = state["kind"]
    if kind == "mlp_step":
        model = state["model"]
        loss = model.train_step_device(state["x"])
        return {"loss": loss, "weights": [[l.w_gu, l.w_down] for l in model.layers],
                "grads": [[l.g_gu, l.g_down] for l in model.layers]}
    if kind == "mlp_forward":
        return state["model"].forward(state["x"])
    if kind == "moe_step":
        model = state["model"]
        loss = model.train_step_device(state["x"], state["logits"])
        return {"loss": loss, "out": model.out, "dx": model.dx, "dlogits": model.dlogits,
                "weights": [model.w_gu, model.w_down], "grads": [model.g_gu, model.g_down]}
    if kind == "moe_forward":
        return state["model"].forward(state["x"], state["logits"])
    if kind == "gemm":
        return gemm(state["a"], state["b"], state["out"], **state["kw"])
    h = state["hyper"]
    sgd_step(state["w"], state["g"], h["lr"], state["m"], h["momentum"], h["weight_decay"])
    return {"w": state["w"], "m": state["m"]}


# ------------------------------------------------------------------------------ work and bounds

def work(case):
    """Each input (weights among them) read once and each result written once."""
    kind = case["kind"]
    if kind in ("mlp_step", "mlp_forward"):
        d, f, t, n = case["d_model"], case["ffn"], case["tokens"], case["layers"]
        params, acts = 3 * d * f * n, t * d
        if kind == "mlp_forward":
            return {"bytes": 2.0 * (params + 2 * acts), "flops": 6.0 * t * d * f * n}
        return {"bytes": 2.0 * (3 * params + acts), "flops": 18.0 * t * d * f * n}
    if kind in ("moe_step", "moe_forward"):
        e, h, f, t = case["experts"], case["hidden"], case["ffn"], case["tokens"]
        params, acts, logits = 3 * e * h * f, t * h, t * e
        if kind == "moe_forward":
            used = 1.0 - (1.0 - 1.0 / e) ** (2 * t)  # share of the experts that some token is routed to
            return {"bytes": 2.0 * (params * used + 2 * acts) + 4.0 * logits, "flops": 12.0 * t * h * f}
        return {"bytes": 2.0 * (3 * params + 3 * acts) + 8.0 * logits, "flops": 36.0 * t * h * f}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        out = {"store": 2, "accum": 4, "f32": 4}[case["epilogue"]]
        return {"bytes": 2.0 * (m * k + n * k) + out * m * n, "flops": 2.0 * m * n * k}
    per = 14 if case["momentum"] else 6
    return {"bytes": float(per * case["n"]), "flops": 6.0 * case["n"]}


def tolerance(case):
    """About four times the error that each path shows against a float64 evaluation of it."""
    kind = case["kind"]
    if kind == "gemm":
        if case["epilogue"] == "f32":
            return {"rel": 3e-5, "max": 2e-4}   # float32 sums over up to 16384 products: 5e-6 at 5000
        return {"rel": 6e-3, "max": 2e-2}       # one rounding to bf16: 1.7e-3
    if kind == "sgd":
        return {"rel": 6e-3, "max": 2e-2}       # the same rounding of the weights; the momentum is float32
    return {"rel": 2e-2, "max": 0.2}            # chains of products rounded to bf16: 3e-3 to 1e-2


# ---------------------------------------------------------------------------- the same in 64 bits

def _swiglu_mlp(x, w_gu, w_down):
    gate, up = (x @ w_gu.t()).chunk(2, -1)
    return (torch.nn.functional.silu(gate) * up) @ w_down.t()


def _stack(x, weights):
    for w_gu, w_down in weights:
        x = x + _swiglu_mlp(x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6), w_gu, w_down)
    return x


def _experts(x, logits, w_gu, w_down):
    """Top-2 routing with the softmax of the two winners as gate weights; ``w_gu`` and ``w_down`` are per expert."""
    top, idx = logits.topk(2, -1)
    gates = top.softmax(-1)
    out = torch.zeros_like(x)
    for e in range(logits.shape[1]):
        token, slot = (idx == e).nonzero(as_tuple=True)
        if token.numel():
            y = _swiglu_mlp(x[token], w_gu[e], w_down[e])
            out = out.index_add(0, token, y * gates[token, slot].unsqueeze(1))
    return out


def exact(case, seed):
    """What :func:`run` returns, by plain torch in float64 from the inputs that :func:`prepare` makes."""
    if work(case)["flops"] > 1.5e14:  # too long on one GPU
        return None
    kind, s = case["kind"], prepare(case, seed)
    if kind == "gemm":
        a, b = s["a"].double(), s["b"].double()
        out = (a.t() if case["a_mn"] else a) @ (b if case["b_mn"] else b.t())
        return out if s["out"] is None else out + s["out"].double()
    if kind == "sgd":
        w, h = s["w"].double(), s["hyper"]
        step = s["g"].double() + h["weight_decay"] * w
        if s["m"] is None:
            return {"w": w - h["lr"] * step, "m": None}
        m = h["momentum"] * s["m"].double() + step
        return {"w": w - h["lr"] * m, "m": m}
    model, x = s["model"], s["x"].double()
    lr = model.cfg.lr
    if kind in ("mlp_step", "mlp_forward"):
        weights = [[l.w_gu.double(), l.w_down.double()] for l in model.layers]
        del s, model
        if kind == "mlp_forward":
            return _stack(x, weights)
        flat = [w.requires_grad_() for pair in weights for w in pair]
        out = _stack(x, weights)
        loss = out.pow(2).mean()
        grads = torch.autograd.grad(loss, flat)
        with torch.no_grad():
            new = [w.detach() - lr * g for w, g in zip(flat, grads)]
        pairs = lambda v: [list(v[i:i + 2]) for i in range(0, len(v), 2)]  # noqa: E731
        return {"loss": loss.detach().view(1), "weights": pairs(new), "grads": pairs(grads)}
    experts, hidden = case["experts"], case["hidden"]
    logits = s["logits"].double()
    w_gu, w_down = model.w_gu.double(), model.w_down.double()
    del s, model
    per = lambda w_gu, w_down: (w_gu.view(experts, -1, hidden), w_down.view(experts, hidden, -1))  # noqa: E731
    if kind == "moe_forward":
        return _experts(x, logits, *per(w_gu, w_down))
    wanted = [t.requires_grad_() for t in (x, logits, w_gu, w_down)]
    out = _experts(x, logits, *per(w_gu, w_down))
    loss = out.pow(2).mean()
    dx, dlogits, g_gu, g_down = torch.autograd.grad(loss, wanted)
    return {"loss": loss.detach().view(1), "out": out.detach(), "dx": dx, "dlogits": dlogits,
            "weights": [w_gu.detach() - lr * g_gu, w_down.detach() - lr * g_down], "grads": [g_gu, g_down]}

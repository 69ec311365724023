"""The work that a program using this framework has it do, as cases that can be timed and compared.

Every kind below is one entry point or one short chain of entry points of ``cme213_final_project_b200.ops``, or a
whole optimizer step of ``Trainer`` on the native engine.  A case names its kind and its sizes; ``listed`` holds the
sizes of the configurations in ``config.PRESETS`` (the single-block parity models, char-gpt, GPT-2 small and medium),
``draw`` others of the same ranges.
"""
import math

import torch

from cme213_final_project_b200 import ops

DEV = "cuda"
F32, BF16, F64 = torch.float32, torch.bfloat16, torch.float64
LN_EPS = 1e-5


def _dtype(case):
    return F32 if case["dtype"] == "fp32" else BF16


def _esize(case):
    return 4 if case["dtype"] == "fp32" else 2


# ------------------------------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the loss of a character model (65 symbols) over one char-gpt batch: the shortest call, bound by latency
        {"name": "loss-char-gpt", "kind": "loss", "rows": 16384, "vocab": 65, "dtype": "bf16"},
        # a whole training step of the smallest parity model, replayed as one graph: tens of kernels of a few us each
        {"name": "step-parity-h128", "kind": "step", "mode": "parity", "batch": 32, "seq": 64, "hidden": 128, "heads": 4,
         "layers": 1, "vocab": 65, "dtype": "bf16"},
        # a whole training step of the character GPT, the ordinary single-GPU run
        {"name": "step-char-gpt", "kind": "step", "mode": "gpt", "batch": 64, "seq": 256, "hidden": 384, "heads": 6,
         "layers": 6, "vocab": 65, "dtype": "bf16"},
        # GPT-2 small's attention layer, forward and backward: causal, standard head split
        {"name": "attn-gpt2-small", "kind": "attention", "batch": 16, "heads": 12, "seq": 1024, "head_dim": 64,
         "layout": "split", "causal": True, "dtype": "bf16"},
        # parity-h512's attention: head size 128, 64 tokens, the flat head view, not causal
        {"name": "attn-parity-h512", "kind": "attention", "batch": 32, "heads": 4, "seq": 64, "head_dim": 128,
         "layout": "flat", "causal": False, "dtype": "bf16"},
        # the same layer on fp32 storage: what the strict and the tf32 modes run
        {"name": "attn-parity-h512-fp32", "kind": "attention", "batch": 32, "heads": 4, "seq": 64, "head_dim": 128,
         "layout": "flat", "causal": False, "dtype": "fp32"},
        # the LayerNorm between two GPT-2 small blocks, residual add fused, forward and backward
        {"name": "layernorm-gpt2-small", "kind": "layernorm", "rows": 16384, "cols": 768, "dtype": "bf16"},
        # GPT-2 small's feed-forward block, forward and backward, GELU
        {"name": "mlp-gpt2-small", "kind": "mlp", "rows": 16384, "hidden": 768, "ff": 3072, "act": "gelu", "dtype": "bf16"},
        # parity-h512's feed-forward block on fp32 storage, products in tf32, ReLU and bias as kernels of their own
        {"name": "mlp-parity-h512-tf32", "kind": "mlp", "rows": 2048, "hidden": 512, "ff": 2048, "act": "relu",
         "dtype": "fp32"},
        # the tied output head and its loss, forward and backward, half a GPT-2 small batch: the largest call
        {"name": "head-gpt2-small", "kind": "head", "rows": 8192, "vocab": 50304, "hidden": 768, "dtype": "bf16"},
        # GPT-2 small's embedding tables, gather and scatter, token ids distributed like those of a text
        {"name": "embedding-gpt2-small", "kind": "embedding", "batch": 16, "seq": 1024, "vocab": 50304, "hidden": 768,
         "dtype": "bf16"},
        # the optimizer over GPT-2 small's arena: global norm, clip, AdamW, bf16 copy of the weights
        {"name": "adamw-gpt2-small", "kind": "adamw", "count": 124475904, "dtype": "bf16"},
    ]


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(["loss", "step", "attention", "attention", "layernorm", "mlp", "head", "embedding", "adamw"])
    dtype = rng.choice(["bf16", "bf16", "fp32"])
    if kind == "loss":        # characters to a few thousand sub-words, odd sizes among them
        return {"kind": kind, "rows": _log(rng, 256, 32768), "vocab": _log(rng, 16, 4096), "dtype": dtype}
    if kind == "step":        # the two model families between tiny-gpt's and char-gpt's sizes
        mode = rng.choice(["parity", "gpt"])
        if mode == "parity":
            return {"kind": kind, "mode": mode, "batch": _log(rng, 8, 64), "seq": 64, "hidden": rng.choice([128, 256, 512]),
                    "heads": 4, "layers": 1, "vocab": rng.randint(40, 128), "dtype": "bf16"}
        heads = rng.randint(2, 6)
        return {"kind": kind, "mode": mode, "batch": _log(rng, 4, 64), "seq": _log(rng, 32, 256, 8), "hidden": 64 * heads,
                "heads": heads, "layers": rng.randint(1, 6), "vocab": rng.randint(40, 512), "dtype": "bf16"}
    if kind == "attention":
        layout = rng.choice(["split", "flat"])
        causal = rng.random() < 0.5
        if dtype == "bf16" and rng.random() < 0.67:      # head size 64, any length
            seq = _log(rng, 48, 1024)
            heads = rng.randint(4, 16)
            return {"kind": kind, "batch": rng.randint(1, max(1, min(64, 192 * 1024 // (heads * seq)))), "heads": heads,
                    "seq": seq, "head_dim": 64, "layout": layout, "causal": causal, "dtype": "bf16"}
        # tiny-gpt's and the parity models' head sizes, and all of fp32 storage: short sequences
        return {"kind": kind, "batch": rng.randint(4, 32), "heads": 4, "seq": _log(rng, 32, 128), "layout": layout,
                "head_dim": rng.choice([32, 64, 128]), "causal": causal, "dtype": dtype}
    if kind == "layernorm":
        cols = _log(rng, 64, 1024, 8) if rng.random() < 0.8 else _log(rng, 64, 1024)
        return {"kind": kind, "rows": _log(rng, 256, 16384), "cols": cols, "dtype": dtype}
    if kind == "mlp":
        hidden = _log(rng, 128, 768, 8)
        return {"kind": kind, "rows": _log(rng, 256, 16384), "hidden": hidden, "ff": 4 * hidden,
                "act": rng.choice(["gelu", "relu"]), "dtype": dtype}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 512, 8192), "vocab": _log(rng, 2048, 50304, 8),
                "hidden": _log(rng, 128, 768, 64), "dtype": "bf16"}
    if kind == "embedding":
        vocab = rng.randint(65, 250) if rng.random() < 0.4 else _log(rng, 8192, 50304)      # characters or sub-words
        return {"kind": kind, "batch": rng.randint(1, 16), "seq": _log(rng, 64, 1024), "vocab": vocab,
                "hidden": _log(rng, 64, 768, 8), "dtype": dtype}
    return {"kind": "adamw", "count": _log(rng, 200000, 124475904), "dtype": dtype}


# ------------------------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------------------------
def _inputs(case, seed):
    """The tensors of a case, from the seed alone; ``prepare`` hands them to this framework, ``exact`` to plain torch."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    dt = _dtype(case)

    def rnd(*shape, scale=1.0, dtype=dt, shift=0.0):
        return (torch.randn(*shape, generator=g, device=DEV) * scale + shift).to(dtype)

    def ids(n, hi):
        return torch.randint(0, hi, (n,), generator=g, device=DEV, dtype=torch.int32)

    k = case["kind"]
    if k == "loss":
        return {"logits": rnd(case["rows"], case["vocab"], scale=2.0), "targets": ids(case["rows"], case["vocab"])}
    if k == "attention":
        n, d = case["batch"] * case["seq"], case["heads"] * case["head_dim"]
        return {"q": rnd(n, d), "k": rnd(n, d), "v": rnd(n, d), "dout": rnd(n, d)}
    if k == "layernorm":
        r, c = case["rows"], case["cols"]
        return {"x": rnd(r, c), "res": rnd(r, c, shift=0.5), "dy": rnd(r, c), "dres": rnd(r, c),
                "gamma": rnd(c, scale=0.1, shift=1.0), "beta": rnd(c, scale=0.1)}
    if k == "mlp":
        m, d, f = case["rows"], case["hidden"], case["ff"]
        return {"x": rnd(m, d), "res": rnd(m, d), "dy": rnd(m, d), "w1": rnd(d, f, scale=d ** -0.5), "b1": rnd(f, scale=0.1),
                "w2": rnd(f, d, scale=f ** -0.5), "b2": rnd(d, scale=0.1)}
    if k == "head":
        return {"x": rnd(case["rows"], case["hidden"]), "tok": rnd(case["vocab"], case["hidden"], scale=0.05),
                "targets": ids(case["rows"], case["vocab"])}
    if k == "embedding":
        n, v, d = case["batch"] * case["seq"], case["vocab"], case["hidden"]
        # frequencies of sub-words fall off like 1 / (rank + 20): the inverse of that distribution at uniform points
        u = torch.rand(n, generator=g, device=DEV)
        rank = (20 * ((1 + v / 20) ** u - 1)).long().clamp_(0, v - 1)
        name = torch.randperm(v, generator=g, device=DEV)
        return {"tokens": name[rank].to(torch.int32), "tok": rnd(v, d, scale=0.02), "pos": rnd(case["seq"], d, scale=0.02),
                "dout": rnd(n, d)}
    if k == "adamw":
        n = case["count"]
        cut = [n // 3 // 64 * 64, n // 2 // 64 * 64, n - n % 64]      # biases and norms between the weights: no decay
        return {"master": rnd(n, scale=0.02, dtype=F32), "grads": rnd(n, scale=1e-3), "m": rnd(n, scale=1e-4, dtype=F32),
                "v": rnd(n, scale=1e-3, dtype=F32).square_(),
                "nodecay": torch.tensor([[cut[0], cut[0] + 768], [cut[1], cut[1] + 3072], [cut[2] - 1536, cut[2]]],
                                        dtype=torch.int64, device=DEV)}
    n = case["batch"] * case["seq"]
    flat = torch.zeros(_arena(case)[1], device=DEV)
    for name, shape, at in _arena(case)[0]:
        size = math.prod(shape)
        gain = "gamma" in name
        flat[at:at + size] = rnd(size, scale=0.1 if gain else 0.02, dtype=F32, shift=1.0 if gain else 0.0)
    return {"tokens": ids(n, case["vocab"]), "targets": ids(n, case["vocab"]), "flat": flat}


def _arena(case):
    """The tensors of the flat parameter arena as (name, shape, offset), and its size: the order is the one in which
    backward finishes the gradients, every tensor starts at a multiple of 64 elements."""
    D, V, T = case["hidden"], case["vocab"], case["seq"]
    FF, gpt = 4 * D, case["mode"] == "gpt"
    order = [("lnf_gamma", (D,)), ("lnf_beta", (D,))] if gpt else [("Wout", (D, V))]
    for l in reversed(range(case["layers"])):
        qkv = [("Wqkv", (D, 3 * D))] if gpt else [("Wq", (D, D)), ("Wk", (D, D)), ("Wv", (D, D))]
        order += [("%d.%s" % (l, n), s) for n, s in
                  [("W2", (FF, D)), ("b2", (D,)), ("W1", (D, FF)), ("b1", (FF,)), ("ln2_gamma", (D,)), ("ln2_beta", (D,)),
                   ("Wo", (D, D))] + qkv + [("ln1_gamma", (D,)), ("ln1_beta", (D,))]]
    order += [("tok", (V, D)), ("pos", (T, D))]
    at, out = 0, []
    for name, shape in order:
        out.append((name, shape, at))
        at += -(-math.prod(shape) // 64) * 64
    return out, at


def _hyper(case):
    if case["mode"] == "gpt":
        return dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, clip_norm=0.0)
    return dict(lr=1e-4, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.0, clip_norm=1.0)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "adamw":
        s["step"] = torch.full((1,), 10, dtype=torch.int32, device=DEV)
        s["lr"] = torch.full((1,), 3e-4, device=DEV)
        s["compute"] = None if case["dtype"] == "fp32" else s["master"].to(BF16)
    elif case["kind"] == "step":
        from cme213_final_project_b200.config import ModelConfig, OptimConfig, RunConfig
        from cme213_final_project_b200.models.engine import NativeEngine
        from cme213_final_project_b200.parallel.dist import DistributedContext
        from cme213_final_project_b200.trainer import Trainer
        gpt = case["mode"] == "gpt"
        cfg = ModelConfig(mode=case["mode"], vocab_size=case["vocab"], seq_len=case["seq"], hidden=case["hidden"],
                          heads=case["heads"], ff=4 * case["hidden"], layers=case["layers"], batch_size=case["batch"],
                          activation="gelu" if gpt else "relu", causal=gpt, head_layout="split" if gpt else "flat",
                          tied_embeddings=gpt, final_layernorm=gpt, init="normal")
        optim = OptimConfig(**_hyper(case))
        run_cfg = RunConfig(cuda_graph=True, synthetic=True)
        ctx = DistributedContext().init(backend="auto", device=DEV)
        model = NativeEngine(cfg, optim, run_cfg, ctx, seed=seed)
        trainer = Trainer(model, ctx, run_cfg, optim)
        trainer.enable_cuda_graph(warmup_steps=1)
        for _ in range(2):                        # one eager step, one that captures
            trainer.step([s["tokens"]], [s["targets"]])
        flat = s.pop("flat")
        model.load_state(flat, torch.zeros_like(flat), torch.zeros_like(flat), 0)
        s["model"], s["trainer"] = model, trainer
    return s


# ------------------------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "loss":
        loss, grad, losses = ops.cross_entropy(s["logits"], s["targets"])
        return {"loss": loss, "grad": grad, "losses": losses}
    if k == "attention":
        shape = (case["batch"], case["heads"], case["seq"], case["layout"], case["causal"])
        out, lse = ops.attention_fwd(s["q"], s["k"], s["v"], *shape)
        dq, dk, dv = ops.attention_bwd(s["q"], s["k"], s["v"], out, lse, s["dout"], *shape)
        return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if k == "layernorm":
        y, mean, rstd, summed = ops.layernorm_fwd(s["x"], s["gamma"], s["beta"], LN_EPS, residual=s["res"], save_sum=True)
        dx, dgamma, dbeta = ops.layernorm_bwd(s["dy"], summed, s["gamma"], mean, rstd, dres=s["dres"])
        return {"y": y, "mean": mean, "rstd": rstd, "summed": summed, "dx": dx, "dgamma": dgamma, "dbeta": dbeta}
    if k == "mlp":
        return _run_mlp(s, case)
    if k == "head":
        logits = ops.gemm(s["x"], s["tok"], b_trans=True)
        loss, grad, losses = ops.cross_entropy(logits, s["targets"], inplace=True)
        return {"loss": loss, "losses": losses, "grad": grad, "dx": ops.gemm(grad, s["tok"]),
                "dtok": ops.gemm(grad, s["x"], a_trans=True)}
    if k == "embedding":
        out = ops.embedding_fwd(s["tokens"], s["tok"], s["pos"])
        dtok, dpos = ops.embedding_bwd(s["tokens"], s["dout"], case["vocab"], case["seq"])
        return {"out": out, "dtok": dtok, "dpos": dpos}
    if k == "adamw":
        normsq = ops.grad_normsq(s["grads"])
        ops.adam_step(s["master"], s["grads"], s["m"], s["v"], s["step"], s["lr"], compute=s["compute"], normsq=normsq,
                      beta2=0.95, weight_decay=0.1, clip_norm=1.0, nodecay=s["nodecay"])
        return {"normsq": normsq, "master": s["master"], "m": s["m"], "v": s["v"], "compute": s["compute"]}
    s["trainer"].step([s["tokens"]], [s["targets"]])
    m = s["model"]
    return {"loss": m.loss_dev, "grads": m.grads, "master": m.master, "params": m.params}


def _run_mlp(s, case):
    x, w1, w2, dy, act = s["x"], s["w1"], s["w2"], s["dy"], case["act"]
    if case["dtype"] == "bf16":               # bias, activation, derivative, residual and bias gradient in the epilogues
        gelu = act == "gelu"
        aux = torch.empty(case["rows"], case["ff"], dtype=BF16, device=DEV) if gelu else None
        a = ops.gemm(x, w1, bias=s["b1"], act=act, aux_out=aux, aux_deriv=gelu)
        y = ops.gemm(a, w2, bias=s["b2"], residual=s["res"])
        db1 = torch.empty_like(s["b1"])
        da = ops.gemm(dy, w2, b_trans=True, dact=act, aux_in=aux if gelu else a, aux_deriv=gelu, dbias=db1)
    else:                                     # fp32 storage: plain tf32 products between element-wise kernels
        a, pre = ops.bias_act_residual(ops.gemm(x, w1), s["b1"], act, save_pre=True)
        y, _ = ops.bias_act_residual(ops.gemm(a, w2), s["b2"], None, s["res"])
        da, db1 = ops.dact_colsum(ops.gemm(dy, w2, b_trans=True), pre, act)
    dw2 = ops.gemm(a, dy, a_trans=True)
    _, db2 = ops.dact_colsum(dy, want_g=False)
    return {"a": a, "y": y, "dx": ops.gemm(da, w1, b_trans=True), "dw1": ops.gemm(x, da, a_trans=True), "db1": db1,
            "dw2": dw2, "db2": db2}


# ------------------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def work(case):
    k, e = case["kind"], _esize(case)
    if k == "loss":
        return {"bytes": 2 * e * case["rows"] * case["vocab"], "flops": 0}
    if k == "attention":
        n = case["batch"] * case["seq"] * case["heads"] * case["head_dim"]
        products = 7 * 2.0 * n * case["seq"] * (0.5 if case["causal"] else 1.0)       # two forward, five backward
        return {"bytes": 8 * e * n, "flops": products}
    if k == "layernorm":
        return {"bytes": 7 * e * case["rows"] * case["cols"], "flops": 0}
    if k == "mlp":
        m, d, f = case["rows"], case["hidden"], case["ff"]
        return {"bytes": e * (5 * m * d + m * f + 4 * d * f), "flops": 12.0 * m * d * f}
    if k == "head":
        m, v, d = case["rows"], case["vocab"], case["hidden"]
        return {"bytes": e * (2 * m * d + 2 * v * d + m * v), "flops": 6.0 * m * v * d}
    if k == "embedding":
        n, v, d = case["batch"] * case["seq"], case["vocab"], case["hidden"]
        seen = min(n, v)
        return {"bytes": e * d * (2 * n + seen + v + 2 * case["seq"]), "flops": 0}
    if k == "adamw":
        return {"bytes": 28 * case["count"], "flops": 0}
    n, d, t = case["batch"] * case["seq"], case["hidden"], case["seq"]
    size = _arena(case)[1]
    dense = sum(math.prod(shape) for name, shape, _ in _arena(case)[0] if len(shape) == 2 and name != "pos"
                and (name != "tok" or case["mode"] == "gpt"))
    attention = 7 * 2.0 * n * t * d * case["layers"] * (0.5 if case["mode"] == "gpt" else 1.0)
    return {"bytes": 30 * size, "flops": 6.0 * n * dense + attention}


def tolerance(case):
    bf16 = case["dtype"] == "bf16"
    k = case["kind"]
    if k == "loss":
        return {"rel": 8e-3 if bf16 else 1e-5}
    if k == "attention":
        return {"rel": 1e-2 if bf16 else 1e-5}
    if k == "layernorm":
        return {"rel": 1e-2 if bf16 else 1e-5}
    if k == "mlp":       # ReLU: a pre-activation that rounding takes across zero switches its whole gradient on or off
        return {"rel": 3e-2 if case["act"] == "relu" else 1.2e-2 if bf16 else 4e-3}
    if k == "head":
        return {"rel": 8e-3}
    if k == "embedding":
        # a frequent id's row is a sum of over a hundred bf16 values, rounded as often, in any order
        return {"rel": 3e-2 if bf16 else 1e-5, "max": 0.9 if bf16 else 1e-3}
    if k == "adamw":
        return {"rel": 8e-3 if bf16 else 1e-5}
    return {"rel": 3e-2}        # the parity step's gradients are 2.9e-2 off their 64-bit values, for the ReLU's reason


# ------------------------------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------------------------
def _layer_norm(x, gamma, beta):
    mean = x.mean(-1, keepdim=True)
    rstd = ((x - mean).square().mean(-1, keepdim=True) + LN_EPS).rsqrt()
    return (x - mean) * rstd * gamma + beta, mean, rstd


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _act(x, act):
    return _gelu(x) if act == "gelu" else torch.relu(x)


def _heads(t, batch, heads, seq, layout):
    if layout == "flat":
        return t.reshape(batch * heads, seq, -1)
    return t.reshape(batch, seq, heads, -1).transpose(1, 2).reshape(batch * heads, seq, -1)


def _attention(q, k, v, batch, heads, seq, layout, causal):
    q, k, v = (_heads(t, batch, heads, seq, layout) for t in (q, k, v))
    sc = q @ k.transpose(1, 2) / math.sqrt(q.shape[-1])
    if causal:
        sc = sc.masked_fill(torch.ones(seq, seq, dtype=torch.bool, device=sc.device).triu(1), -math.inf)
    lse = torch.logsumexp(sc, -1)
    out = torch.exp(sc - lse[..., None]) @ v
    if layout == "split":
        out = out.reshape(batch, heads, seq, -1).transpose(1, 2)
    return out.reshape(batch * seq, -1), lse.reshape(-1)


def _loss(logits, targets, prob_eps=0.0):
    picked = logits.gather(1, targets.long()[:, None])[:, 0] - torch.logsumexp(logits, -1)
    return -torch.log(torch.exp(picked) + prob_eps) if prob_eps else -picked


def exact(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    if k == "adamw":
        return _exact_adamw(s, case)
    if k == "step":
        return _exact_step(s, case)
    d = {n: t.double() if t.is_floating_point() else t for n, t in s.items()}
    if k == "loss":
        x = d["logits"].requires_grad_(True)
        losses = _loss(x, d["targets"])
        return {"loss": losses.mean()[None].detach(), "grad": torch.autograd.grad(losses.mean(), x)[0],
                "losses": losses.detach()}
    if k == "attention":
        leaves = [d[n].requires_grad_(True) for n in ("q", "k", "v")]
        out, lse = _attention(*leaves, case["batch"], case["heads"], case["seq"], case["layout"], case["causal"])
        dq, dk, dv = torch.autograd.grad(out, leaves, d["dout"])
        return {"out": out.detach(), "lse": lse.detach(), "dq": dq, "dk": dk, "dv": dv}
    if k == "layernorm":
        summed = d["x"] + d["res"]
        leaves = [t.requires_grad_(True) for t in (summed, d["gamma"], d["beta"])]
        y, mean, rstd = _layer_norm(*leaves)
        dx, dgamma, dbeta = torch.autograd.grad(y, leaves, d["dy"])
        return {"y": y.detach(), "mean": mean.detach()[:, 0], "rstd": rstd.detach()[:, 0], "summed": summed.detach(),
                "dx": dx + d["dres"], "dgamma": dgamma, "dbeta": dbeta}
    if k == "mlp":
        leaves = [d[n].requires_grad_(True) for n in ("x", "w1", "b1", "w2", "b2")]
        x, w1, b1, w2, b2 = leaves
        a = _act(x @ w1 + b1, case["act"])
        y = a @ w2 + b2 + d["res"]
        dx, dw1, db1, dw2, db2 = torch.autograd.grad(y, leaves, d["dy"])
        return {"a": a.detach(), "y": y.detach(), "dx": dx, "dw1": dw1, "db1": db1, "dw2": dw2, "db2": db2}
    if k == "head":
        x, tok = d["x"].requires_grad_(True), d["tok"].requires_grad_(True)
        logits = x @ tok.t()
        losses = _loss(logits, d["targets"])
        grad, dx, dtok = torch.autograd.grad(losses.mean(), [logits, x, tok])
        return {"loss": losses.mean()[None].detach(), "losses": losses.detach(), "grad": grad, "dx": dx, "dtok": dtok}
    tokens = d["tokens"].long()
    out = d["tok"][tokens] + d["pos"].repeat(case["batch"], 1)
    dtok = torch.zeros_like(d["tok"]).index_add_(0, tokens, d["dout"])
    return {"out": out, "dtok": dtok, "dpos": d["dout"].reshape(case["batch"], case["seq"], -1).sum(0)}


def _adam(p, g, m, v, step, decays, o, gscale):
    g = g * gscale
    m = o["beta1"] * m + (1 - o["beta1"]) * g
    v = o["beta2"] * v + (1 - o["beta2"]) * g * g
    p = p * (1 - o["lr"] * o["weight_decay"] * decays) - o["lr"] * (m / (1 - o["beta1"] ** step)) / (
        (v / (1 - o["beta2"] ** step)).sqrt() + o["eps"])
    return p, m, v


def _exact_adamw(s, case):
    o = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)
    g = s["grads"].double()
    normsq = g.square().sum()
    decays = torch.ones(case["count"], device=DEV)
    for a, b in s["nodecay"].tolist():
        decays[a:b] = 0
    p, m, v = _adam(s["master"].double(), g, s["m"].double(), s["v"].double(), 10, decays, o,
                    min(1.0, 1.0 / float(normsq.sqrt())))
    return {"normsq": normsq[None], "master": p, "m": m, "v": v, "compute": None if case["dtype"] == "fp32" else p}


def _exact_step(s, case):
    D, H, T, B, gpt = case["hidden"], case["heads"], case["seq"], case["batch"], case["mode"] == "gpt"
    where, size = _arena(case)
    low = s["flat"].to(BF16).double()                         # products read the bf16 copy of the fp32 weights
    P = {n: low[at:at + math.prod(shape)].view(shape).requires_grad_(True) for n, shape, at in where}
    tokens = s["tokens"].long()
    x = P["tok"][tokens] + P["pos"].repeat(B, 1)
    for l in range(case["layers"]):
        p = lambda n: P["%d.%s" % (l, n)]                     # noqa: E731
        h = _layer_norm(x, p("ln1_gamma"), p("ln1_beta"))[0]
        q, k, v = (h @ p("Wqkv")).split(D, -1) if gpt else (h @ p("Wq"), h @ p("Wk"), h @ p("Wv"))
        x = x + _attention(q, k, v, B, H, T, "split" if gpt else "flat", gpt)[0] @ p("Wo")
        h = _layer_norm(x, p("ln2_gamma"), p("ln2_beta"))[0]
        x = x + _act(h @ p("W1") + p("b1"), "gelu" if gpt else "relu") @ p("W2") + p("b2")
    if gpt:
        x = _layer_norm(x, P["lnf_gamma"], P["lnf_beta"])[0]
    loss = _loss(x @ (P["tok"].t() if gpt else P["Wout"]), s["targets"], 0.0 if gpt else 1e-9).mean()
    grads = torch.zeros(size, dtype=F64, device=DEV)
    decays = torch.zeros(size, device=DEV)
    for (n, shape, at), g in zip(where, torch.autograd.grad(loss, [P[n] for n, _, _ in where])):
        grads[at:at + g.numel()] = g.reshape(-1)
        decays[at:at + g.numel()] = float(len(shape) == 2)
    o = _hyper(case)
    clip = min(1.0, o["clip_norm"] / float(grads.norm())) if o["clip_norm"] > 0 else 1.0
    zero = torch.zeros_like(grads)
    master, _, _ = _adam(s["flat"].double(), grads, zero, zero, 1, decays, o, clip)
    return {"loss": loss[None].detach(), "grads": grads, "master": master, "params": master}

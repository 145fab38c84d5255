"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of ``deers_b200``: the fused attention op (forward and backward,
f16 and f32), the attention module built from the library's operators, decode-time attention against a key / value
cache, and the GPT object (training steps, evaluation, prefix-by-prefix sampling).

  listed()         the cases by name
  draw(rng)        one more case of the same ranges
  prepare(c, seed) what a program holds before the call, on the GPU
  run(state)       one pass; returns its outputs
  work(c)          bytes and floating-point operations of one pass that the path cannot do without
  tolerance(c)     how far two correct implementations of the same precision may be apart
"""
import math

import numpy as np
import torch

from deers_b200 import gpt, ops

# Causal forward + backward work, B*H*T^2*D, of the largest listed attention case: drawn ones stay below it.
MOST_SCORES = 64 * 32 * 2048 * 2048 * 128
MOST_VALUES = 64 * 32 * 2048 * 128


def listed():
    return [
        # The attention of the README's GPT (n_embd 192, 6 heads) in one training step, f32: latency and launches.
        {"name": "train_f32_readme", "kind": "train", "dtype": "f32", "B": 4, "H": 6, "T": 256, "D": 32},
        # One layer's attention of a small f16 model with 64-wide heads, forward and backward.
        {"name": "train_f16_d64", "kind": "train", "dtype": "f16", "B": 8, "H": 12, "T": 1024, "D": 64},
        # Long context: few slices, many tiles per slice.
        {"name": "train_f16_long", "kind": "train", "dtype": "f16", "B": 2, "H": 16, "T": 8192, "D": 128},
        # The full batch of a large model on one GPU: throughput, power and memory bound.
        {"name": "train_f16_full", "kind": "train", "dtype": "f16", "B": 64, "H": 32, "T": 2048, "D": 128},
        # head_dim = n_embd / n_head is free in the reference: 640 / 8 heads, a sequence that fills no tile.
        {"name": "train_f16_d80_ragged", "kind": "train", "dtype": "f16", "B": 4, "H": 8, "T": 1000, "D": 80},
        # Reading one prompt: forward only, a handful of tiles, an odd length.
        {"name": "prefill_f16_prompt", "kind": "prefill", "dtype": "f16", "B": 1, "H": 12, "T": 333, "D": 64},
        # One new token of one sequence: the smallest call there is.
        {"name": "decode_f16_one", "kind": "decode", "dtype": "f16", "B": 1, "H": 12, "Tq": 1, "Tk": 777, "D": 64},
        # One new token for a batch of served sequences with a long cache: pure cache bandwidth.
        {"name": "decode_f16_batch", "kind": "decode", "dtype": "f16", "B": 64, "H": 32, "Tq": 1, "Tk": 2048, "D": 128},
        # The attention module around the op: fused q|k|v projection, rotary pack, attention, output projection;
        # forward and the whole backward.
        {"name": "module_f16", "kind": "module", "B": 8, "H": 12, "T": 1024, "D": 64},
        # The training loop of the README GPT: optimizer steps on fresh batches, then the evaluation forward.
        {"name": "gpt_train_readme", "kind": "gpt_train", "vocab": 50257, "layers": 6, "H": 6, "D": 32, "mlp": 768,
         "B": 4, "T": 256, "steps": 4},
        # A smaller model with a short ragged context: the launch-bound end of the same loop.
        {"name": "gpt_train_small", "kind": "gpt_train", "vocab": 5003, "layers": 3, "H": 4, "D": 48, "mlp": 500,
         "B": 3, "T": 77, "steps": 4},
        # Sampling as the reference does it: the whole prefix goes through the model again for every new token, so
        # each call has another length.
        {"name": "gpt_sample_readme", "kind": "gpt_sample", "vocab": 50257, "layers": 6, "H": 6, "D": 32, "mlp": 768,
         "B": 1, "T": 100, "tokens": 8},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["train16", "train16", "train16_odd", "train32", "prefill", "decode", "decode", "module", "gpt_train",
                       "gpt_sample"])
    if kind in ("train16", "train16_odd", "train32"):
        while True:
            if kind == "train32":
                D = rng.choice([16, 32, 48, 64, 96, 128])
                c = {"kind": "train", "dtype": "f32", "B": _log_int(rng, 1, 16), "H": rng.randint(1, 12),
                     "T": _log_int(rng, 16, 2048), "D": D}
                most = MOST_SCORES // 64
            else:
                D = rng.choice([64, 128]) if kind == "train16" else 8 * rng.choice([1, 2, 3, 4, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15])
                c = {"kind": "train", "dtype": "f16", "B": _log_int(rng, 1, 64), "H": rng.randint(1, 32),
                     "T": _log_int(rng, 32, 8192), "D": D}
                most = MOST_SCORES if kind == "train16" else MOST_SCORES // 4
            values = c["B"] * c["H"] * c["T"] * D
            if values * c["T"] <= most and values <= MOST_VALUES:
                return c
    if kind == "prefill":
        while True:
            c = {"kind": "prefill", "dtype": rng.choice(["f16", "f16", "f32"]), "B": _log_int(rng, 1, 16),
                 "H": rng.randint(1, 32), "T": _log_int(rng, 8, 8192), "D": rng.choice([32, 64, 96, 128])}
            scores = c["B"] * c["H"] * c["T"] * c["T"] * c["D"]
            if scores <= MOST_SCORES // (1 if c["dtype"] == "f16" else 64):
                return c
    if kind == "decode":
        while True:
            c = {"kind": "decode", "dtype": rng.choice(["f16", "f16", "f32"]), "B": _log_int(rng, 1, 64),
                 "H": rng.randint(1, 32), "Tq": rng.choice([1, 1, 1, 1, rng.randint(2, 8)]),
                 "Tk": _log_int(rng, 8, 32768), "D": rng.choice([32, 64, 80, 96, 128])}
            if c["B"] * c["H"] * c["Tk"] * c["D"] <= MOST_VALUES:
                return c
    if kind == "module":
        while True:
            c = {"kind": "module", "B": _log_int(rng, 1, 16), "H": rng.randint(2, 24), "T": _log_int(rng, 64, 2048),
                 "D": rng.choice([32, 64, 64, 128])}
            if c["B"] * c["T"] <= 16384 and c["H"] * c["D"] <= 2048:
                return c
    D = rng.choice([16, 32, 48, 64])
    H = rng.randint(2, max(2, min(8, 384 // D)))
    c = {"kind": kind, "vocab": _log_int(rng, 1024, 50257), "layers": rng.randint(1, 8), "H": H, "D": D,
         "mlp": rng.choice([2, 3, 4]) * H * D}
    if kind == "gpt_train":
        c.update(B=rng.randint(1, 8), T=_log_int(rng, 16, 512), steps=4)
        c["B"] = max(1, min(c["B"], 1024 // c["T"]))
    else:
        c.update(B=rng.randint(1, 2), T=_log_int(rng, 4, 248), tokens=8)
    return c


def _dtype(c):
    return torch.float16 if c.get("dtype", "f16") == "f16" else torch.float32


def _normal(g, shape, dtype, scale=1.0):
    t = torch.randn(shape, device="cuda", dtype=dtype, generator=g)
    return t if scale == 1.0 else t * scale


def _model(c, g, tokens):
    """A model with the reference's initial distributions (standard normal embedding, uniform +-1/sqrt(in) weights)."""
    C = c["H"] * c["D"]
    m = gpt.GPT(gpt.GPTConfig(c["vocab"], tokens, c["layers"], c["H"], C, c["mlp"]),
                torch.device("cuda", torch.cuda.current_device()), c["B"])
    params = []
    for name, (rows, cols) in m.named_parameters():
        if name == "wte.weight":
            params.append(torch.randn((rows, cols), device="cuda", generator=g).cpu().numpy())
        else:
            u = torch.rand((rows, cols), device="cuda", generator=g)
            params.append(((u * 2 - 1) / math.sqrt(rows)).cpu().numpy())
    m.load_parameters(params)
    return m


def prepare(case, seed):
    c = dict(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    s = {"c": c}
    if c["kind"] in ("train", "prefill"):
        shape = (c["B"], c["H"], c["T"], c["D"])
        for name in ("q", "k", "v") + (("do",) if c["kind"] == "train" else ()):
            s[name] = _normal(g, shape, _dtype(c))
    elif c["kind"] == "decode":
        # the cache is allocated for the longest sequence and used up to Tk, as a server holds it
        rows = (c["Tk"] + 127) // 64 * 64
        s["k"], s["v"] = (_normal(g, (c["B"], c["H"], rows, c["D"]), _dtype(c)) for _ in range(2))
        s["q"] = _normal(g, (c["B"], c["H"], c["Tq"], c["D"]), _dtype(c))
    elif c["kind"] == "module":
        C, T = c["H"] * c["D"], c["T"]
        s["x"], s["dy"] = (_normal(g, (c["B"], T, C), torch.float16) for _ in range(2))
        s["wqkv"] = _normal(g, (C, 3 * C), torch.float16, 1.0 / math.sqrt(C))
        s["wo"] = _normal(g, (C, C), torch.float16, 1.0 / math.sqrt(C))
        s["cos"], s["sin"] = ops.precompute_rotary_embeddings(T, c["D"], dtype=torch.float16, device="cuda")
    else:
        tokens = c["T"] + (c["tokens"] if c["kind"] == "gpt_sample" else 0)
        m = _model(c, g, tokens)
        n = c["steps"] + 1 if c["kind"] == "gpt_train" else 1
        ids = torch.randint(0, c["vocab"], (n, c["B"], tokens + 1), device="cuda", generator=g)
        if c["kind"] == "gpt_train":
            # resumed from a checkpoint: the optimizer has history, so an update is a smooth function of the gradient
            for i, (_, (rows, cols)) in enumerate(m.named_parameters()):
                mom = torch.randn((rows, cols), device="cuda", generator=g) * 1e-4
                var = (torch.rand((rows, cols), device="cuda", generator=g) + 0.5) * 1e-7
                m.load_moments(i, mom.cpu().numpy(), var.cpu().numpy())
            m.step_count = 1000
            s["targets"] = [ids[i, :, 1:].contiguous() for i in range(n)]
            s["ids"] = [ids[i, :, :-1].contiguous() for i in range(n)]
        else:
            s["ids"] = [ids[0, :, :c["T"] + i].contiguous() for i in range(c["tokens"])]
        s["model"] = m
    return s


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "train":
        op = ops.CausalAttention.new(s["q"], s["k"], s["v"])
        o = op.forward()
        grads = ops.GradientStore()
        op.backward(grads, s["do"])
        return {"o": o, "lse": op.lse, "dq": grads.get(s["q"]), "dk": grads.get(s["k"]), "dv": grads.get(s["v"])}
    if kind == "prefill":
        return ops.causal_attention(s["q"], s["k"], s["v"])
    if kind == "decode":
        return ops.attention_decode(s["q"], s["k"][:, :, :c["Tk"]], s["v"][:, :, :c["Tk"]])
    if kind == "module":
        return _module(s)
    m = s["model"]
    if kind == "gpt_train":
        said = [m.train_step(s["ids"][i], s["targets"][i], lr=5e-4, weight_decay=0.1, max_grad_norm=1.0)
                for i in range(c["steps"])]
        return {"loss": [loss for loss, _ in said], "norm": [norm for _, norm in said], "logits": m.forward(s["ids"][-1])}
    return [m.forward(ids) for ids in s["ids"]]


def _module(s):
    """CausalSelfAttention, forward and backward, on the library's operators: q, k and v are views of one fused
    projection, their gradients land in one fused buffer."""
    c = s["c"]
    B, T, H, D = c["B"], c["T"], c["H"], c["D"]
    C = H * D
    lin_qkv = ops.Linear.new(s["x"], s["wqkv"])
    qkv = lin_qkv.forward()
    q4, k4, v4 = (qkv[..., i * C:(i + 1) * C].view(B, T, H, D) for i in range(3))
    rq, rk = ops.RotaryPack.new(q4, s["cos"], s["sin"]), ops.RotaryPack.new(k4, s["cos"], s["sin"])
    qh, kh, vh = rq.forward(), rk.forward(), v4.permute(0, 2, 1, 3)
    att = ops.CausalAttention.new(qh, kh, vh, token_major_out=True)
    y_att = att.forward().permute(0, 2, 1, 3).reshape(B, T, C)
    lin_o = ops.Linear.new(y_att, s["wo"])
    y = lin_o.forward()

    grads = ops.GradientStore()
    lin_o.backward(grads, s["dy"])
    d_att = grads.get(y_att).view(B, T, H, D).permute(0, 2, 1, 3)
    dqkv = torch.empty_like(qkv)
    dq4, dk4, dv4 = (dqkv[..., i * C:(i + 1) * C].view(B, T, H, D) for i in range(3))
    dqh, dkh, _ = ops.attention_bwd(qh, kh, vh, att.o, att.lse, d_att, att.scale, True, dv_out=dv4.permute(0, 2, 1, 3))
    rq.backward(grads, dqh, dx_out=dq4)
    rk.backward(grads, dkh, dx_out=dk4)
    lin_qkv.backward(grads, dqkv)
    return {"y": y, "dx": grads.get(s["x"]), "dwqkv": grads.get(s["wqkv"]), "dwo": grads.get(s["wo"])}


def _gpt_params(c):
    """(all parameters, those of matrix products) of the model."""
    C = c["H"] * c["D"]
    products = c["layers"] * (4 * C * C + 2 * C * c["mlp"]) + C * c["vocab"]
    return products + c["vocab"] * C, products


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind in ("train", "prefill"):
        es = 2 if _dtype(c) == torch.float16 else 4
        rows = c["B"] * c["H"] * c["T"]
        scores = rows * c["T"] * c["D"]
        if kind == "train":                        # read q, k, v, dO; write O, lse, dQ, dK, dV
            return {"bytes": 8 * rows * c["D"] * es + 4 * rows, "flops": 7 * scores}
        return {"bytes": 4 * rows * c["D"] * es, "flops": 2 * scores}
    if kind == "decode":
        es = 2 if _dtype(c) == torch.float16 else 4
        slices = c["B"] * c["H"]
        return {"bytes": slices * (2 * c["Tk"] + 2 * c["Tq"]) * c["D"] * es, "flops": 4 * slices * c["Tq"] * c["Tk"] * c["D"]}
    C = c["H"] * c["D"]
    if kind == "module":                           # read x, dy, the weights; write y, dx and the weight gradients
        n = c["B"] * c["T"]
        return {"bytes": 2 * (4 * n * C + 8 * C * C), "flops": 6 * n * 4 * C * C + 7 * n * c["T"] * C}
    every, products = _gpt_params(c)
    if kind == "gpt_train":                        # a step reads and writes weights and both moments
        n = c["B"] * c["T"]
        step = 6 * n * products + 7 * c["layers"] * n * c["T"] * C
        evaluation = 2 * n * products + 2 * c["layers"] * n * c["T"] * C
        return {"bytes": c["steps"] * 24 * every + 4 * products + 4 * n * c["vocab"], "flops": c["steps"] * step + evaluation}
    lengths = [c["T"] + i for i in range(c["tokens"])]
    return {"bytes": sum(4 * products + 4 * c["B"] * t * c["vocab"] for t in lengths),
            "flops": sum(2 * c["B"] * t * products + 2 * c["layers"] * c["B"] * t * t * C for t in lengths)}


def tolerance(case):
    c = dict(case)
    if c["kind"] in ("train", "prefill", "decode"):
        # f16: operands, probabilities and results carry 2^-11 each; f32: sums of up to T terms
        return {"rel": 2e-3} if _dtype(c) == torch.float16 else {"rel": 1e-5}
    if c["kind"] == "module":
        return {"rel": 4e-3}                       # a chain of f16 results, each rounded to 2^-11
    return {"rel": 3e-5}                           # f32 sums through every layer, and for training through four updates

"""Performance cases: the calls a training or inference program makes, at the sizes it makes them.

Sizes come from the configurations this repository ships (GPT-2 small and Llama-3-8B layers, the headline
training step, the convolution of the kernel benchmark) and from the ranges around them. ``listed()`` names
the fixed ones, ``draw(rng)`` gives further ones of the same ranges, odd sizes included.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
import torch.utils.checkpoint

from momijo_b200 import ops
from momijo_b200.models.gpt2 import GPT2, GPT2Config
from momijo_b200.models.llama import LlamaBlock, LlamaConfig
from momijo_b200.ops.conv import conv2d
from momijo_b200.parallel import AdamWConfig, ShardedDataParallel
from momijo_b200.parallel.tp import TPContext

BF16 = torch.bfloat16
EPS = 1e-5
ADAM = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)


def listed():
    return [
        # one projection of a handful of rows without gradients: the smallest call an inference loop makes
        {"name": "linear_few_rows", "kind": "linear", "rows": 8, "k": 768, "n": 2304, "grad": False},
        # GPT-2 small's MLP over a micro-batch of 16 x 1024 tokens, forward and backward
        {"name": "mlp_gpt2", "kind": "mlp", "rows": 16384, "d": 768, "ff": 3072},
        # GPT-2 small's attention over the same micro-batch: 64-wide heads, causal, forward and backward
        {"name": "attn_gpt2", "kind": "attn", "b": 16, "t": 1024, "hq": 12, "hkv": 12, "d": 64, "causal": True,
         "rope": False, "grad": True},
        # Llama-3-8B's attention: grouped heads, 128 wide, rotary positions, forward and backward
        {"name": "attn_llama", "kind": "attn", "b": 2, "t": 4096, "hq": 32, "hkv": 8, "d": 128, "causal": True,
         "rope": True, "grad": True},
        # an encoder's attention over sequences of an odd length: no mask, no gradients
        {"name": "attn_ragged", "kind": "attn", "b": 6, "t": 1777, "hq": 16, "hkv": 16, "d": 128, "causal": False,
         "rope": False, "grad": False},
        # one Llama-3-8B decoder block over 4096 tokens, forward and backward: the large products
        {"name": "block_llama8b", "kind": "block", "b": 1, "t": 4096, "hq": 32, "hkv": 8, "d": 128, "ff": 14336},
        # GPT-2 small's LayerNorm fused with the residual add, forward and backward
        {"name": "norm_gpt2", "kind": "norm", "rows": 16384, "c": 768, "rms": False},
        # GPT-2 small's tied head with its cross-entropy, forward and backward
        {"name": "head_gpt2", "kind": "head", "rows": 16384, "d": 768, "v": 50257},
        # the update of GPT-2 small's parameters: global gradient norm, clipping factor, AdamW
        {"name": "update_gpt2", "kind": "update", "n": 124439808, "g32": False},
        # a convolution layer of an image classifier in fp32, forward and backward
        {"name": "conv_f32", "kind": "conv", "n": 32, "c": 64, "hw": 56, "oc": 64, "k": 3, "stride": 1, "f32": True},
        # logits of one short prompt through all of GPT-2 small: latency and launches count
        {"name": "logits_gpt2", "kind": "logits", "b": 1, "t": 113, "layers": 12, "heads": 12, "v": 50257},
        # the headline: one optimisation step of GPT-2 small at micro-batch 16 x 1024
        {"name": "train_gpt2", "kind": "train", "b": 16, "t": 1024, "layers": 12, "heads": 12, "v": 50257},
    ]


def _log(rng, lo, hi, mult=1):
    """A whole multiple of ``mult`` spread over the logarithm of [lo, hi]."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // mult, max(-(-lo // mult), round(v / mult))) * mult


def draw(rng):
    kind = rng.choice(["linear", "mlp", "attn", "attn", "block", "norm", "head", "update", "conv", "logits", "train"])
    if kind == "linear":
        return {"kind": kind, "rows": _log(rng, 1, 20000), "k": _log(rng, 64, 4096, 8), "n": _log(rng, 64, 8192, 8),
                "grad": rng.random() < 0.6}
    if kind == "mlp":
        d = _log(rng, 128, 2048, 64)
        return {"kind": kind, "rows": _log(rng, 100, 16384), "d": d, "ff": 4 * d}
    if kind == "attn":
        d = rng.choice([64, 128])
        hkv = rng.choice([1, 2, 4, 8])
        hq = hkv * rng.choice([1, 2, 4])
        t = _log(rng, 50, 4096)
        return {"kind": kind, "b": _log(rng, 1, max(1, 32768 // t)), "t": t, "hq": hq, "hkv": hkv, "d": d,
                "causal": rng.random() < 0.7, "rope": rng.random() < 0.5, "grad": rng.random() < 0.6}
    if kind == "block":
        d = rng.choice([64, 128])
        hkv = rng.choice([2, 4, 8])
        return {"kind": kind, "b": rng.choice([1, 2, 3]), "t": _log(rng, 128, 1365), "hq": hkv * rng.choice([1, 2, 4]),
                "hkv": hkv, "d": d, "ff": _log(rng, 512, 14336, 64)}
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 64, 40000), "c": _log(rng, 256, 4096, 8), "rms": rng.random() < 0.5}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 256, 16384), "d": _log(rng, 256, 1024, 8), "v": _log(rng, 1000, 50257)}
    if kind == "update":
        return {"kind": kind, "n": _log(rng, 100000, 124439808), "g32": rng.random() < 0.3}
    if kind == "conv":
        return {"kind": kind, "n": _log(rng, 4, 32), "c": rng.choice([3, 16, 24, 32, 64]), "hw": rng.randint(20, 56),
                "oc": rng.choice([16, 32, 48, 64]), "k": rng.choice([1, 3, 5]), "stride": rng.choice([1, 1, 2]),
                "f32": rng.random() < 0.6}
    if kind == "logits":
        t = _log(rng, 16, 512)
        return {"kind": kind, "b": _log(rng, 1, max(1, 1024 // t)), "t": t, "layers": rng.choice([4, 8, 12]),
                "heads": rng.choice([6, 8, 12]), "v": _log(rng, 1000, 50257)}
    t = _log(rng, 64, 1024)
    return {"kind": kind, "b": _log(rng, 1, 16384 // t), "t": t, "layers": rng.choice([2, 4, 6]),
            "heads": rng.choice([4, 6, 8, 12]), "v": _log(rng, 1000, 50257)}


# ---- inputs ---------------------------------------------------------------------------------------------------
class _Rand:
    """Seeded normal tensors on the device that the case runs on."""

    def __init__(self, seed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.g = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return (torch.randn(*shape, generator=self.g, device=self.dev) * std + mean).to(dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device=self.dev)


def _inputs(case, seed):
    """The tensors of a case, by name, from the seed alone."""
    r, k = _Rand(seed), case["kind"]
    if k == "linear":
        m, kk, n = case["rows"], case["k"], case["n"]
        return {"x": r.normal(m, kk), "w": r.normal(n, kk, std=kk ** -0.5), "b": r.normal(n, std=0.1),
                "dy": r.normal(m, n)}
    if k == "mlp":
        m, d, f = case["rows"], case["d"], case["ff"]
        return {"x": r.normal(m, d), "w1": r.normal(f, d, std=d ** -0.5), "b1": r.normal(f, std=0.1),
                "w2": r.normal(d, f, std=f ** -0.5), "b2": r.normal(d, std=0.1), "dy": r.normal(m, d)}
    if k == "attn":
        rows, cols = case["b"] * case["t"], (case["hq"] + 2 * case["hkv"]) * case["d"]
        return {"qkv": r.normal(rows, cols), "dout": r.normal(rows, case["hq"] * case["d"])}
    if k == "block":
        c, dq = case["hq"] * case["d"], (case["hq"] + 2 * case["hkv"]) * case["d"]
        m, f = case["b"] * case["t"], case["ff"]
        return {"res": r.normal(m, c), "attn_norm": r.normal(c, std=0.1, mean=1.0),
                "mlp_norm": r.normal(c, std=0.1, mean=1.0), "wqkv": r.normal(dq, c, std=c ** -0.5),
                "wo": r.normal(c, c, std=c ** -0.5), "w_gu": r.normal(2 * f, c, std=c ** -0.5),
                "w_down": r.normal(c, f, std=f ** -0.5), "ddelta": r.normal(m, c), "dres": r.normal(m, c)}
    if k == "norm":
        m, c = case["rows"], case["c"]
        return {"x": r.normal(m, c), "res": r.normal(m, c), "g": r.normal(c, std=0.1, mean=1.0),
                "b": r.normal(c, std=0.1), "dy": r.normal(m, c), "dres": r.normal(m, c)}
    if k == "head":
        vp = ops.pad_vocab(case["v"])
        return {"x": r.normal(case["rows"], case["d"]), "wte": r.normal(vp, case["d"], std=0.05),
                "targets": r.ints(case["v"], case["rows"])}
    if k == "update":
        n = case["n"]
        return {"grad": r.normal(n, std=1e-3, dtype=torch.float32 if case["g32"] else BF16),
                "master": r.normal(n, std=0.02, dtype=torch.float32), "m": r.normal(n, std=1e-4, dtype=torch.float32),
                "v": r.normal(n, std=1e-3, dtype=torch.float32).square_()}
    if k == "conv":
        dt = torch.float32 if case["f32"] else BF16
        c, oc, ks = case["c"], case["oc"], case["k"]
        x = r.normal(case["n"], c, case["hw"], case["hw"], dtype=dt)
        o = (case["hw"] + 2 * (ks // 2) - ks) // case["stride"] + 1
        return {"x": x, "w": r.normal(oc, c, ks, ks, std=(c * ks * ks) ** -0.5, dtype=dt),
                "b": r.normal(oc, std=0.1, dtype=dt), "dy": r.normal(case["n"], oc, o, o, dtype=dt)}
    b, t = case["b"], case["t"]
    return {"tokens": r.ints(case["v"], b, t), "targets": r.ints(case["v"], b, t), "weights": _gpt2_weights(case, r)}


def _gpt2_config(case):
    c = case["heads"] * 64
    return GPT2Config(vocab_size=case["v"], n_layer=case["layers"], n_head=case["heads"], d_model=c, d_ff=4 * c)


def _gpt2_weights(case, r):
    """Parameters in the order the model declares them: wte, wpe, the final norm, then twelve of each block."""
    c, f, vp = case["heads"] * 64, case["heads"] * 256, ops.pad_vocab(case["v"])
    std2 = 0.02 / math.sqrt(2 * case["layers"])
    gain = lambda: r.normal(c, std=0.1, mean=1.0)
    bias = lambda n: r.normal(n, std=0.02)
    out = {"wte": r.normal(vp, c, std=0.02), "wpe": r.normal(1024, c, std=0.02), "lnf_g": gain(), "lnf_b": bias(c)}
    for i in range(case["layers"]):
        out.update({f"blocks.{i}.ln1_g": gain(), f"blocks.{i}.ln1_b": bias(c),
                    f"blocks.{i}.w_qkv": r.normal(3 * c, c, std=0.02), f"blocks.{i}.b_qkv": bias(3 * c),
                    f"blocks.{i}.w_o": r.normal(c, c, std=std2), f"blocks.{i}.b_o": bias(c),
                    f"blocks.{i}.ln2_g": gain(), f"blocks.{i}.ln2_b": bias(c),
                    f"blocks.{i}.w_fc": r.normal(f, c, std=0.02), f"blocks.{i}.b_fc": bias(f),
                    f"blocks.{i}.w_proj": r.normal(c, f, std=std2), f"blocks.{i}.b_proj": bias(c)})
    return out


def prepare(case, seed):
    t = _inputs(case, seed)
    k, dev = case["kind"], "cuda"
    s = {"case": case}
    if k in ("logits", "train"):
        with torch.device(dev):
            model = GPT2(_gpt2_config(case))
        with torch.no_grad():
            for name, p in model.named_parameters():
                p.copy_(t["weights"][name])
        if k == "train":
            s["engine"] = ShardedDataParallel(model, AdamWConfig(lr=ADAM["lr"], betas=(0.9, 0.95), weight_decay=0.1))
        s.update(model=model, tokens=t["tokens"], targets=t["targets"])
        return s
    if k == "block":
        cfg = LlamaConfig(n_layer=1, d_model=case["hq"] * case["d"], n_head=case["hq"], n_kv_head=case["hkv"],
                          head_dim=case["d"], d_ff=case["ff"])
        with torch.device(dev):
            blk = LlamaBlock(cfg, TPContext())
        pairs = [("attn_norm", blk.attn_norm), ("mlp_norm", blk.mlp_norm), ("wqkv", blk.wqkv.weight),
                 ("wo", blk.wo.weight), ("w_gu", blk.w_gu.weight), ("w_down", blk.w_down.weight)]
        with torch.no_grad():
            for name, p in pairs:
                p.copy_(t[name])
        s.update(block=blk, res=t["res"].requires_grad_(), ddelta=t["ddelta"], dres=t["dres"])
        s["leaves"] = [s["res"]] + [p for _, p in pairs]
        return s
    if k == "update":
        t["param"] = t["master"].to(BF16)
    elif k == "attn" and case["rope"]:
        s["table"] = ops.rope_table(case["t"], case["d"], 500000.0, torch.device(dev))
    if case.get("grad", True) and k != "update":
        for name in ("x", "res", "w", "b", "w1", "b1", "w2", "b2", "g", "qkv", "wte"):
            if name in t and not (name == "b" and k == "norm" and case["rms"]):
                t[name].requires_grad_()
    s.update(t)
    return s


# ---- one pass -------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    grad = torch.autograd.grad
    if k == "linear":
        if not case["grad"]:
            with torch.no_grad():
                return ops.linear(s["x"], s["w"], s["b"])
        y = ops.linear(s["x"], s["w"], s["b"])
        return [y, *grad(y, [s["x"], s["w"], s["b"]], s["dy"])]
    if k == "mlp":
        y = ops.mlp_gelu(s["x"], s["w1"], s["b1"], s["w2"], s["b2"])
        return [y, *grad(y, [s["x"], s["w1"], s["b1"], s["w2"], s["b2"]], s["dy"])]
    if k == "attn":
        def attend():
            return ops.attention_packed(s["qkv"], case["b"], case["t"], case["hq"], case["hkv"], case["d"],
                                        causal=case["causal"], rope=s.get("table"))
        if not case["grad"]:
            with torch.no_grad():
                return attend()
        y = attend()
        return [y, *grad(y, [s["qkv"]], s["dout"])]
    if k == "block":
        delta, res = s["block"](None, s["res"], case["b"], case["t"])
        return [delta, res, *grad([delta, res], s["leaves"], [s["ddelta"], s["dres"]])]
    if k == "norm":
        if case["rms"]:
            y, r = ops.rms_norm(s["x"], s["g"], EPS, residual=s["res"])
            return [y, r, *grad([y, r], [s["x"], s["res"], s["g"]], [s["dy"], s["dres"]])]
        y, r = ops.layer_norm(s["x"], s["g"], s["b"], EPS, residual=s["res"])
        return [y, r, *grad([y, r], [s["x"], s["res"], s["g"], s["b"]], [s["dy"], s["dres"]])]
    if k == "head":
        loss = ops.lm_head_cross_entropy(s["x"], s["wte"], s["targets"], case["v"])
        return [loss, *grad(loss, [s["x"], s["wte"]])]
    if k == "update":
        sq = ops.sq_norm(s["grad"])
        factor = torch.clamp(1.0 / (sq.sqrt() + 1e-6), max=1.0)
        ops.adamw_flat(s["grad"], s["master"], s["m"], s["v"], s["param"], step=10, grad_scale_dev=factor, **ADAM)
        return [sq, s["param"], s["master"], s["m"], s["v"]]
    if k == "conv":
        y = conv2d(s["x"], s["w"], s["b"], stride=case["stride"], pad=case["k"] // 2)
        return [y, *grad(y, [s["x"], s["w"], s["b"]], s["dy"])]
    if k == "logits":
        with torch.no_grad():
            return s["model"].logits(s["tokens"])
    loss = s["engine"](s["tokens"], s["targets"])
    loss.backward()
    s["engine"].step()
    return [loss, s["engine"].flat.grad, s["engine"].flat.param]


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _attn_flops(b, t, hq, d, causal):
    return 4.0 * b * hq * t * t * d * (0.5 if causal else 1.0)


def _gpt2_work(case):
    c, m, n_l = case["heads"] * 64, case["b"] * case["t"], case["layers"]
    vp = ops.pad_vocab(case["v"])
    params = vp * c + 1024 * c + n_l * (12 * c * c + 13 * c) + 2 * c
    flops = 2.0 * m * (12 * c * c * n_l + c * vp) + n_l * _attn_flops(case["b"], case["t"], case["heads"], 64, True)
    return params, m, flops


def work(case):
    k = case["kind"]
    if k == "linear":
        m, kk, n = case["rows"], case["k"], case["n"]
        one = 2.0 * (m * kk + n * kk + n + m * n)
        return {"bytes": 2 * one if case["grad"] else one, "flops": (6.0 if case["grad"] else 2.0) * m * n * kk}
    if k == "mlp":
        m, d, f = case["rows"], case["d"], case["ff"]
        return {"bytes": 2.0 * (4 * m * d + 4 * d * f + 2 * (d + f)), "flops": 12.0 * m * d * f}
    if k == "attn":
        m, cols, o = case["b"] * case["t"], (case["hq"] + 2 * case["hkv"]) * case["d"], case["hq"] * case["d"]
        fl = _attn_flops(case["b"], case["t"], case["hq"], case["d"], case["causal"])
        if case["grad"]:
            return {"bytes": 4.0 * m * (cols + o), "flops": 3.5 * fl}
        return {"bytes": 2.0 * m * (cols + o), "flops": fl}
    if k == "block":
        m, c, dq, f = case["b"] * case["t"], case["hq"] * case["d"], (case["hq"] + 2 * case["hkv"]) * case["d"], case["ff"]
        weights = c * dq + c * c + 3 * c * f
        return {"bytes": 2.0 * (2 * weights + 6 * m * c),
                "flops": 6.0 * m * weights + 3.5 * _attn_flops(case["b"], case["t"], case["hq"], case["d"], True)}
    if k == "norm":
        return {"bytes": 2.0 * 7 * case["rows"] * case["c"], "flops": 0.0}
    if k == "head":
        m, d, vp = case["rows"], case["d"], ops.pad_vocab(case["v"])
        return {"bytes": 4.0 * (m * d + vp * d) + 8.0 * m, "flops": 6.0 * m * d * vp}
    if k == "update":
        return {"bytes": case["n"] * ((4 if case["g32"] else 2) + 24.0 + 2.0), "flops": 0.0}
    if k == "conv":
        n, c, hw, oc, ks = case["n"], case["c"], case["hw"], case["oc"], case["k"]
        o = (hw + 2 * (ks // 2) - ks) // case["stride"] + 1
        e = 4 if case["f32"] else 2
        return {"bytes": e * (2.0 * n * c * hw * hw + 2.0 * n * oc * o * o + 2.0 * oc * (c * ks * ks + 1)),
                "flops": 6.0 * n * oc * o * o * c * ks * ks}
    params, m, flops = _gpt2_work(case)
    if k == "logits":
        return {"bytes": 2.0 * params + 2.0 * m * case["v"], "flops": flops}
    # fp32 master weights and moments read and written, bf16 parameters and gradients written
    return {"bytes": params * 30.0, "flops": 3.0 * flops}


def tolerance(case):
    """About four times what a pass at the present precision shows against 64 bits."""
    k = case["kind"]
    if k == "update":
        return {"rel": 7e-3, "max": 0.03}       # the bf16 parameters' rounding; the fp32 state is far closer
    if k == "conv":
        return {"rel": 1e-5 if case["f32"] else 1.2e-2, "max": 1e-3 if case["f32"] else 0.4}
    if k in ("block", "train"):
        return {"rel": 0.03, "max": 0.9}        # several layers of bf16 activations and gradients in a row
    if k == "logits":
        return {"rel": 0.03, "max": 0.9}        # twelve layers of bf16 activations; 0.009 seen
    return {"rel": 1.2e-2, "max": 0.4}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------
def _attn64(qkv, case, table):
    """Attention of packed rows in 64 bits, one (sequence, key head) at a time so that scores stay small."""
    b, t, hq, hkv, d = case["b"], case["t"], case["hq"], case["hkv"], case["d"]
    x = qkv.view(b, t, hq + 2 * hkv, d)
    if table is not None:
        c, s = table[..., 0].double()[:, None], table[..., 1].double()[:, None]
        lo, hi = x[:, :, :hq + hkv, :d // 2], x[:, :, :hq + hkv, d // 2:]
        x = torch.cat([torch.cat([lo * c - hi * s, hi * c + lo * s], -1), x[:, :, hq + hkv:]], 2)
    mask = torch.ones(t, t, dtype=torch.bool, device=qkv.device).tril() if case.get("causal", True) else None
    g, seqs = hq // hkv, []

    def head(q, kk, v):
        sc = q @ kk.t() / math.sqrt(d)
        if mask is not None:
            sc = sc.masked_fill(~mask, -math.inf)
        return torch.softmax(sc, -1) @ v

    for i in range(b):
        heads = []
        for h in range(hq):
            args = (x[i, :, h], x[i, :, hq + h // g], x[i, :, hq + hkv + h // g])
            heads.append(torch.utils.checkpoint.checkpoint(head, *args, use_reentrant=False))
        seqs.append(torch.stack(heads, 1))
    return torch.stack(seqs).reshape(b * t, hq * d)


def _rope64(t, d, dev):
    inv = 500000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device=dev) / d)
    a = torch.arange(t, dtype=torch.float64, device=dev)[:, None] * inv
    return torch.stack([a.cos(), a.sin()], -1).float()


def _gpt2_hidden64(p, tokens, case):
    b, t = tokens.shape
    c = case["heads"] * 64
    shape = {"b": b, "t": t, "hq": case["heads"], "hkv": case["heads"], "d": 64}
    x = (p["wte"][tokens] + p["wpe"][:t]).reshape(b * t, c)
    for i in range(case["layers"]):
        q = lambda n: p[f"blocks.{i}.{n}"]
        h = F.layer_norm(x, (c,), q("ln1_g"), q("ln1_b"), EPS)
        x = x + F.linear(_attn64(F.linear(h, q("w_qkv"), q("b_qkv")), shape, None), q("w_o"), q("b_o"))
        h = F.layer_norm(x, (c,), q("ln2_g"), q("ln2_b"), EPS)
        x = x + F.linear(F.gelu(F.linear(h, q("w_fc"), q("b_fc")), approximate="tanh"), q("w_proj"), q("b_proj"))
    return F.layer_norm(x, (c,), p["lnf_g"], p["lnf_b"], EPS)


def _flat(tensors, align=128):
    """One buffer of all parameters, each padded with zeros to a multiple of 128 elements."""
    return torch.cat([F.pad(v.reshape(-1), (0, -v.numel() % align)) for v in tensors])


def _train64(case, t):
    order = list(t["weights"])
    p = {n: w.double().requires_grad_() for n, w in t["weights"].items()}
    total = 0.0
    for i in range(case["b"]):   # one sequence at a time: the graph of a whole micro-batch would not fit
        h = _gpt2_hidden64(p, t["tokens"][i:i + 1], case)
        loss = F.cross_entropy((h @ p["wte"].t())[:, :case["v"]], t["targets"][i]) / case["b"]
        loss.backward()
        total += float(loss.detach())
    grads, new = [], []
    for n in order:
        w, g = p[n].detach(), p[n].grad if p[n].grad is not None else torch.zeros_like(p[n])
        step = g / (g.abs() + ADAM["eps"])          # first step: both moments are the gradient's own
        grads.append(g)
        new.append(w - ADAM["lr"] * (step + ADAM["weight_decay"] * w))
    return [torch.tensor(total, dtype=torch.float64), _flat(grads), _flat(new)]


def exact(case, seed):
    t = _inputs(case, seed)
    k = case["kind"]
    if k == "train":
        if _gpt2_work(case)[2] * 6 > 1.2e14:
            return None
        return _train64(case, t)
    if k == "logits":
        p = {n: w.double() for n, w in t["weights"].items()}
        with torch.no_grad():
            return (_gpt2_hidden64(p, t["tokens"], case) @ p["wte"].t())[:, :case["v"]].view(case["b"], case["t"], -1)
    if k == "update":
        g, w, m, v = (t[n].double() for n in ("grad", "master", "m", "v"))
        sq = g.square().sum().reshape(1)
        g = g * torch.clamp(1.0 / (sq.sqrt() + 1e-6), max=1.0)
        m = ADAM["beta1"] * m + (1 - ADAM["beta1"]) * g
        v = ADAM["beta2"] * v + (1 - ADAM["beta2"]) * g * g
        up = (m / (1 - ADAM["beta1"] ** 10)) / ((v / (1 - ADAM["beta2"] ** 10)).sqrt() + ADAM["eps"])
        w = w - ADAM["lr"] * (up + ADAM["weight_decay"] * w)
        return [sq, w, w, m, v]
    d = {n: v.double() if v.is_floating_point() else v for n, v in t.items()}
    leaf = lambda *names: [d[n].requires_grad_() for n in names]
    grad = torch.autograd.grad
    if k == "linear":
        if not case["grad"]:
            return F.linear(d["x"], d["w"], d["b"])
        ls = leaf("x", "w", "b")
        y = F.linear(*ls)
        return [y, *grad(y, ls, d["dy"])]
    if k == "mlp":
        ls = leaf("x", "w1", "b1", "w2", "b2")
        y = F.linear(F.gelu(F.linear(d["x"], d["w1"], d["b1"]), approximate="tanh"), d["w2"], d["b2"])
        return [y, *grad(y, ls, d["dy"])]
    if k == "attn":
        table = _rope64(case["t"], case["d"], d["qkv"].device) if case["rope"] else None
        if not case["grad"]:
            with torch.no_grad():
                return _attn64(d["qkv"], case, table)
        ls = leaf("qkv")
        y = _attn64(d["qkv"], case, table)
        return [y, *grad(y, ls, d["dout"])]
    if k == "block":
        ls = leaf("res", "attn_norm", "mlp_norm", "wqkv", "wo", "w_gu", "w_down")
        rms = lambda x, g: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * g
        qkv = rms(d["res"], d["attn_norm"]) @ d["wqkv"].t()
        res = d["res"] + _attn64(qkv, case, _rope64(case["t"], case["d"], qkv.device)) @ d["wo"].t()
        gate, up = (rms(res, d["mlp_norm"]) @ d["w_gu"].t()).chunk(2, -1)
        delta = (F.silu(gate) * up) @ d["w_down"].t()
        return [delta, res, *grad([delta, res], ls, [d["ddelta"], d["dres"]])]
    if k == "norm":
        names = ("x", "res", "g") if case["rms"] else ("x", "res", "g", "b")
        ls = leaf(*names)
        r = d["x"] + d["res"]
        if case["rms"]:
            y = r * torch.rsqrt(r.square().mean(-1, keepdim=True) + EPS) * d["g"]
        else:
            y = F.layer_norm(r, (case["c"],), d["g"], d["b"], EPS)
        return [y, r, *grad([y, r], ls, [d["dy"], d["dres"]])]
    if k == "head":
        ls = leaf("x", "wte")
        loss = F.cross_entropy((d["x"] @ d["wte"].t())[:, :case["v"]], d["targets"])
        return [loss, *grad(loss, ls)]
    # convolution: patches and a product, which 64-bit arithmetic runs as one large contraction
    ls = leaf("x", "w", "b")
    n, oc, ks = case["n"], case["oc"], case["k"]
    cols = F.unfold(d["x"], ks, padding=ks // 2, stride=case["stride"])
    o = (case["hw"] + 2 * (ks // 2) - ks) // case["stride"] + 1
    y = (d["w"].view(oc, -1) @ cols + d["b"][:, None]).view(n, oc, o, o)
    return [y, *grad(y, ls, d["dy"])]

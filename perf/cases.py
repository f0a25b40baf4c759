"""Performance cases of the framework: what a program that uses it has it do, through its public entry points.

Each case is a dict of plain values; ``kind`` selects the path.  ``listed()`` names one representative of each use,
``draw(rng)`` gives another size of the same ranges, ``prepare`` builds what a program holds before the call, ``run`` is
one pass, ``work`` its unavoidable bytes and operations, ``tolerance`` how far another correct implementation of the
same precision may be, ``exact`` what the pass gives in 64 bits.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

import spiraltorch_b200 as st
from spiraltorch_b200 import vision
from spiraltorch_b200.models.contrastive import ContrastiveEncoder, contrastive_step
from spiraltorch_b200.models.conv_classifier import STAGES, ConvClassifier
from spiraltorch_b200.models.gpt import GPTConfig, GPTModel
from spiraltorch_b200.nn import functional as fn
from spiraltorch_b200.ops import rank, spectral
from spiraltorch_b200.optim.flat import FlatAdamW, FlatSGD
from spiraltorch_b200.training import LMTrainer

DEV = "cuda"


def listed():
    return [
        # the 1.3B language model of the headline benchmark: one optimizer step from host token ids, a micro-batch of 8
        # sequences of 2048
        {"name": "lm_train_1p3b", "kind": "lm_train", "d": 2048, "layers": 24, "heads": 16, "ffn": 8192, "vocab": 50304,
         "seq": 2048, "batch": 8, "micro": 8, "norm": "rms", "pos": "rope"},
        # the byte-level language model of the data-parallel benchmark: 32 sequences of 512, learned positions, LayerNorm
        {"name": "lm_train_bytes", "kind": "lm_train", "d": 768, "layers": 12, "heads": 12, "ffn": 3072, "vocab": 256,
         "seq": 512, "batch": 32, "micro": 32, "norm": "layer", "pos": "learned"},
        # scoring one prompt of an ordinary (odd) length with the 1.3B model: logits of every position
        {"name": "lm_logits_prompt", "kind": "lm_logits", "d": 2048, "layers": 24, "heads": 16, "ffn": 8192,
         "vocab": 50304, "seq": 777, "batch": 1},
        # the conv-pool image classifier of the data-parallel benchmark: one SGD step on 256 images of 64 x 64
        {"name": "conv_train", "kind": "conv_train", "batch": 256, "image": 64, "classes": 100},
        # classifying a small batch with it
        {"name": "conv_logits", "kind": "conv_logits", "batch": 24, "image": 64, "classes": 100},
        # self-supervised encoder of the contrastive benchmark: loss and gradients of two views of 1024 vectors
        {"name": "contrastive_train", "kind": "contrastive", "batch": 1024, "in": 512, "hidden": 2048, "out": 256},
        # attention of the layer API with per-key bias and valid lengths (a padded batch), forward and backward, fp32 tensors
        {"name": "attention_padded", "kind": "attention", "contexts": 96, "seq": 1000, "dim": 64, "causal": False,
         "z_bias": True, "lengths": True},
        # a small perceptron trained through SpiralSession / ModuleTrainer: one epoch of four batches of 256
        {"name": "mlp_epoch", "kind": "mlp", "batch": 256, "batches": 4, "in": 64, "hidden": 128, "out": 8},
        # one training step of the recurrent mixer (WaveRnn + Linear) of the layer benchmark, the layer protocol called directly
        {"name": "wave_rnn_step", "kind": "rnn", "cell": "wave", "batch": 32, "steps": 16, "in": 32, "hidden": 64,
         "out": 8},
        # a batch of complex spectra, forward and inverse transform
        {"name": "fft_rows", "kind": "fft", "rows": 8192, "n": 4096},
        # the 32 best of 4096 scores for every one of 4096 queries
        {"name": "topk_rows", "kind": "topk", "rows": 4096, "cols": 4096, "k": 32, "mode": "topk"},
        # classification preprocessing of one photograph, from pinned host memory to pinned host memory
        {"name": "image_pipeline", "kind": "image", "batch": 1, "height": 512, "width": 512, "size": 224,
         "resize_to": 256},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _lm_shape(rng):
    dim = rng.choice([64, 128])
    heads = rng.choice([4, 6, 8, 12, 16] if dim == 128 else [4, 6, 8, 12, 16, 24])
    d = heads * dim
    return {"d": d, "heads": heads, "layers": rng.randint(2, 24), "ffn": d * rng.choice([3, 4]),
            "vocab": rng.choice([256, 1000, 5000, 32000, 50304])}


def draw(rng):
    kind = rng.choice(["lm_train", "lm_logits", "conv_train", "conv_logits", "contrastive", "attention", "mlp", "rnn",
                       "fft", "topk", "image"])
    c = {"kind": kind}
    if kind in ("lm_train", "lm_logits"):
        c.update(_lm_shape(rng))
        c["seq"] = _log(rng, 64, 2048)
        most = 16384 if kind == "lm_train" else 8192
        c["batch"] = _log(rng, 1, max(1, min(32, most // c["seq"])))
        if kind == "lm_train":
            c["micro"] = c["batch"]
            if c["batch"] % 2 == 0 and rng.random() < 0.5:
                c["micro"] = c["batch"] // 2
            c["norm"], c["pos"] = rng.choice([("rms", "rope"), ("layer", "learned")])
    elif kind in ("conv_train", "conv_logits"):
        c.update(batch=_log(rng, 4, 256), image=rng.choice([32, 48, 64]), classes=rng.choice([10, 37, 100, 1000]))
    elif kind == "contrastive":
        c.update(batch=_log(rng, 128, 4096), hidden=8 * _log(rng, 32, 256), out=rng.choice([64, 128, 256, 512]))
        c["in"] = 8 * _log(rng, 16, 128)
    elif kind == "attention":
        c.update(seq=_log(rng, 96, 2048), dim=rng.choice([64, 128]), causal=rng.random() < 0.3,
                 z_bias=rng.random() < 0.6, lengths=rng.random() < 0.6)
        c["contexts"] = _log(rng, 4, max(8, min(256, 160000 // c["seq"])))
    elif kind == "mlp":
        c.update(batch=_log(rng, 32, 4096), batches=rng.randint(1, 6), hidden=8 * _log(rng, 4, 256),
                 out=_log(rng, 1, 100))
        c["in"] = 8 * _log(rng, 1, 128)
    elif kind == "rnn":
        c.update(cell=rng.choice(["wave", "lstm", "tanh"]), batch=_log(rng, 8, 512), steps=_log(rng, 4, 64),
                 hidden=8 * rng.randint(4, 12), out=_log(rng, 1, 32))
        c["in"] = 8 * _log(rng, 2, 16)
    elif kind == "fft":
        n = 2 ** rng.randint(6, 13)
        if rng.random() < 0.2:
            n = _log(rng, 50, 1000)
        c.update(n=n, rows=_log(rng, 16, max(64, (2 ** 25 if n & (n - 1) == 0 else 2 ** 21) // n)))
    elif kind == "topk":
        c.update(cols=_log(rng, 64, 50000), mode=rng.choice(["topk", "topk", "bottomk", "midk"]))
        if c["mode"] == "midk":
            c["cols"] = min(c["cols"], 8000)
        c["k"] = _log(rng, 1, min(128, c["cols"] // 4))
        c["rows"] = _log(rng, 1, max(4, min(8192, 2 ** 24 // c["cols"])))
    else:
        c.update(batch=_log(rng, 1, 16), height=_log(rng, 230, 1024), width=_log(rng, 230, 1024),
                 size=rng.choice([160, 192, 224]), resize_to=rng.choice([232, 256]))
    return c


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1 + seed)


def _lm_config(c):
    return GPTConfig(vocab_size=c["vocab"], d_model=c["d"], n_layers=c["layers"], n_heads=c["heads"], ffn=c["ffn"],
                     seq_len=c["seq"], norm=c.get("norm", "rms"), positional=c.get("pos", "rope"))


def prepare(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    rn = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
    if kind == "lm_train":
        model = GPTModel(_lm_config(c), device=DEV, seed=seed)
        trainer = LMTrainer(model, FlatAdamW(model, lr=3e-4), micro_batch=c["micro"])
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g, device=DEV).cpu()
        return {"kind": kind, "trainer": trainer, "tokens": ids[:, :-1].contiguous().pin_memory(),
                "targets": ids[:, 1:].contiguous().pin_memory()}
    if kind == "lm_logits":
        model = GPTModel(_lm_config(c), device=DEV, seed=seed)
        return {"kind": kind, "model": model,
                "tokens": torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g, device=DEV)}
    if kind in ("conv_train", "conv_logits"):
        model = ConvClassifier(num_classes=c["classes"], image=c["image"], device=DEV, seed=seed)
        s = {"kind": kind, "model": model, "images": rn(c["batch"], 3, c["image"], c["image"]).bfloat16()}
        if kind == "conv_train":
            s["labels"] = torch.randint(0, c["classes"], (c["batch"],), generator=g, device=DEV)
            s["opt"] = FlatSGD(model, lr=0.005, momentum=0.9)
        return s
    if kind == "contrastive":
        return {"kind": kind, "encoder": ContrastiveEncoder(c["in"], c["hidden"], c["out"], device=DEV, seed=seed),
                "base": rn(c["batch"], c["in"]), "seed": seed}
    if kind == "attention":
        shape = (c["contexts"], c["seq"], c["dim"])
        s = {"kind": kind, "q": rn(*shape), "k": rn(*shape), "v": rn(*shape), "grad": rn(*shape), "causal": c["causal"],
             "z_bias": rn(*shape[:2]) if c["z_bias"] else None, "lengths": None}
        if c["lengths"]:
            s["lengths"] = torch.randint(c["seq"] // 2, c["seq"] + 1, (c["contexts"],), generator=g, device=DEV,
                                         dtype=torch.int32)
        return s
    if kind == "mlp":
        net = st.nn.Sequential()
        net.add(st.nn.Linear(c["in"], c["hidden"], name="fc1").init_normal(1 / math.sqrt(c["in"]), seed=seed))
        net.add(st.nn.LayerNorm("ln", c["hidden"]))
        net.add(st.nn.Relu())
        net.add(st.nn.Linear(c["hidden"], c["out"], name="head").init_normal(1 / math.sqrt(c["hidden"]), seed=seed + 1))
        net.to(DEV)
        batches = [(st.Tensor(rn(c["batch"], c["in"])), st.Tensor(rn(c["batch"], c["out"]))) for _ in range(c["batches"])]
        return {"kind": kind, "net": net, "batches": batches, "loss": st.nn.MeanSquaredError(),
                "trainer": st.SpiralSession("cuda", seed=7).trainer(fallback_learning_rate=1e-2)}
    if kind == "rnn":
        layer = {"wave": st.nn.WaveRnn, "lstm": st.nn.Lstm, "tanh": st.nn.SpiralRnn}[c["cell"]]
        net = st.nn.Sequential()
        net.add(layer("cell", c["in"], c["hidden"], c["steps"]))
        net.add(st.nn.Linear(c["hidden"], c["out"], name="head").init_normal(1 / math.sqrt(c["hidden"]), seed=seed))
        net.to(DEV)
        return {"kind": kind, "net": net, "x": st.Tensor(rn(c["batch"], c["steps"] * c["in"])),
                "y": st.Tensor(rn(c["batch"], c["out"])), "loss": st.nn.MeanSquaredError()}
    if kind == "fft":
        return {"kind": kind, "x": torch.view_as_complex(rn(c["rows"], c["n"], 2))}
    if kind == "topk":
        return {"kind": kind, "x": rn(c["rows"], c["cols"]), "k": c["k"], "mode": c["mode"]}
    photo = torch.rand(c["batch"], 3, c["height"], c["width"], generator=g, device=DEV).cpu().pin_memory()
    return {"kind": kind, "photo": photo, "size": c["size"], "resize_to": c["resize_to"],
            "out": torch.empty(c["batch"], 3, c["size"], c["size"]).pin_memory()}


def run(s):
    kind = s["kind"]
    if kind == "lm_train":
        t = s["trainer"]
        loss = t.train_step(s["tokens"], s["targets"])
        return {"loss": loss, "weights": t.model.flat_w, "moments": t.optimizer.m}
    if kind == "lm_logits":
        return s["model"](s["tokens"])
    if kind == "conv_train":
        loss = s["model"].forward_backward(s["images"], s["labels"])
        s["opt"].step()
        return {"loss": loss, "weights": s["opt"].master, "momentum": s["opt"].buf}
    if kind == "conv_logits":
        return s["model"](s["images"])
    if kind == "contrastive":
        enc = s["encoder"]
        enc.zero_grad(set_to_none=True)
        loss = contrastive_step(enc, s["base"], 0.1, seed=s["seed"])
        return [loss] + [p.grad for p in enc.parameters()]
    if kind == "attention":
        q, k, v = (s[n].detach().requires_grad_(True) for n in "qkv")
        o = fn.scaled_dot_attention(q, k, v, z_bias=s["z_bias"], causal=s["causal"], lengths=s["lengths"])
        return (o.detach(),) + torch.autograd.grad(o, (q, k, v), s["grad"])
    if kind == "mlp":
        stats = s["trainer"].train_epoch(s["net"], s["loss"], s["batches"])
        return [stats.average_loss] + [p.value for p in s["net"].parameters()]
    if kind == "rnn":
        net, x, y = s["net"], s["x"], s["y"]
        pred = net.forward(x)
        value = s["loss"].forward(pred, y)
        dx = net.backward(x, s["loss"].backward(pred, y))
        net.apply_step(1e-2)
        return [value.torch(), dx.torch()] + [p.value for p in net.parameters()]
    if kind == "fft":
        z = spectral.fft(s["x"])
        return z, spectral.fft(z, inverse=True)
    if kind == "topk":
        return rank.rank_select(s["x"], s["k"], s["mode"])
    y = vision.classification_pipeline(s["photo"].to(DEV, non_blocking=True), s["size"], s["resize_to"])
    s["out"].copy_(y, non_blocking=True)
    torch.cuda.current_stream().synchronize()
    return s["out"]


def work(case):
    c, kind = case, case["kind"]
    if kind in ("lm_train", "lm_logits"):
        cfg, tokens = _lm_config(c), c["batch"] * c["seq"]
        if kind == "lm_train":      # fp32 master and two moments read and written, bf16 weights read and written, token ids
            return {"bytes": cfg.param_count() * 28.0 + tokens * 16.0, "flops": cfg.flops_per_token() * tokens}
        return {"bytes": cfg.param_count() * 2.0 + tokens * (8.0 + 2.0 * c["vocab"]),
                "flops": cfg.flops_per_token() / 3 * tokens}
    if kind in ("conv_train", "conv_logits"):
        macs, params, ic, hw = 0.0, 0.0, 3, c["image"] ** 2
        first = 0.0
        for oc in STAGES:
            for _ in range(2):
                macs += hw * 9.0 * ic * oc
                params += 9.0 * ic * oc + oc
                first = first or macs
                ic = oc
            hw //= 4
        macs, params = macs + 512.0 * c["classes"], params + 513.0 * c["classes"]
        images = c["batch"] * 3.0 * c["image"] ** 2 * 2
        if kind == "conv_train":
            return {"bytes": images + params * 20.0, "flops": 2.0 * c["batch"] * (3 * macs - first)}
        return {"bytes": images + params * 2.0 + c["batch"] * c["classes"] * 2.0, "flops": 2.0 * c["batch"] * macs}
    if kind == "contrastive":
        params = c["in"] * c["hidden"] + c["hidden"] ** 2 + c["hidden"] * c["out"]
        b = c["batch"]
        return {"bytes": params * 4.0 + b * c["in"] * 12.0,
                "flops": 12.0 * b * params - 4.0 * b * c["in"] * c["hidden"] + 6.0 * b * b * c["out"]}
    if kind == "attention":
        n = c["contexts"] * c["seq"] * c["dim"]
        share = (0.5 if c["causal"] else 1.0) * (0.5833 if c["lengths"] else 1.0)   # E[(length / seq)^2] = 7/12
        return {"bytes": n * 8 * 4.0, "flops": 14.0 * n * c["seq"] * share}
    if kind == "mlp":
        params = c["in"] * c["hidden"] + c["hidden"] * c["out"] + 3.0 * c["hidden"] + c["out"]
        rows = c["batch"] * c["batches"]
        return {"bytes": rows * (c["in"] + c["out"]) * 4.0 + params * 8.0, "flops": 6.0 * rows * params}
    if kind == "rnn":
        gates = {"wave": 2, "lstm": 4, "tanh": 1}[c["cell"]] * c["hidden"]
        params = (c["in"] + c["hidden"] + 1.0) * gates + (c["hidden"] + 1.0) * c["out"]
        rows = c["batch"] * c["steps"]
        return {"bytes": rows * c["in"] * 8.0 + params * 8.0, "flops": 6.0 * rows * (c["in"] + c["hidden"]) * gates}
    if kind == "fft":
        n = float(c["rows"]) * c["n"]
        return {"bytes": n * 8 * 4.0, "flops": 10.0 * n * math.log2(c["n"])}
    if kind == "topk":
        return {"bytes": c["rows"] * (c["cols"] * 4.0 + c["k"] * 8.0), "flops": float(c["rows"]) * c["cols"]}
    src, dst = c["batch"] * 3.0 * c["height"] * c["width"], c["batch"] * 3.0 * c["size"] ** 2
    return {"bytes": 2 * 4 * (src + dst), "flops": 40.0 * dst + src}


def tolerance(case):
    """About four times what the path differs by from itself with other sums: the language model with its two attention
    kernels, the others against the same modules on the CPU (bf16 roundings at the same places, or fp64 where the entry
    point takes it).  Gradients of a deep bf16 model differ by 1 to 3 % that way, single elements by their own size."""
    kind = case["kind"]
    if kind in ("lm_train", "conv_train"):      # measured: moments 1.4e-2, momentum 1.1e-2 to 2.9e-2; single values 0.9
        return {"rel": 3e-2, "max": 0.99}
    if kind in ("lm_logits", "conv_logits"):    # measured: 1.4e-2, single values 7.8e-2
        return {"rel": 3e-2, "max": 0.3}
    if kind == "contrastive":                   # measured: 4.5e-3, single values 2e-2
        return {"rel": 1.8e-2, "max": 0.08}
    if kind == "attention":                     # measured: 4.4e-3, single values 0.1
        return {"rel": 1.8e-2, "max": 0.4}
    if kind == "mlp":                           # measured: 7.5e-3, single values 3.8e-2
        return {"rel": 3e-2, "max": 0.15}
    if kind == "rnn":                           # measured: 3.4e-3, single values 5.7e-2
        return {"rel": 1.4e-2, "max": 0.23}
    if kind == "fft":                           # measured against fp64: 7.2e-7, single values 3.5e-6
        return {"rel": 3e-6, "max": 1.4e-5}
    if kind == "topk":
        return "exact"
    return {"rel": 1e-6, "max": 1e-5}           # measured: 8e-8, single values 4.4e-7


# ---- 64-bit references ------------------------------------------------------------------------------------------------
# The inputs and initial weights are those of ``prepare``; everything after that is plain torch in 64 bits.

def _leaf(t):
    return t.detach().double().requires_grad_(True)


def _lm_exact(c, s):
    model = s["trainer"].model if c["kind"] == "lm_train" else s["model"]
    cfg, heads, dim = model.cfg, c["heads"], c["d"] // c["heads"]
    w = {n: _leaf(p) for n, p in model.p.items()}
    tokens = s["tokens"].to(DEV)
    b, length = tokens.shape

    def norm(x, name):
        if cfg.norm == "rms":
            return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + cfg.norm_eps) * w[name + ".gamma"]
        return F.layer_norm(x, (c["d"],), w[name + ".gamma"], w[name + ".beta"], cfg.norm_eps)

    half = torch.arange(0, dim, 2, dtype=torch.float64, device=DEV) / dim
    angle = torch.arange(length, dtype=torch.float64, device=DEV)[:, None] / cfg.rope_base ** half
    cos, sin = angle.cos(), angle.sin()

    def turn(x):
        if cfg.positional != "rope":
            return x
        u, v = x.chunk(2, -1)
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    keys = torch.arange(length, device=DEV)
    dead = keys[None, :] > keys[:, None]

    def block(x, n):
        qkv = (norm(x, f"h{n}.norm1") @ w[f"h{n}.qkv.weight"].t()).view(b, length, 3, heads, dim).permute(2, 0, 3, 1, 4)
        q, k, v = turn(qkv[0]), turn(qkv[1]), qkv[2]
        o = []
        for i in range(b):
            p = torch.softmax((q[i] @ k[i].transpose(-1, -2) / math.sqrt(dim)).masked_fill(dead, float("-inf")), -1)
            o.append(p @ v[i])
        o = torch.stack(o).transpose(1, 2).reshape(b, length, c["d"])
        x = x + o @ w[f"h{n}.proj.weight"].t()
        return x + F.gelu(norm(x, f"h{n}.norm2") @ w[f"h{n}.fc1.weight"].t(), approximate="tanh") @ w[f"h{n}.fc2.weight"].t()

    x = w["embed.weight"][tokens]
    if cfg.positional == "learned":
        x = x + w["pos.weight"][:length]
    for n in range(c["layers"]):
        x = checkpoint(block, x, n, use_reentrant=False)
    logits = norm(x, "norm_f").reshape(b * length, -1) @ w["embed.weight"].t()
    if c["kind"] == "lm_logits":
        return logits.detach()
    loss = F.cross_entropy(logits, s["targets"].to(DEV).reshape(-1))
    loss.backward()
    opt = s["trainer"].optimizer
    total = math.sqrt(sum(float(t.grad.pow(2).sum()) for t in w.values()))
    clip = min(1.0, opt.max_grad_norm / (total + 1e-6)) if opt.max_grad_norm > 0 else 1.0
    weights, moments = torch.zeros_like(opt.master, dtype=torch.float64), torch.zeros_like(opt.m, dtype=torch.float64)
    for name, at, n, _ in model.named_flat_views():
        g = w[name].grad.reshape(-1) * clip
        old = w[name].detach().reshape(-1)
        decay = opt.weight_decay if at < opt.decay_elems else 0.0
        weights[at:at + n] = old - opt.lr * (g / (g.abs() + opt.eps) + decay * old)
        moments[at:at + n] = (1 - opt.betas[0]) * g
    return {"loss": loss.item(), "weights": weights, "moments": moments}


def _conv_exact(c, s):
    model = s["model"]
    w = {n: _leaf(p) for n, p in model.p.items()}
    x, ic = s["images"].double(), 3
    for stage, oc in enumerate(STAGES):
        for i in range(2):
            k = w[f"conv{stage}_{i}.weight"].view(oc, 3, 3, ic).permute(0, 3, 1, 2)
            x = torch.relu(F.conv2d(x, k, w[f"conv{stage}_{i}.bias"], padding=1))
            ic = oc
        x = F.max_pool2d(x, 2)
    logits = (x.mean((2, 3)) @ w["head.weight"].t() + w["head.bias"])[:, :c["classes"]]
    if c["kind"] == "conv_logits":
        return logits.detach()
    loss = F.cross_entropy(logits, s["labels"])
    loss.backward()
    weights, momentum = s["opt"].master.double(), torch.zeros_like(s["opt"].buf, dtype=torch.float64)
    for name, (at, n, _) in model._offsets.items():
        g = w[name].grad.reshape(-1)
        momentum[at:at + n] = g
        weights[at:at + n] -= s["opt"].lr * g
    return {"loss": loss.item(), "weights": weights, "momentum": momentum}


def _contrastive_exact(c, s):
    p = [_leaf(t) for t in s["encoder"].parameters()]
    weight, bias, gamma, beta = p[0:3], p[3:6], p[6:8], p[8:10]
    g = torch.Generator(device=DEV).manual_seed(s["seed"])
    noise = [torch.randn(s["base"].shape, generator=g, device=DEV) for _ in range(2)]

    def embed(x):
        for i in range(3):
            x = x @ weight[i].t() + bias[i]
            if i < 2:
                x = F.gelu(F.layer_norm(x, (x.shape[-1],), gamma[i], beta[i], 1e-5), approximate="tanh")
        return F.normalize(x, dim=-1)

    a, b = (embed(s["base"].double() + 0.1 * n.double()) for n in noise)
    loss = F.cross_entropy(a @ b.t() / 0.1, torch.arange(c["batch"], device=DEV))
    loss.backward()
    return [loss.item()] + [t.grad for t in p]


def _attention_exact(c, s):
    q, k, v = (_leaf(s[n]) for n in "qkv")
    o, keys = [], torch.arange(c["seq"], device=DEV)
    grads = [torch.empty_like(q) for _ in range(3)]
    for i in range(c["contexts"]):
        n = int(s["lengths"][i]) if c["lengths"] else c["seq"]
        score = q[i, :n] @ k[i, :n].t() / math.sqrt(c["dim"])
        if c["z_bias"]:
            score = score + s["z_bias"][i, :n].double()
        if c["causal"]:
            score = score.masked_fill(keys[None, :n] > keys[:n, None], float("-inf"))
        y = F.pad(torch.softmax(score, -1) @ v[i, :n], (0, 0, 0, c["seq"] - n))
        for g, t in zip(grads, torch.autograd.grad(y, (q, k, v), s["grad"][i].double())):
            g[i] = t[i]
        o.append(y.detach())
    return (torch.stack(o), *grads)


def _mlp_exact(c, s):
    p = [t.value.double() for t in s["net"].parameters()]     # fc1 weight and bias, gain, offset, head weight and bias
    total = 0.0
    for x, y in s["batches"]:
        leaf = [_leaf(t) for t in p]
        h = torch.relu(F.layer_norm(x.torch().double() @ leaf[0] + leaf[1], (c["hidden"],), leaf[2].reshape(-1), leaf[3].reshape(-1), 1e-5))
        loss = F.mse_loss(h @ leaf[4] + leaf[5], y.torch().double())
        p = [t.detach() - 1e-2 / c["batch"] * g for t, g in zip(leaf, torch.autograd.grad(loss, leaf))]
        total += loss.item()
    return [total / c["batches"]] + p


def _rnn_exact(c, s):
    leaf = [_leaf(t.value) for t in s["net"].parameters()]    # input weights, recurrent weights, bias, head weight and bias
    x, hidden = _leaf(s["x"].torch()), c["hidden"]
    h = cell = torch.zeros(c["batch"], hidden, dtype=torch.float64, device=DEV)
    past = []
    for t in range(c["steps"]):
        into = h + past[t - 2] if c["cell"] == "wave" and t >= 2 else h
        z = x[:, t * c["in"]:(t + 1) * c["in"]] @ leaf[0] + into @ leaf[1] + leaf[2]
        if c["cell"] == "tanh":
            h = torch.tanh(z)
        elif c["cell"] == "wave":
            h = torch.tanh(z[:, :hidden]) * torch.sigmoid(z[:, hidden:])
        else:
            i, f, g, o = z.chunk(4, 1)
            cell = torch.sigmoid(f) * cell + torch.sigmoid(i) * torch.tanh(g)
            h = torch.sigmoid(o) * torch.tanh(cell)
        past.append(h)
    loss = F.mse_loss(h @ leaf[3] + leaf[4], s["y"].torch().double())
    dx, *grads = torch.autograd.grad(loss, [x] + leaf)
    return [loss.detach().reshape(1, 1), dx] + [t.detach() - 1e-2 / c["batch"] * g for t, g in zip(leaf, grads)]


def _image_exact(c, s):
    x, r = s["photo"].to(DEV).double(), c["resize_to"]
    means = (x * 1.1).mean((0, 2, 3)).view(1, 3, 1, 1)
    x = F.interpolate(x, (r, r), mode="bilinear", align_corners=False)
    at = (r - c["size"]) // 2
    x = x[:, :, at:at + c["size"], at:at + c["size"]] * 1.1
    x = (x - means) * 1.1 + means
    gray = (x * torch.tensor([0.29899597, 0.587096, 0.11390703], dtype=torch.float64, device=DEV).view(1, 3, 1, 1)).sum(1, keepdim=True)
    red, green, blue = ((x - gray) * 1.1 + gray).unbind(1)
    y = 0.299 * red + 0.587 * green + 0.114 * blue
    u, v = -0.14713 * red - 0.28886 * green + 0.436 * blue, 0.615 * red - 0.51499 * green - 0.10001 * blue
    u, v = u * math.cos(0.05) - v * math.sin(0.05), u * math.sin(0.05) + v * math.cos(0.05)
    return torch.stack([y + 1.13983 * v, y - 0.39465 * u - 0.5806 * v, y + 2.03211 * u], 1).flip(-1).cpu()


def exact(case, seed):
    """The outputs of ``run`` in 64 bits; ``None`` for a selection, whose values are inputs, and for work of over 4e14
    operations."""
    c, kind = case, case["kind"]
    if kind == "topk" or work(case)["flops"] > 4e14:
        return None
    s = prepare(case, seed)
    if kind == "fft":
        z = torch.fft.fft(s["x"].to(torch.complex128))
        return z, torch.fft.ifft(z)
    form = {"lm_train": _lm_exact, "lm_logits": _lm_exact, "conv_train": _conv_exact, "conv_logits": _conv_exact,
            "contrastive": _contrastive_exact, "attention": _attention_exact, "mlp": _mlp_exact, "rnn": _rnn_exact,
            "image": _image_exact}[kind]
    with torch.set_grad_enabled(kind not in ("lm_logits", "conv_logits", "image")):
        return form(c, s)

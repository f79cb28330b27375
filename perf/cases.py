"""What a user of kaon_b200 has it do: optimizer steps over the parameter lists of real training runs.

A case names a recipe (an optimizer with the constructor arguments it is run with) and a parameter list.
``prepare`` builds the list in flat buffers (weights, gradients, optimizer state: the layout of a sharded
run, and the reason a pass can hand back everything it wrote), takes two steps so that momentum, statistics
and plan are those of a run under way, and draws fresh gradients in between; ``run`` is one ``opt.step()``.
"""
from __future__ import annotations

import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "k-optimizers_b200"))
import kaon_b200  # noqa: E402
from kaon_b200 import workloads  # noqa: E402

BF16, F32 = "bfloat16", "float32"

# recipe -> (class, weight dtype, constructor arguments, share of gradient elements scaled x100)
RECIPES = {
    # the headline configuration: sign momentum in 4 bits, cautious mask, stochastic rounding
    "lion_4bit": ("Lion", BF16, dict(lr=2e-4, betas=(0.95, 0.98), momentum_dtype="4bit"), 0.0),
    # Lion as constructed by default (bf16 momentum) on fp32 master weights, with weight decay
    "lion_f32": ("Lion", F32, dict(lr=1e-4, weight_decay=0.05), 0.0),
    # factored second moment, int8 momentum, gradients with outliers
    "adakaon_int8": ("Adakaon", BF16, dict(lr=1e-4, momentum_dtype="int8"), 0.01),
    # Adakaon's default momentum with the Kahan weight write
    "adakaon_kahan": ("Adakaon", BF16, dict(lr=1e-4, weight_decay=0.01, bf16_method="kahan"), 0.0),
    # Adakaon's defaults on fp32 weights, as adapters are trained
    "adakaon_f32": ("Adakaon", F32, dict(lr=1e-4), 0.0),
    # Nekaon's defaults (4-bit momentum, lookahead, weight decay), beta1 of the benchmark configuration
    "nekaon_4bit": ("Nekaon", BF16, dict(lr=1e-4, betas=(0.2, 0.999)), 0.0),
    # orthogonalised momentum of the DiT configuration, and AdaMuon's defaults
    "adamuon_int8": ("AdaMuon", BF16, dict(lr=1e-3, ns_steps=2, momentum_dtype="int8"), 0.0),
    "adamuon_bf16": ("AdaMuon", BF16, dict(lr=1e-3), 0.0),
    # two momenta, both in 4 bits
    "adapnm_4bit": ("AdaPNM", BF16, dict(lr=1e-4, momentum_dtype="4bit"), 0.0),
    # KProdigy's defaults once the distance estimate has settled
    "kprodigy": ("KProdigy", BF16, dict(d0=1e-4, growth_rate=1.0), 0.0),
}

# recipe -> the kinds of list it is drawn with
KINDS = {
    "lion_4bit": ("unet", "lora", "bag", "ragged"),
    "lion_f32": ("unet", "lora", "ragged"),
    "adakaon_int8": ("unet", "lora", "ragged"),
    "adakaon_kahan": ("unet", "ragged"),
    "adakaon_f32": ("lora", "bag", "unet"),
    "nekaon_4bit": ("unet", "lora"),
    "adamuon_int8": ("dit", "unet"),
    "adamuon_bf16": ("unet", "dit"),
    "adapnm_4bit": ("unet", "lora"),
    "kprodigy": ("unet", "lora"),
}


def _block(w):
    return [(w, w)] * 4 + [(8 * w, w), (w, 4 * w)] + [(w,)] * 6


def shapes_of(case):
    """The parameter list of a case."""
    kind = case["list"]
    if kind in workloads.WORKLOADS:
        return workloads.WORKLOADS[kind]()
    if kind == "c1":        # one linear layer, one convolution, one bias: a single call's worth of work
        return [(1024, 1024), (320, 320, 3, 3), (1024,)]
    if kind == "bag":       # many tiny adapter matrices
        return [(8, 16)] * case["count"]
    w, n = case["width"], case["count"]
    if kind == "lora":      # low-rank pairs on the four attention projections of every block
        r = case["rank"]
        return [s for _ in range(n) for _ in range(4) for s in ((r, w), (w, r))]
    if kind == "dit":
        return [(3 * w, w), (w, w), (4 * w, w), (w, 4 * w), (w,), (w,)] * n
    if kind == "unet":      # transformer blocks and 3x3 convolutions; `ends`: the odd tensors at a UNet's ends
        out = _block(w) * n + [(w, w, 3, 3)] * case["convs"]
        return out + ([(w, 4, 3, 3), (4, w, 3, 3), (333, 77)] if case["ends"] else [])
    if kind == "ragged":    # tables, convolutions and biases whose sizes are multiples of nothing
        rng, out = random.Random(n), []
        for _ in range(n):
            out.append((rng.randrange(w // 2, 2 * w) | 1, rng.randrange(w // 2, w) | 1))
            out.append((rng.randrange(w // 8, w // 2) | 1, rng.randrange(3, 67), 3, 3))
            out.append((rng.randrange(w // 2, 2 * w) | 1,))
        return out
    raise ValueError(kind)


def listed():
    return [
        # the smallest steps: a bag of adapters, one layer, the low-rank pairs of a whole UNet
        {"name": "lion_4bit_bag", "recipe": "lion_4bit", "list": "bag", "count": 512},
        {"name": "adakaon_int8_c1", "recipe": "adakaon_int8", "list": "c1"},
        {"name": "adakaon_f32_lora", "recipe": "adakaon_f32", "list": "lora", "width": 1280, "count": 90, "rank": 8},
        # AdaMuon on a small UNet with its odd end tensors
        {"name": "adamuon_bf16_small", "recipe": "adamuon_bf16", "list": "unet", "width": 320, "count": 2, "convs": 4, "ends": True},
        # sizes that are multiples of nothing, fp32 weights
        {"name": "lion_f32_ragged", "recipe": "lion_f32", "list": "ragged", "width": 1500, "count": 16},
        # part of a UNet per GPU (a sharded run, a smaller model)
        {"name": "nekaon_4bit_mid", "recipe": "nekaon_4bit", "list": "unet_mid"},
        {"name": "adapnm_4bit_mid", "recipe": "adapnm_4bit", "list": "unet_mid"},
        {"name": "kprodigy_mid", "recipe": "kprodigy", "list": "unet_mid"},
        {"name": "adakaon_kahan_mid_odd", "recipe": "adakaon_kahan", "list": "unet_mid_odd"},
        # AdaMuon on DiT blocks: the one step bound by the tensor cores
        {"name": "adamuon_int8_dit", "recipe": "adamuon_int8", "list": "dit", "width": 3072, "count": 4},
        # a full fine-tune of the 2.6 B-parameter UNet on one GPU
        {"name": "lion_4bit_unet", "recipe": "lion_4bit", "list": "unet_2p6b"},
        {"name": "adakaon_int8_unet", "recipe": "adakaon_int8", "list": "unet_2p6b"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a recipe, a kind of list it is used with, sizes spread over their logarithm."""
    recipe = rng.choice(sorted(RECIPES))
    kind = rng.choice(KINDS[recipe])
    case = {"recipe": recipe, "list": kind}
    muon = recipe.startswith("adamuon")
    if kind == "bag":
        case.update(count=_log(rng, 16, 2048))
    elif kind == "lora":
        case.update(width=64 * _log(rng, 5, 24), count=_log(rng, 1, 120), rank=rng.choice((4, 8, 16, 32, 64)))
    elif kind == "ragged":
        case.update(width=_log(rng, 64, 1999), count=_log(rng, 1, 24))
    elif kind == "dit":
        case.update(width=128 * _log(rng, 3, 24), count=1)
        case["count"] = _log(rng, 1, max(1, 4 * (3072 // case["width"])))
    else:
        w = 64 * _log(rng, 2, 20)
        w = w if w <= 896 else w // 128 * 128
        case.update(width=w, count=_log(rng, 1, 4 if muon else 8), convs=rng.choice((0, 1, 2, 4)), ends=rng.random() < 0.5)
    return case


def _fill(flat, gen, std, outliers):
    flat.normal_(0.0, std, generator=gen)
    if outliers:
        for part in flat.split(1 << 28):
            hot = torch.rand(part.shape, generator=gen, device=part.device, dtype=torch.float32) < outliers
            part.mul_(hot.to(part.dtype).mul_(99.0).add_(1.0))


def _flat(tensors):
    """One buffer for tensors of one dtype (each on a 512-byte boundary, as an allocation of its own is) and the views."""
    step = 512 // tensors[0].element_size()
    at, starts = 0, []
    for t in tensors:
        starts.append(at)
        at += -(-t.numel() // step) * step
    buf = torch.zeros(at, dtype=tensors[0].dtype, device=tensors[0].device)
    return buf, [buf[a:a + t.numel()].view(t.shape) for a, t in zip(starts, tensors)]


def prepare(case, seed):
    cls, dtype, kw, outliers = RECIPES[case["recipe"]]
    dtype = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    like = [torch.empty(s, dtype=dtype, device="meta") for s in shapes_of(case)]
    step = 512 // dtype.itemsize
    total = sum(-(-t.numel() // step) * step for t in like)
    weights, grads = (torch.empty(total, dtype=dtype, device="cuda") for _ in range(2))
    params, at = [], 0
    for t in like:
        p = torch.nn.Parameter(weights[at:at + t.numel()].view(t.shape))
        p.grad = grads[at:at + t.numel()].view(t.shape)
        params.append(p)
        at += -(-t.numel() // step) * step
    _fill(weights, gen, 0.02, 0.0)
    _fill(grads, gen, 1e-3, outliers)

    def build():
        opt = getattr(kaon_b200, cls)(params, **kw)
        opt.sr_seed = int(seed)
        return opt, getattr(opt, "base_optimizer", opt)

    first, inner = build()
    first.step()
    opt, kept = build()
    for old, new in zip(inner.param_groups, kept.param_groups):     # the counters of the optimizers that keep some there
        new.update({k: v for k, v in old.items() if k != "params"})
    state = {}
    for key in sorted({k for p in params for k in inner.state[p]}):
        have = [p for p in params if key in inner.state[p]]
        if not torch.is_tensor(inner.state[have[0]][key]):
            for p in have:
                kept.state[p][key] = inner.state[p][key]
            continue
        old = [inner.state[p][key] for p in have]
        state[key], views = _flat(old)
        torch._foreach_copy_(views, old)
        for p, v in zip(have, views):
            kept.state[p][key] = v
    _fill(grads, gen, 1e-3, outliers)
    opt.step()
    return {"opt": opt, "groups": kept.param_groups, "weights": weights, "grads": grads, "state": state}


def run(s):
    s["opt"].step()
    out = {"weights": s["weights"], **s["state"]}
    if "d" in s["groups"][0]:
        out["d"] = float(s["groups"][0]["d"])
    return out


def work(case):
    """Bytes: gradient read, weights and state read and written, each once.  Flops: the three products of a
    Newton-Schulz iteration, the symmetric two of them counted by half."""
    cls, dtype, kw, _ = RECIPES[case["recipe"]]
    wb = getattr(torch, dtype).itemsize
    md = kw.get("momentum_dtype", "4bit" if cls == "Nekaon" else "bfloat16")
    nbytes = flops = 0.0
    for s in shapes_of(case):
        n = math.prod(s)
        r, c = (s[0], n // s[0]) if len(s) > 1 else (0, 0)
        m = {"bfloat16": 2 * n, "int8": n + 4 * (r or 1), "4bit": n / 2 + 4 * math.ceil(n / 128)}[md]
        b = 3 * wb * n + 2 * m
        if cls == "AdaPNM":
            b += m                              # the second momentum is read only
        if kw.get("bf16_method") == "kahan":
            b += 2 * wb * n
        if cls == "KProdigy":
            b += 4 * (2 + 1 + 2) * n            # s, p0, v
        elif cls != "Lion":
            b += 8 * ((r + c) if r else n)
        nbytes += b
        if cls == "AdaMuon" and r:
            lo, hi = min(r, c), max(r, c)
            flops += kw.get("ns_steps", 2) * (3.0 * lo * lo * hi + 1.0 * lo ** 3)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    cls, _, kw, _ = RECIPES[case["recipe"]]
    if cls == "AdaMuon":        # statistics and weights come out of a chain of bf16 matrix products
        return {"rel": 1e-2, "max": 0.1, "differ": 2e-3}
    # sums in another order: a rare momentum code one step off (and with it the next scale of its row or block, by
    # 1/127 or 1/7), a rare weight on the other bf16 neighbour
    four = kw.get("momentum_dtype", "4bit" if cls == "Nekaon" else "") == "4bit"
    return {"rel": 1e-3, "max": 0.16 if four else 0.03, "differ": 2e-3}

"""The work that performance is judged on: which calls a program that serves a quantised model makes, at which sizes.

A model served by this library spends its time in six ways, and each has its cases here:

  projections   the linear projections of a layer (and the output head) on M activation rows through ``matmul``: decode of one
                row, a small batch or speculative verification of several rows, a short prompt, a long prompt
  token         one decoded token with every fused form: embedding row, RMSNorm into Q+K+V, output projection plus residual,
                RMSNorm into gate+up, silu*up into down plus residual, output head, greedy choice
  linear        one projection by itself, the smallest call there is
  experts       the routed-expert feed-forward step of a mixture-of-experts layer
  host          a decode step whose activations and results live in pinned host memory

Sizes are those of the benchmark's configurations (Llama-3 8B and 70B projections, the 128-expert layer of hidden size 2048)
and ragged ones between.  Row counts, odd ones among them, run from 1 to 2048.  ``draw`` takes sizes from the same ranges.
"""
from __future__ import annotations

import math

import torch

import backpack_b200 as bp
from backpack_b200 import q4k

BLOCK = {"q4_k": 144, "q5_k": 176, "q6_k": 224}                       # stored bytes of 256 weights (Q6_K in its padded device layout)
FILE_BLOCK = {"q4_k": 144, "q5_k": 176, "q6_k": 210}                  # bytes that carry information
QTYPE = {"q4_k": q4k.Q4_K, "q5_k": q4k.Q5_K, "q6_k": q4k.Q6_K_PADDED}
MODE = {"f16x3": q4k.PREFILL_F16X3, "f16": q4k.PREFILL_F16, "bf16": q4k.PREFILL_BF16}

# hidden size, rows of Q+K+V, feed-forward size, rows of the output head
LLAMA_8B = {"hidden": 4096, "qkv": 6144, "ffn": 14336}
LLAMA_70B = {"hidden": 8192, "qkv": 10240, "ffn": 28672}
HEAD = 128256
PROJECTIONS = {"path": "projections", "type": "q4_k", "down": "q4_k", "mode": "f16x3", "head": 0}


def listed():
    return [
        # the key or value projection of one token: nothing but latency
        {"name": "linear_1", "path": "linear", "m": 1, "n": 1024, "k": 4096, "type": "q4_k", "bias": False},
        # one token through the projections of a layer and the output head, all Q4_K: plain decode
        dict(PROJECTIONS, name="decode_1", m=1, head=HEAD, **LLAMA_8B),
        # one token of a "Q4_K_M" file (down projection and head in Q6_K) with every fused form, two layers deep
        dict(LLAMA_8B, name="token_q4km", path="token", layers=2, type="q4_k", down="q6_k", head=HEAD),
        # eight rows through a 70B layer: a small batch, or the check of eight speculated tokens
        dict(PROJECTIONS, name="batch_8_70b", m=8, **LLAMA_70B),
        # a ragged batch between decode and prefill
        dict(PROJECTIONS, name="batch_13", m=13, head=HEAD, **LLAMA_8B),
        # a short prompt: a chat turn of a few words
        dict(PROJECTIONS, name="prompt_37", m=37, head=HEAD, **LLAMA_8B),
        # a middling prompt of a "Q5_K_M" file (Q6_K down projection)
        dict(PROJECTIONS, name="prompt_200_q5km", m=200, **dict(LLAMA_8B, type="q5_k", down="q6_k")),
        # the prefill configuration, in the mode that keeps float accuracy (the default) and in the bfloat16 mode
        dict(PROJECTIONS, name="prompt_512", m=512, head=HEAD, **LLAMA_8B),
        dict(PROJECTIONS, name="prompt_512_bf16", m=512, head=HEAD, **dict(LLAMA_8B, mode="bf16")),
        # a long prompt through a 70B layer: the largest
        dict(PROJECTIONS, name="prompt_2048_70b", m=2048, **LLAMA_70B),
        # speculative verification through a mixture-of-experts layer: eight rows, eight of 128 experts each
        {"name": "experts_8", "path": "experts", "m": 8, "topk": 8, "experts": 128, "hidden": 2048, "ffn": 768, "type": "q4_k"},
        # a decode step driven from host memory: activations up, results down, one wait
        dict(LLAMA_8B, name="host_1", path="host", m=1, type="q4_k", head=HEAD),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def width(lo, hi):  # a contraction length: whole super-blocks
        return max(1, log_int(lo, hi) // 256) * 256

    path = rng.choice(["linear", "projections", "projections", "projections", "token", "experts", "host"])
    if path == "linear":
        return {"path": path, "m": log_int(1, 64), "n": log_int(64, 16384), "k": width(256, 16384),
                "type": rng.choice(["q4_k", "q4_k", "q5_k", "q6_k"]), "bias": rng.random() < 0.3}
    hidden = width(2048, 8192)
    shape = {"hidden": hidden, "qkv": hidden + 2 * log_int(256, hidden // 2), "ffn": width(2 * hidden, 3.5 * hidden)}
    if path == "projections":
        return dict(PROJECTIONS, m=log_int(1, 2048), **dict(shape, type=rng.choice(["q4_k", "q4_k", "q4_k", "q5_k"]),
                    down=rng.choice(["q4_k", "q4_k", "q6_k"]), mode=rng.choice(["f16x3", "f16x3", "f16x3", "f16", "bf16"])))
    if path == "token":
        return dict(shape, path=path, layers=rng.randint(1, 3), type=rng.choice(["q4_k", "q5_k"]), down=rng.choice(["q5_k", "q6_k"]),
                    head=log_int(16384, 131072))
    if path == "experts":
        return {"path": path, "m": log_int(1, 32), "topk": rng.choice([2, 4, 8]), "experts": rng.choice([32, 64, 128]),
                "hidden": width(1024, 4096), "ffn": width(512, 1536), "type": rng.choice(["q4_k", "q4_k", "q5_k"])}
    return dict(shape, path=path, m=log_int(1, 8), type="q4_k", head=log_int(16384, 131072))


# ---- inputs ------------------------------------------------------------------------------------------------------------

_contexts = {}


def _context(mode="f16x3"):
    """One handle per precision mode for the whole process, as a serving program keeps it."""
    if mode not in _contexts:
        _contexts[mode] = bp.Q4KContext(torch.cuda.current_device())
        _contexts[mode].set_option(q4k.OPT_PREFILL_MODE, MODE[mode])
    return _contexts[mode]


def _weight(kind, n, k, gen):
    """Random super-blocks whose weights are spread as a trained model's are: zero mean, standard deviation about 0.02.
    4- and 5-bit types: w = d*sc*q - dmin*mn with mn near sc and dmin*mn near the middle of the codes' range."""
    nblk, bb = n * (k // 256), BLOCK[kind]
    raw = torch.empty((nblk, bb), dtype=torch.uint8, device="cuda")
    raw.view(torch.int64).random_(generator=gen)  # (63 random bits a word: the eighth bytes are half as wide, rewritten next)
    raw[:, 7::8].random_(generator=gen)

    def halves(lo, hi):
        return torch.empty(nblk, device="cuda").uniform_(lo, hi, generator=gen).half()

    if kind == "q6_k":
        raw[:, 192:208] = torch.randint(20, 101, (nblk, 16), generator=gen, device="cuda", dtype=torch.int16).to(torch.uint8)
        raw[:, 192:208:3] = (256 - raw[:, 192:208:3].to(torch.int16)).to(torch.uint8)   # some scales are negative
        raw[:, 208:210] = halves(1e-5, 3e-5).view(torch.uint8).view(nblk, 2)
        raw[:, 210:] = 0
    else:
        codes = 15 if kind == "q4_k" else 31
        d = halves(2e-3 / codes, 3e-3 / codes)
        raw[:, 0:2] = d.view(torch.uint8).view(nblk, 2)
        raw[:, 2:4] = (d.float() * (codes / 2)).half().view(torch.uint8).view(nblk, 2)
        sc = torch.randint(20, 64, (nblk, 8), generator=gen, device="cuda", dtype=torch.int32)
        mn = (sc + torch.randint(-3, 4, (nblk, 8), generator=gen, device="cuda", dtype=torch.int32)).clamp_(0, 63)
        raw[:, 4:8] = (sc[:, :4] | ((sc[:, 4:] >> 4) << 6)).to(torch.uint8)
        raw[:, 8:12] = (mn[:, :4] | ((mn[:, 4:] >> 4) << 6)).to(torch.uint8)
        raw[:, 12:16] = ((sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)).to(torch.uint8)
    return bp.Q4KWeight(raw.view(-1), n, k, (k // 256) * bb // 4, QTYPE[kind])


def _normal(gen, *shape):
    return torch.empty(shape, device="cuda").normal_(generator=gen)


def _shapes(case):
    """(rows, contraction length, type) of the projections of a layer, and of the head if there is one."""
    h, f, t = case["hidden"], case["ffn"], case["type"]
    down = case.get("down", t)
    s = [(case["qkv"], h, t), (h, h, t), (2 * f, h, t), (h, f, down)]
    return s + ([(case["head"], h, down)] if case.get("head") else [])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    path = case["path"]
    s = {"case": case, "ctx": _context(case.get("mode", "f16x3"))}
    if path == "linear":
        s["w"] = _weight(case["type"], case["n"], case["k"], gen)
        s["x"] = _normal(gen, case["m"], case["k"])
        s["bias"] = _normal(gen, case["n"]) if case["bias"] else None
        s["y"] = torch.empty(case["m"], case["n"], device="cuda")
    elif path == "projections":
        s["calls"] = [(_normal(gen, case["m"], k), _weight(t, n, k, gen), torch.empty(case["m"], n, device="cuda"))
                      for n, k, t in _shapes(case)]
    elif path == "token":
        h, f, q = case["hidden"], case["ffn"], case["qkv"]
        s["head"] = _weight(case["down"], case["head"], h, gen)     # also the embedding table
        s["token"] = torch.randint(0, case["head"], (1,), generator=gen, device="cuda", dtype=torch.int32)
        s["norm"] = 1.0 + 0.1 * _normal(gen, h)
        s["hidden"] = [torch.empty(1, h, device="cuda") for _ in range(2 * case["layers"] + 1)]
        s["layers"] = [{"qkv_w": _weight(case["type"], q, h, gen), "o_w": _weight(case["type"], h, h, gen),
                        "gate_up_w": _weight(case["type"], 2 * f, h, gen), "down_w": _weight(case["down"], h, f, gen),
                        "norm1": 1.0 + 0.1 * _normal(gen, h), "norm2": 1.0 + 0.1 * _normal(gen, h),
                        "attention": _normal(gen, 1, h),            # attention is not part of this library: its result
                        "qkv": torch.empty(1, q, device="cuda"), "gate_up": torch.empty(1, 2 * f, device="cuda")}
                       for _ in range(case["layers"])]
        s["logits"] = torch.empty(1, case["head"], device="cuda")
        s["next"] = torch.empty(1, dtype=torch.int32, device="cuda")
    elif path == "experts":
        e, h, f, t = case["experts"], case["hidden"], case["ffn"], case["m"]
        s["gate"], s["up"], s["down"] = (_weight(case["type"], e * n, k, gen) for n, k in ((f, h), (f, h), (h, f)))
        s["x"] = _normal(gen, t, h)
        s["residual"] = _normal(gen, t, h)
        scores = torch.rand(t, e, generator=gen, device="cuda")
        top = scores.topk(case["topk"], dim=1)                       # distinct experts, each equally likely
        s["ids"] = top.indices.to(torch.int32).contiguous()
        s["route"] = torch.softmax(_normal(gen, t, case["topk"]), dim=1).contiguous()
        s["y"] = torch.empty(t, h, device="cuda")
        s["work"] = torch.empty(s["ctx"].lib.bpq4k_moe_ffn_work_floats(t, case["topk"], h, f), device="cuda")
    else:
        items = []
        for n, k, t in _shapes(case):
            w = _weight(t, n, k, gen)
            x = torch.empty(case["m"], k, pin_memory=True)
            x.copy_(_normal(gen, case["m"], k))
            y = torch.empty(case["m"], n, pin_memory=True)
            items.append((x, w, y))
        s["keep"] = items
        s["outputs"] = [y.numpy() for _, _, y in items]
        s["batch"] = s["ctx"].make_host_batch([(x.numpy(), w, y.numpy(), None) for x, w, y in items])
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------

EPS = 1e-5


def run(s):
    ctx, path = s["ctx"], s["case"]["path"]
    if path == "linear":
        return ctx.matmul(s["x"], s["w"], bias=s["bias"], out=s["y"])
    if path == "projections":
        return [ctx.matmul(x, w, out=y) for x, w, y in s["calls"]]
    if path == "token":
        f = s["case"]["ffn"]
        h = ctx.gather(s["head"], s["token"], out=s["hidden"][0])
        out = []
        for i, l in enumerate(s["layers"]):
            ctx.matmul_fused(h, l["qkv_w"], q4k.PROLOGUE_RMSNORM, aux=l["norm1"], eps=EPS, out=l["qkv"])
            h = ctx.matmul_fused(l["attention"], l["o_w"], residual=h, out=s["hidden"][2 * i + 1])
            gu = ctx.matmul_fused(h, l["gate_up_w"], q4k.PROLOGUE_RMSNORM, aux=l["norm2"], eps=EPS, out=l["gate_up"])
            h = ctx.matmul_fused(gu[:, :f], l["down_w"], q4k.PROLOGUE_SILU_MUL, aux=gu[:, f:], residual=h, out=s["hidden"][2 * i + 2])
            out += [l["qkv"], gu, h]
        ctx.matmul_fused(h, s["head"], q4k.PROLOGUE_RMSNORM, aux=s["norm"], eps=EPS, out=s["logits"])
        return out + [s["logits"], ctx.argmax(s["logits"], out=s["next"])]
    if path == "experts":
        s["y"].copy_(s["residual"])
        return ctx.moe_ffn(s["x"], s["gate"], s["up"], s["down"], s["ids"], s["route"], s["y"], s["case"]["experts"], work=s["work"])
    ctx.matmul_host_batch(s["batch"])
    return s["outputs"]


# ---- what a pass cannot do without, and how exact it is -----------------------------------------------------------------

def _matmul_work(m, n, k, kind):
    return n * (k // 256) * FILE_BLOCK[kind] + 4 * m * (k + n), 2 * m * n * k


def work(case):
    path = case["path"]
    if path == "linear":
        parts = [_matmul_work(case["m"], case["n"], case["k"], case["type"])]
    elif path == "experts":
        pairs, e, h, f = case["m"] * case["topk"], case["experts"], case["hidden"], case["ffn"]
        touched = e * (1.0 - (1.0 - case["topk"] / e) ** case["m"])   # distinct experts, on average
        per = 3 * f * (h // 256) * FILE_BLOCK[case["type"]]
        parts = [(touched * per + 4 * 3 * case["m"] * h + 8 * pairs, 6.0 * pairs * h * f)]
    else:
        m = case.get("m", 1)
        layer = [_matmul_work(m, *shape) for shape in _shapes(dict(case, head=0))]
        head = [_matmul_work(m, case["head"], case["hidden"], case.get("down", case["type"]))] if case.get("head") else []
        parts = layer * case.get("layers", 1) + head
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    if case.get("mode") == "bf16":   # measured against 64-bit sums: 4.9e-3, largest 2.8e-2
        return {"rel": 1.2e-2, "max": 8e-2}
    if case.get("mode") == "f16":
        return {"rel": 1.6e-3, "max": 1e-2}
    # Measured against 64-bit sums: 4e-7 (one to 24 rows), 4.9e-6 (three-term half products, whose sums the tensor core truncates)
    if case["path"] in ("linear", "projections") and case["m"] >= 25:
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 1e-5 if case["path"] in ("token", "experts") else 4e-6, "max": 1e-4, "differ": 0.0}

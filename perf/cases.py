"""The work that a user of this framework has it do, as cases whose speed and results can be measured.

A case is one call of a public entry point: an op of ``llmss_b200.ops``, a block of ``llmss_b200.models`` or a whole model.  The
ranges: 1 to 8192 packed tokens (one token of one sequence up to a prompt round of the engine), batches of 1 to 64 sequences of
unequal lengths, contexts up to 4096 tokens, the layer sizes of the presets in ``llmss_b200.utils.checkpoint`` and of the served
model shapes of ``bench.py`` (widths 2048 to 5120), bfloat16 and float16 (recurrent states and their inputs: 32-bit), 64-token
pages in scattered order.

``listed()`` names twelve cases, ``draw(rng)`` makes more of the same ranges, ``prepare`` / ``run`` make the inputs and do one pass,
``exact`` computes the same results in 64 bits with plain torch, ``work`` and ``tolerance`` say what a pass cannot do without and how
far two correct implementations lie apart.
"""
import math

import torch
import torch.nn.functional as F

from llmss_b200 import ops
from llmss_b200.engine.batch import BatchInput
from llmss_b200.engine.kv_cache import HybridCache
from llmss_b200.models.blocks import LatentAttention, RoutedExperts
from llmss_b200.models.decoder import ArchSpec, DecoderLM, LayerWeights
from llmss_b200.models.mixers import DeltaMixer, LayerCacheView

PAGE = 64
F32, F64 = torch.float32, torch.float64
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}
ACTS = {"none": ops.ACT_NONE, "gelu": ops.ACT_GELU_TANH, "silu": ops.ACT_SILU, "relu2": ops.ACT_RELU2}

# linear layers: (rows, columns, activation, rows without activation, gated, 32-bit result)
PROJECTIONS = {
    "gptj_in": (28672, 4096, "gelu", 12288, False, False),      # [k | v | q | up] of a GPT-J-6B block in one product
    "gptj_out": (4096, 20480, "none", 0, False, False),         # [out | down] of the same block
    "gptj_head": (50400, 4096, "none", 0, False, True),
    "qkv_2k": (6144, 2048, "none", 0, False, True),             # input product of a 2k-wide layer with a 32-bit residual stream
    "up_2k": (4096, 2048, "relu2", 0, False, False),
    "out_2k": (2048, 2048, "none", 0, False, True),
    "square_4k": (4096, 4096, "none", 0, False, False),         # attention output of a 7B-class layer
    "gate_up_4k": (22016, 4096, "silu", 0, True, False),        # Llama-2-7B gate / up
    "down_4k": (4096, 11008, "none", 0, False, False),
    "qkv_5k": (15360, 5120, "none", 0, False, False),           # Llama-2-13B q / k / v
    "gpt2_head": (50257, 1600, "none", 0, False, True),
}
# attention: query heads, key / value heads, head size
HEADS = {"gptj": (16, 16, 256), "llama": (32, 32, 128), "grouped": (32, 8, 128), "multi_query": (48, 1, 128), "small": (16, 16, 64)}
# linear recurrences: heads, query / key heads, key size, value size, kind of decay, read before the update
SCANS = {
    "wkv": (32, 32, 64, 64, "channel", True),                   # RWKV-style time mixing with a bonus
    "hgrn": (16, 16, 128, 128, "channel", False),               # gated linear recurrence
    "lightning": (16, 16, 128, 128, "head", False),             # one fixed decay per head
    "ssd": (32, 4, 128, 64, "token", False),                    # state-space layer, keys shared by groups of heads
}
# routed experts: width, experts, top, groups, kept groups, expert size, activation, gated, score
EXPERTS = {
    "bedovik": (2048, 16, 4, 4, 2, 1024, "relu2", False, "softmax"),
    "ninelix": (2048, 8, 2, 1, 1, 2048, "silu", True, "softmax"),
    "zenorax": (4096, 32, 4, 8, 4, 1536, "relu2", False, "sigmoid"),
}
# latent attention: width, heads, head size, latent size
LATENTS = {"2k": (2048, 16, 128, 128), "4k": (4096, 32, 128, 128)}
# gated delta rule: width, heads, key heads, head size
DELTAS = {"2k": (2048, 16, 8, 128), "4k": (4096, 32, 16, 128)}
VOCABS = (32000, 50257, 50400)


def listed():
    return [
        # the smallest product of a step: one to a few sequences, where the launch and the latency count
        {"name": "linear_few_tokens", "kind": "linear", "layer": "square_4k", "tokens": 3, "dtype": "float16"},
        # the input product of a GPT-J-6B decode step at the benchmark's batch
        {"name": "linear_decode", "kind": "linear", "layer": "gptj_in", "tokens": 64, "dtype": "bfloat16"},
        # gate and up of a prompt round, the largest products of a model
        {"name": "linear_prompt", "kind": "linear", "layer": "gate_up_4k", "tokens": 4096, "dtype": "bfloat16"},
        # a decode step over a batch of requests at different points of their answers
        {"name": "attention_decode", "kind": "attention", "heads": "gptj", "seqs": 64, "tokens": 1, "context": 1040, "dtype": "bfloat16"},
        # a prompt round of unequal prompts
        {"name": "attention_prompt", "kind": "attention", "heads": "llama", "seqs": 8, "tokens": 1024, "context": 0, "dtype": "bfloat16"},
        # a latent-attention block (projection, absorption, attention, output) of the same prompt round
        {"name": "latent_prompt", "kind": "latent", "size": "4k", "seqs": 8, "tokens": 1024, "context": 0, "dtype": "bfloat16"},
        # the recurrence of a prompt round, decays per channel
        {"name": "scan_prompt", "kind": "scan", "flavour": "wkv", "seqs": 8, "tokens": 1024, "context": 0},
        # the recurrence of a decode step: states read and written once
        {"name": "scan_decode", "kind": "scan", "flavour": "lightning", "seqs": 64, "tokens": 1, "context": 16},
        # a delta-rule layer (projection, convolution, recurrence, norm, output) of a prompt round
        {"name": "delta_prompt", "kind": "delta", "size": "2k", "seqs": 8, "tokens": 1024, "dtype": "bfloat16"},
        # router and experts of a prompt round
        {"name": "experts_prompt", "kind": "experts", "size": "bedovik", "tokens": 8192, "dtype": "bfloat16"},
        # the sampler at the end of a decode step, requests with different settings
        {"name": "sample_step", "kind": "sample", "rows": 64, "vocab": 50400},
        # a whole model: the logits of a prompt round of unequal prompts
        {"name": "model_prompt", "kind": "model", "width": 2048, "layers": 6, "seqs": 4, "tokens": 1001, "context": 0, "dtype": "bfloat16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, most):
    """Sequences and tokens of each, ``most`` tokens in all: single tokens over a context, or prompts."""
    if rng.random() < 0.4:
        return rng.randint(1, 64), 1
    total = _log(rng, 16, most)
    seqs = _log(rng, 1, min(32, max(1, total // 2)))
    return seqs, max(2, total // seqs)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "attention", "attention", "latent", "scan", "scan", "delta", "experts", "sample", "model"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float16"])
    if kind == "linear":
        layer = rng.choice(sorted(PROJECTIONS))
        n, k = PROJECTIONS[layer][:2]
        most = min(8192, int(4096 * 22016 * 4096 / (n * k)))
        if PROJECTIONS[layer][5] and layer.endswith("head"):
            most = min(most, 256)          # the head runs on one row per sequence
        return {"kind": kind, "layer": layer, "tokens": _log(rng, 1, most), "dtype": dtype}
    if kind == "attention":
        heads = rng.choice(sorted(HEADS))
        if rng.random() < 0.5:
            hq, hkv, d = HEADS[heads]
            seqs = _log(rng, 1, 64)
            most = int(min(4096, 64 * 1040 * 16 * 256 / (seqs * hkv * d)))
            return {"kind": kind, "heads": heads, "seqs": seqs, "tokens": 1, "context": _log(rng, 16, max(17, most)), "dtype": dtype}
        seqs = _log(rng, 1, 8)
        context = 0 if rng.random() < 0.6 else _log(rng, 16, 1024)
        return {"kind": kind, "heads": heads, "seqs": seqs, "tokens": max(2, _log(rng, 16, 4096 if not context else 2048) // seqs), "context": context,
                "dtype": dtype}
    if kind == "latent":
        seqs, tokens = _split(rng, 8192)
        seqs = min(seqs, 8192 // tokens)
        tokens = min(tokens, 2048)
        return {"kind": kind, "size": rng.choice(sorted(LATENTS)), "seqs": seqs, "tokens": tokens,
                "context": _log(rng, 16, 2048) if tokens == 1 else 0, "dtype": dtype}
    if kind == "scan":
        seqs, tokens = _split(rng, 8192)
        return {"kind": kind, "flavour": rng.choice(sorted(SCANS)), "seqs": seqs, "tokens": min(tokens, 4096),
                "context": 16 if tokens == 1 or rng.random() < 0.3 else 0}
    if kind == "delta":
        size = rng.choice(sorted(DELTAS))
        seqs, tokens = _split(rng, 8192 if size == "2k" else 4096)
        return {"kind": kind, "size": size, "seqs": seqs, "tokens": min(tokens, 1536), "dtype": dtype}
    if kind == "experts":
        size = rng.choice(sorted(EXPERTS))
        return {"kind": kind, "size": size, "tokens": _log(rng, 1, 8192 if size != "zenorax" else 2048), "dtype": dtype}
    if kind == "sample":
        return {"kind": kind, "rows": _log(rng, 1, 64), "vocab": rng.choice(VOCABS)}
    seqs = _log(rng, 1, 16)
    if rng.random() < 0.4:
        return {"kind": kind, "width": 2048, "layers": rng.randint(1, 6), "seqs": seqs, "tokens": 1, "context": _log(rng, 16, 1024), "dtype": dtype}
    return {"kind": kind, "width": 2048, "layers": rng.randint(1, 6), "seqs": seqs, "tokens": max(2, _log(rng, 16, 4000) // seqs), "context": 0,
            "dtype": dtype}


# ----------------------------------------------------------------------------- what the cases share
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0, mean=0.0, dtype=F32):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=F32) * std + mean).to(dtype)


def _weight(g, n, k, dtype):
    return _randn(g, n, k, std=k ** -0.5, dtype=dtype)


def _spread(mean, n):
    """n unequal lengths between half and one and a half times the mean (a function of the case alone, so its work is known)."""
    if mean <= 1:
        return [mean] * n
    return [max(1, round(mean * (0.5 + ((7 * i + 3) % n + 0.5) / n))) for i in range(n)]


def _lengths(case):
    """(new tokens, tokens in the cache) of every sequence."""
    n = case["seqs"]
    return _spread(case["tokens"], n), _spread(case.get("context", 0), n)


def _batch(case, seed, states=False):
    """The packed batch of a case and the number of cache blocks; a sequence's pages lie in scattered order."""
    new, ctx = _lengths(case)
    need = [-(-(a + b) // PAGE) for a, b in zip(new, ctx)]
    blocks = 1 + sum(need)
    order = (torch.randperm(blocks - 1, generator=torch.Generator().manual_seed(seed)) + 1).tolist()
    tables, at = [], 0
    for n in need:
        tables.append(order[at:at + n])
        at += n
    toks = torch.randint(0, 32000, (sum(new),), generator=torch.Generator().manual_seed(seed + 1)).tolist()
    lists, at = [], 0
    for n in new:
        lists.append(toks[at:at + n])
        at += n
    return BatchInput.build(lists, ctx, tables, PAGE, "cuda", state_slots=list(range(len(new))) if states else None), blocks


def _act64(x, act):
    if act == "gelu":
        return F.gelu(x, approximate="tanh")
    if act == "silu":
        return F.silu(x)
    return F.relu(x).square() if act == "relu2" else x


def _causal64(q, k, v, scale):
    """Softmax attention in 64 bits: q [ql, hq, d] are the last ql positions of k [L, hkv, d], v [L, hkv, dv]."""
    ql, hq, L, hkv = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    seen = torch.arange(L, device="cuda")[None, :] <= torch.arange(L - ql, L, device="cuda")[:, None]
    out = []
    for h in range(hkv):
        g = hq // hkv
        s = torch.einsum("qhd,kd->hqk", q[:, h * g:(h + 1) * g], k[:, h]) * scale
        out.append(torch.einsum("hqk,kd->qhd", torch.softmax(s.masked_fill(~seen, -math.inf), -1), v[:, h]))
    return torch.cat(out, 1)


def _pairs(case):
    """Query / key pairs that causal attention looks at."""
    return sum(n * c + n * (n + 1) // 2 for n, c in zip(*_lengths(case)))


# ----------------------------------------------------------------------------- linear layers
def _linear_inputs(case, seed):
    n, k, act, start, gated, f32 = PROJECTIONS[case["layer"]]
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    return {"x": _randn(g, case["tokens"], k, dtype=dt), "w": _weight(g, n, k, dt), "b": _randn(g, n, std=0.1, dtype=dt)}


def _linear_run(s):
    n, k, act, start, gated, f32 = PROJECTIONS[s["case"]["layer"]]
    return ops.linear(s["x"], s["w"], s["b"], act=ACTS[act], gated=gated, act_start=start, out_dtype=F32 if f32 else None)


def _linear_exact(case, seed):
    n, k, act, start, gated, f32 = PROJECTIONS[case["layer"]]
    s = _linear_inputs(case, seed)
    y = s["x"].double() @ s["w"].double().t() + s["b"].double()
    if gated:
        return _act64(y[:, 0::2], act) * y[:, 1::2]
    return torch.cat([y[:, :start], _act64(y[:, start:], act)], 1)


def _linear_work(case):
    n, k, act, start, gated, f32 = PROJECTIONS[case["layer"]]
    t = case["tokens"]
    return {"bytes": 2 * (t * k + n * k + n) + t * (n // 2 if gated else n) * (4 if f32 else 2), "flops": 2 * t * n * k}


# ----------------------------------------------------------------------------- multi-head attention over pages
def _attention_inputs(case, seed):
    hq, hkv, d = HEADS[case["heads"]]
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    batch, blocks = _batch(case, seed)
    T = batch.tokens.numel()
    s = {"batch": batch, "qkv": _randn(g, T, (hq + 2 * hkv) * d, dtype=dt),
         "k": _randn(g, blocks, hkv, PAGE, d, dtype=dt), "v": _randn(g, blocks, hkv, PAGE, d, dtype=dt)}
    # this step's keys and values are in their pages already, as the layer leaves them
    ops.rope_kv_write(s["qkv"], batch.positions, batch.slot_mapping, s["k"], s["v"], hq, hkv, d, d, ops.ROPE_NEOX, 10000.0, 0, hq * d,
                      (hq + hkv) * d)
    s["out"] = torch.zeros(T, hq * d, dtype=dt, device="cuda")
    return s


def _attention_run(s):
    hq, hkv, d = HEADS[s["case"]["heads"]]
    return ops.attention(s["qkv"], s["out"], s["batch"], s["k"], s["v"], hq, hkv, d, d ** -0.5, 0, hq * d, (hq + hkv) * d)


def _attention_exact(case, seed):
    hq, hkv, d = HEADS[case["heads"]]
    s = _attention_inputs(case, seed)
    out, at = [], 0
    for i, (n, c) in enumerate(zip(*_lengths(case))):
        pages = s["batch"].block_tables[i, :-(-(n + c) // PAGE)].long()
        k, v = (s[x][pages].transpose(1, 2).reshape(-1, hkv, d)[:n + c].double() for x in ("k", "v"))
        out.append(_causal64(s["qkv"][at:at + n, :hq * d].reshape(n, hq, d).double(), k, v, d ** -0.5).reshape(n, hq * d))
        at += n
    return torch.cat(out)


def _attention_work(case):
    hq, hkv, d = HEADS[case["heads"]]
    new, ctx = _lengths(case)
    return {"bytes": 2 * d * (2 * hq * sum(new) + 2 * hkv * (sum(new) + sum(ctx))), "flops": 4 * hq * d * _pairs(case)}


# ----------------------------------------------------------------------------- latent attention
def _latent_inputs(case, seed):
    W, H, d, R = LATENTS[case["size"]]
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    batch, blocks = _batch(case, seed)
    s = {"batch": batch, "h": _randn(g, batch.tokens.numel(), W, dtype=dt), "cache": _randn(g, blocks, PAGE, R, dtype=dt)}
    s["w"] = {"q": _weight(g, H * d, W, dt), "dkv": _weight(g, R, W, dt), "g": _weight(g, H, W, dt), "norm": _randn(g, R, std=0.05, mean=1.0, dtype=dt),
              "uk": _weight(g, H * d, R, dt), "uv": _weight(g, H * d, R, dt), "o": _weight(g, W, H * d, dt)}
    return s


def _latent_prepare(case, seed):
    W, H, d, R = LATENTS[case["size"]]
    s = _latent_inputs(case, seed)
    block, w = LatentAttention(H, d, d, R, d ** -0.5, True, 1e-6), s["w"]
    block.w_q, block.w_dkv, block.w_g, block.norm_w, block.w_uk, block.w_uv, block.w_o = (
        w["q"], w["dkv"], w["g"], w["norm"], w["uk"], w["uv"], w["o"])
    s["w_in"] = block.in_rows()
    block.bind(0)
    s["block"] = block
    del s["w"]
    return s


def _latent_run(s):
    y = ops.linear(s["h"], s["w_in"], out_dtype=F32)
    return s["block"].forward(y, s["batch"], s["cache"], s["h"].dtype)


def _latent_exact(case, seed):
    W, H, d, R = LATENTS[case["size"]]
    s = _latent_inputs(case, seed)
    w, h = {n: t.double() for n, t in s["w"].items()}, s["h"].double()
    c = h @ w["dkv"].t()
    c = c * torch.rsqrt(c.square().mean(-1, keepdim=True) + 1e-6) * w["norm"]
    q, gate = (h @ w["q"].t()).view(-1, H, d), torch.sigmoid(h @ w["g"].t())
    out, at = [], 0
    for i, (n, ctx) in enumerate(zip(*_lengths(case))):
        pages = s["batch"].block_tables[i, :-(-(n + ctx) // PAGE)].long()
        rows = torch.cat([s["cache"][pages].reshape(-1, R)[:ctx].double(), c[at:at + n]])
        k, v = (rows @ w["uk"].t()).view(-1, H, d), (rows @ w["uv"].t()).view(-1, H, d)
        o = _causal64(q[at:at + n], k, v, d ** -0.5) * gate[at:at + n, :, None]
        out.append(o.reshape(n, H * d) @ w["o"].t())
        at += n
    return torch.cat(out)


def _latent_work(case):
    W, H, d, R = LATENTS[case["size"]]
    new, ctx = _lengths(case)
    T = sum(new)
    weights = W * (H * d + R + H) + 2 * H * d * R + W * H * d
    return {"bytes": 2 * (weights + T * W + R * (T + sum(ctx))) + 4 * T * W, "flops": 2 * T * weights + 4 * H * R * _pairs(case)}


# ----------------------------------------------------------------------------- gated linear recurrences
def _scan_inputs(case, seed):
    """Inputs of the context (if any) and of the step: dicts of q, k, v, decay and the options."""
    H, G, dk, dv, kind, before = SCANS[case["flavour"]]
    g = _rng(seed)
    parts = []
    for lens in (_lengths(case)[1], _lengths(case)[0]):
        T = sum(lens)
        if T == 0:
            parts.append(None)
            continue
        p = {"lens": lens, "q": _randn(g, T, G * dk), "k": _randn(g, T, G * dk), "v": _randn(g, T, H * dv)}
        if case["flavour"] == "hgrn":          # the key is what the forget gate leaves open
            f = torch.sigmoid(_randn(g, T, H * dk, mean=1.0))
            p["q"], p["k"], p["decay"] = F.silu(p["q"]), 1 - f, torch.log(f)
        elif kind == "channel":
            p["decay"] = -torch.exp(_randn(g, T, H * dk, mean=-1.0))
        elif kind == "token":
            dt = F.softplus(_randn(g, T, H, mean=-1.0))
            p["decay"], p["v_scale"] = -1.5 * dt, dt
        else:
            p["q"], p["k"], p["v"] = F.silu(p["q"]), F.silu(p["k"]), F.silu(p["v"])
        parts.append(p)
    opts = {"bonus": _randn(g, H, dk, std=0.5) if before else None}
    if kind == "head":
        opts["decay"] = torch.tensor([1.0 - 2.0 ** -(1.0 + 6.0 * h / (H - 1)) for h in range(H)], dtype=F32, device="cuda")
    return parts, opts


_DECAYS = {"head": ops.DECAY_HEAD, "token": ops.DECAY_TOKEN_HEAD, "channel": ops.DECAY_TOKEN_CHANNEL}


def _scan_call(case, p, opts, batch, state):
    H, G, dk, dv, kind, before = SCANS[case["flavour"]]
    return ops.linear_scan(p["q"], p["k"], p["v"], p.get("decay", opts.get("decay")), _DECAYS[kind], batch, state, H, G, dk, dv, bonus=opts["bonus"],
                           v_scale=p.get("v_scale"), read_before=before)


def _scan_prepare(case, seed):
    H, G, dk, dv, kind, before = SCANS[case["flavour"]]
    (first, step), opts = _scan_inputs(case, seed)
    state = torch.zeros(case["seqs"], H, dk, dv, dtype=F32, device="cuda")
    if first is not None:       # the states that the sequences' earlier tokens have left
        before_batch = _batch({"seqs": case["seqs"], "tokens": case["context"]}, seed, states=True)[0]
        _scan_call(case, first, opts, before_batch, state)
    return {"p": step, "opts": opts, "state": state, "batch": _batch(case, seed, states=True)[0]}


def _scan_run(s):
    return {"out": _scan_call(s["case"], s["p"], s["opts"], s["batch"], s["state"]), "state": s["state"]}


def _scan_exact(case, seed):
    H, G, dk, dv, kind, before = SCANS[case["flavour"]]
    parts, opts = _scan_inputs(case, seed)
    n, bonus = case["seqs"], None if opts["bonus"] is None else opts["bonus"].double()
    S = torch.zeros(n, H, dk, dv, dtype=F64, device="cuda")
    for p in parts:
        if p is None:
            continue
        starts, lens = torch.tensor([0] + p["lens"][:-1]).cumsum(0), torch.tensor(p["lens"])
        out = torch.zeros(sum(p["lens"]), H, dv, dtype=F64, device="cuda")
        q, k = (p[x].double().view(-1, G, dk).repeat_interleave(H // G, 1) for x in ("q", "k"))
        v = p["v"].double().view(-1, H, dv)
        if "v_scale" in p:
            v = v * p["v_scale"].double()[:, :, None]
        if kind == "head":
            a = opts["decay"].double()[None, :, None]
        else:
            a = torch.exp(p["decay"].double()).view(-1, H, dk if kind == "channel" else 1)
        for t in range(max(p["lens"])):
            on = torch.nonzero(lens > t).flatten()
            rows = (starts[on] + t).cuda()
            on = on.cuda()
            kv = k[rows][..., None] * v[rows][:, :, None, :]
            old = S[on]
            new = (a if kind == "head" else a[rows])[..., None] * old + kv
            read = old + bonus[None, :, :, None] * kv if before else new
            out[rows] = torch.einsum("nhkv,nhk->nhv", read, q[rows])
            S[on] = new
    return {"out": out.reshape(-1, H * dv), "state": None}


def _scan_work(case):
    H, G, dk, dv, kind, before = SCANS[case["flavour"]]
    T = sum(_lengths(case)[0])
    decay = {"head": 0, "token": H, "channel": H * dk}[kind]
    state = case["seqs"] * H * dk * dv * (2 if case["context"] else 1)
    return {"bytes": 4 * (T * (2 * G * dk + 2 * H * dv + decay) + state), "flops": 6 * T * H * dk * dv}


# ----------------------------------------------------------------------------- gated delta rule layer
def _delta_inputs(case, seed):
    W, H, G, d = DELTAS[case["size"]]
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    T = sum(_lengths(case)[0])
    w = {"q": _weight(g, G * d, W, dt), "k": _weight(g, G * d, W, dt), "v": _weight(g, H * d, W, dt), "g": _weight(g, H * d, W, dt),
         "a": _weight(g, H, W, dt), "b": _weight(g, H, W, dt), "o": _weight(g, W, H * d, dt)}
    for x, n in (("cq", G * d), ("ck", G * d), ("cv", H * d)):
        w[x] = _randn(g, n, 4, std=0.5)
    w["dt_bias"], w["a_log"], w["norm"] = _randn(g, H, mean=-1.0), _randn(g, H, std=0.7), _randn(g, d, std=0.05, mean=1.0)
    return {"h": _randn(g, T, W, dtype=dt)}, w


def _delta_prepare(case, seed):
    W, H, G, d = DELTAS[case["size"]]
    s, w = _delta_inputs(case, seed)
    mixer = DeltaMixer(W, H, G, d, d, 4, 1e-6)
    mixer.set_weights(w["q"], w["k"], w["v"], w["cq"], w["ck"], w["cv"], w["b"], w["a"], w["dt_bias"], w["a_log"], w["norm"], w["g"], w["o"])
    cache = HybridCache({}, {(0, n): v for n, v in mixer.state_shapes().items()}, 1, PAGE, case["seqs"], DTYPES[case["dtype"]], "cuda")
    s.update(mixer=mixer, lc=LayerCacheView(cache, 0), batch=_batch(case, seed, states=True)[0])
    return s


def _delta_run(s):
    y = s["mixer"].forward(s["h"], s["batch"], s["lc"], s["h"].dtype)
    return {"out": y, "S": s["lc"].state("S"), "conv": s["lc"].state("conv")}


def _delta_exact(case, seed):
    W, H, G, d = DELTAS[case["size"]]
    s, w = _delta_inputs(case, seed)
    w, h = {n: t.double() for n, t in w.items()}, s["h"].double()
    lens = _lengths(case)[0]
    qkv = torch.cat([h @ w[x].t() for x in "qkv"], 1)
    cw = torch.cat([w["cq"], w["ck"], w["cv"]])
    conv, at = [], 0
    for n in lens:
        u = F.pad(qkv[at:at + n], (0, 0, 3, 0))
        conv.append(sum(u[j:j + n] * cw[:, j] for j in range(4)))
        at += n
    qkv = F.silu(torch.cat(conv))
    q, k, v = qkv[:, :G * d].view(-1, G, d), qkv[:, G * d:2 * G * d].view(-1, G, d), qkv[:, 2 * G * d:].view(-1, H, d)
    q, k = (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (q * d ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(h @ w["b"].t())
    a = torch.exp(-torch.exp(w["a_log"]) * F.softplus(h @ w["a"].t() + w["dt_bias"]))
    o = torch.zeros_like(v)
    S = torch.zeros(len(lens), H, d, d, dtype=F64, device="cuda")
    starts, lens_t = torch.tensor([0] + lens[:-1]).cumsum(0), torch.tensor(lens)
    for t in range(max(lens)):
        on = torch.nonzero(lens_t > t).flatten()
        r, on = (starts[on] + t).cuda(), on.cuda()
        St = S[on] * a[r][..., None, None]
        u = beta[r][..., None] * (v[r] - torch.einsum("nhkv,nhk->nhv", St, k[r]))
        St = St + k[r][..., None] * u[:, :, None, :]
        S[on] = St
        o[r] = torch.einsum("nhkv,nhk->nhv", St, q[r])
    o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + 1e-6) * w["norm"]
    y = (o.reshape(-1, H * d) * F.silu(h @ w["g"].t())) @ w["o"].t()
    return {"out": y, "S": None, "conv": None}


def _delta_work(case):
    W, H, G, d = DELTAS[case["size"]]
    T = sum(_lengths(case)[0])
    weights = W * (2 * G * d + 2 * H * d + 2 * H) + W * H * d
    return {"bytes": 2 * (weights + T * W) + 4 * (T * W + case["seqs"] * H * d * d), "flops": 2 * T * weights + 8 * T * H * d * d}


# ----------------------------------------------------------------------------- routed experts
def _experts_inputs(case, seed):
    W, E, top, groups, keep, ff, act, gated, score = EXPERTS[case["size"]]
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    rows = 2 * ff if gated else ff
    return {"h": _randn(g, case["tokens"], W, dtype=dt), "router": _randn(g, E, W, std=2 * W ** -0.5, dtype=dt),
            "up": _randn(g, E, rows, W, std=W ** -0.5, dtype=dt), "down": _randn(g, W, E * ff, std=ff ** -0.5, dtype=dt)}


def _experts_prepare(case, seed):
    W, E, top, groups, keep, ff, act, gated, score = EXPERTS[case["size"]]
    s = _experts_inputs(case, seed)
    block = RoutedExperts(E, top, groups, keep, 2.0, ff, act=ACTS[act], gated=gated, score=score)
    block.w_router, block.w_up, block.w_down = s["router"], s["up"], s["down"]
    return {"h": s["h"], "block": block}


def _experts_run(s):
    return s["block"].forward(s["h"])


def _experts_exact(case, seed):
    W, E, top, groups, keep, ff, act, gated, score = EXPERTS[case["size"]]
    s = _experts_inputs(case, seed)
    h = s["h"].double()
    z = h @ s["router"].double().t()
    p = torch.softmax(z, -1) if score == "softmax" else torch.sigmoid(z)
    best = p.view(-1, groups, E // groups).amax(-1).topk(keep, -1).indices
    open_ = torch.zeros(p.shape[0], groups, dtype=torch.bool, device="cuda").scatter_(1, best, True).repeat_interleave(E // groups, 1)
    wt, ids = p.masked_fill(~open_, -math.inf).topk(top, -1)
    wt = 2.0 * wt / wt.sum(-1, keepdim=True)
    y = torch.zeros_like(h)
    for e in range(E):
        t, j = torch.nonzero(ids == e, as_tuple=True)
        a = h[t] @ s["up"][e].double().t()
        a = _act64(a[:, 0::2], act) * a[:, 1::2] if gated else _act64(a, act)
        y.index_add_(0, t, wt[t, j][:, None] * (a @ s["down"][:, e * ff:(e + 1) * ff].double().t()))
    return y


def _experts_work(case):
    W, E, top, groups, keep, ff, act, gated, score = EXPERTS[case["size"]]
    T, one = case["tokens"], W * ff * (3 if gated else 2)
    return {"bytes": 2 * (W * E + min(E, T * top) * one + T * W) + 4 * T * W, "flops": 2 * T * (W * E + top * one)}


# ----------------------------------------------------------------------------- the sampler
def _sample_prepare(case, seed):
    g, B = _rng(seed), case["rows"]
    # requests of four kinds: greedy, nucleus, few candidates, the whole distribution
    kind = torch.arange(B, device="cuda") % 4
    i32 = torch.int32
    return {"logits": _randn(g, B, case["vocab"], std=2.5), "greedy": (kind == 0).to(i32),
            "temperature": torch.where(kind == 2, 0.7, 1.0).to(F32), "top_k": torch.where(kind == 2, 50, 0).to(i32),
            "top_p": torch.where(kind == 1, 0.9, 1.0).to(F32),
            "rng": torch.randint(0, 1 << 30, (B, 2), generator=g, device="cuda").to(i32)}


def _sample_run(s):
    tokens = ops.sample(s["logits"], s["greedy"], s["temperature"], s["top_k"], s["top_p"], s["rng"])
    return {"tokens": tokens, "rng": s["rng"]}


def _sample_work(case):
    return {"bytes": case["rows"] * (4 * case["vocab"] + 32), "flops": case["rows"] * case["vocab"]}


# ----------------------------------------------------------------------------- a whole model (parallel attention and feed-forward)
def _model_spec(case):
    W = case["width"]
    return ArchSpec("gptj", W, case["layers"], W // 128, W // 128, 128, 2 * W, 32000, 4096, rope=ops.ROPE_GPTJ, rotary_dim=64,
                    act=ops.ACT_GELU_TANH, parallel_residual=True, head_bias=True)


def _model_weights(case, seed):
    W, Ff, V = case["width"], 2 * case["width"], 32000
    g, dt = _rng(seed), DTYPES[case["dtype"]]
    layers = []
    for _ in range(case["layers"]):
        layers.append({"ln_w": _randn(g, W, std=0.05, mean=1.0, dtype=dt), "ln_b": _randn(g, W, std=0.05, dtype=dt), "qkv": _weight(g, 3 * W, W, dt),
                       "o": _weight(g, W, W, dt), "up": _weight(g, Ff, W, dt), "b_up": _randn(g, Ff, std=0.1, dtype=dt),
                       "down": _weight(g, W, Ff, dt), "b_down": _randn(g, W, std=0.1, dtype=dt)})
    top = {"wte": _randn(g, V, W, dtype=dt), "ln_w": _randn(g, W, std=0.05, mean=1.0, dtype=dt), "ln_b": _randn(g, W, std=0.05, dtype=dt),
           "head": _weight(g, V, W, dt), "b_head": _randn(g, V, std=0.1, dtype=dt)}
    # keys and values of the tokens before this step
    blocks = _batch(case, seed)[1]
    top["pages"] = _randn(g, case["layers"], 2, blocks, W // 128, PAGE, 128, dtype=dt) if case["context"] else None
    return layers, top


def _model_prepare(case, seed):
    spec, dt = _model_spec(case), DTYPES[case["dtype"]]
    layers, top = _model_weights(case, seed)
    m = DecoderLM(spec, None, torch.device("cuda"), dt)
    for w in layers:
        L = LayerWeights()
        L.ln1_w, L.ln1_b, L.wqkv, L.wo = w["ln_w"], w["ln_b"], w["qkv"], w["o"]
        L.wup, L.bup, L.wdown, L.bdown = w["up"], w["b_up"], w["down"], w["b_down"]
        m.layers.append(L)
    m.wte, m.lnf_w, m.lnf_b, m.w_head, m.b_head = top["wte"], top["ln_w"], top["ln_b"], top["head"], top["b_head"]
    m.finalize()
    batch, blocks = _batch(case, seed)
    kv = m.make_cache(blocks, PAGE)
    if top["pages"] is not None:
        kv.data.copy_(top["pages"])
    return {"model": m, "batch": batch, "kv": kv}


@torch.no_grad()
def _model_run(s):
    return s["model"](s["batch"], s["kv"])


def _model_exact(case, seed):
    W, H = case["width"], case["width"] // 128
    layers, top = _model_weights(case, seed)
    batch = _batch(case, seed)[0]
    new, ctx = _lengths(case)
    angle = batch.positions.double()[:, None] * 10000.0 ** (-torch.arange(0, 64, 2, device="cuda", dtype=F64) / 64)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def turn(x):        # pairs (2i, 2i + 1) of the first 64 channels of every head
        a, b = x[..., 0:64:2], x[..., 1:64:2]
        return torch.cat([torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2), x[..., 64:]], -1)

    def norm(x, w):
        return F.layer_norm(x, (W,), w["ln_w"].double(), w["ln_b"].double(), 1e-5)

    x = top["wte"][batch.tokens.long()].double()
    for li, w in enumerate(layers):
        h = norm(x, w)
        q, k, v = ((h @ t.double().t()).view(-1, H, 128) for t in w["qkv"].split(W))
        q, k = turn(q), turn(k)
        out, at = [], 0
        for i, (n, c) in enumerate(zip(new, ctx)):
            ks, vs = k[at:at + n], v[at:at + n]
            if c:
                old = top["pages"][li][:, batch.block_tables[i, :-(-c // PAGE)].long()].double().transpose(2, 3).reshape(2, -1, H, 128)[:, :c]
                ks, vs = torch.cat([old[0], ks]), torch.cat([old[1], vs])
            out.append(_causal64(q[at:at + n], ks, vs, 128 ** -0.5).reshape(n, W))
            at += n
        up = F.gelu(h @ w["up"].double().t() + w["b_up"].double(), approximate="tanh")
        x = x + torch.cat(out) @ w["o"].double().t() + up @ w["down"].double().t() + w["b_down"].double()
    return norm(x[batch.last_idx], top) @ top["head"].double().t() + top["b_head"].double()


def _model_work(case):
    W, L, V = case["width"], case["layers"], 32000
    new, ctx = _lengths(case)
    T, one = sum(new), 8 * W * W
    return {"bytes": 2 * (L * one + V * W + T * W + 2 * L * W * (T + sum(ctx))) + 4 * case["seqs"] * V,
            "flops": 2 * T * L * one + 4 * L * W * _pairs(case) + 2 * case["seqs"] * V * W}


# ----------------------------------------------------------------------------- the interface
_KINDS = {
    "linear": (_linear_inputs, _linear_run, _linear_exact, _linear_work),
    "attention": (_attention_inputs, _attention_run, _attention_exact, _attention_work),
    "latent": (_latent_prepare, _latent_run, _latent_exact, _latent_work),
    "scan": (_scan_prepare, _scan_run, _scan_exact, _scan_work),
    "delta": (_delta_prepare, _delta_run, _delta_exact, _delta_work),
    "experts": (_experts_prepare, _experts_run, _experts_exact, _experts_work),
    "sample": (_sample_prepare, _sample_run, None, _sample_work),
    "model": (_model_prepare, _model_run, _model_exact, _model_work),
}


def prepare(case, seed):
    state = _KINDS[case["kind"]][0](case, seed)
    state["case"] = case
    return state


def run(state):
    return _KINDS[state["case"]["kind"]][1](state)


def exact(case, seed):
    fn = _KINDS[case["kind"]][2]
    return None if fn is None else fn(case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"                       # token ids and counters
    if kind == "scan":
        return {"rel": 1e-5}                 # 32-bit sums over up to 4096 tokens
    # 16-bit results of 32-bit sums (linear, attention); a model's and a block's 16-bit values in between are rounded once per stage
    rel = {"model": 2e-2, "linear": 5e-3, "attention": 8e-3}.get(kind, 1e-2)
    return {"rel": rel * (0.125 if case["dtype"] == "float16" else 1.0)}

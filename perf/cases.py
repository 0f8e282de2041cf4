"""What this engine is measured on: passes of ordinary use through its public entry points.

A pass opens requests, runs their prompts and then their following tokens through ``Engine.step`` as the
scheduler would cut them (every request that is past its prompt brings one token, what is left of the
step's token budget goes to prompts, first come first served), keeps the logits of every position that a
next token would be picked from, and closes the requests.  The following tokens are given, as in a
replay: a token picked from logits that are equal but for rounding may differ, and everything behind it
then would.  One case goes through ``Generator.generate`` instead, where the picks are the engine's own.

Sizes are those of this repository's configurations, tests and benchmark.
"""
from __future__ import annotations

import functools
import math
import zlib

import torch

from gibbs_b200 import Engine, Generator, Lfm2Config, SamplingParams, StepEntry, parse_config
from gibbs_b200.parts.model import build_model
from gibbs_b200.weights import TensorDict, expected_tensors

F64 = torch.float64
PAGE = 16


# ---------------------------------------------------------------------------------------------------
# model sizes
# ---------------------------------------------------------------------------------------------------

def _lfm2(**sizes) -> dict:
    return dict(dict(
        architectures=["Lfm2ForCausalLM"], model_type="lfm2", hidden_size=2048, num_hidden_layers=16, num_attention_heads=32,
        num_key_value_heads=8, head_dim=64, vocab_size=65536, intermediate_size=12288, block_auto_adjust_ff_dim=True,
        block_ffn_dim_multiplier=1.0, block_multiple_of=256, conv_L_cache=3, conv_bias=False,
        full_attn_idxs=[2, 5, 8, 10, 12, 14], rope_theta=1000000.0, norm_eps=1e-5, tie_embedding=True,
        max_position_embeddings=8192), **sizes)


def _potivik(wide: bool) -> dict:
    d, vocab, side = (2048, 65536, 256) if wide else (1024, 32768, 128)
    ssm = {"heads": d // 32, "vdim": 64, "state": 128 if wide else 64, "groups": d // 256, "conv": 4, "norm_groups": d // 256}
    dim = 128 if wide else 64
    att = {"heads": 16 if wide else 8, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": 512 if wide else 256,
           "scale": (1.5 * dim) ** -0.5, "mask": {"size": 1024 if wide else 512}, "rot": {"base": 500000.0, "dims": dim // 2}}
    dense = {"kind": "dense", "ff": 4 * d, "limit": 7.0}
    moe = {"kind": "moe", "router": {"experts": 32, "top": 4} if wide else {"experts": 16, "top": 2},
           "expert": {"ff": d // 2, "limit": 7.0}, "shared": {"ff": d, "limit": 7.0}}
    layers = [{"type": "mamba2", "mixer": ssm, "mlp": dense}, {"type": "latent_attention", "mixer": att, "mlp": moe}] * 4
    return {"architecture": "Potivik", "vocab": vocab, "width": d, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "token_side": {"dim": side}, "layers": layers}


def _petelix(wide: bool) -> dict:
    d, vocab = (2048, 65536) if wide else (1024, 32768)
    att = {"heads": d // 64, "kv_heads": d // 256, "dim": 64, "vdim": 64 if wide else 32, "scale": 0.125, "softcap": 30.0,
           "mask": {"size": d // 2}, "rot": {"base": 500000.0, "dims": 32}}
    router = {"experts": 30 if wide else 14, "identity": 2, "top": 4 if wide else 2, "groups": {"count": 4, "keep": 2}}
    moe = {"kind": "moe", "router": router, "expert": {"ff": 1024}}
    layers = [{"type": "attention", "mixer": dict(att, **({"kv_from": i - 1} if i % 2 else {})), "mlp": moe} for i in range(8)]
    return {"architecture": "Petelix", "vocab": vocab, "width": d, "norm": {"eps": 1e-6}, "embedding": {"scale": 8.0},
            "layers": layers}


def _sisadra(wide: bool) -> dict:
    d, vocab, dim = (2048, 65536, 128) if wide else (1024, 32768, 64)
    rule = {"heads": 16, "kv_heads": 8, "dim": dim, "vdim": dim, "conv": 4, "decay_rank": dim, "gate_rank": dim}
    att = {"heads": d // 128, "kv_heads": d // 512, "dim": 64, "vdim": 128, "scale": 0.125, "diff": 0.3, "mask": {"size": d // 2},
           "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    lat = {"heads": d // 128, "dim": dim, "vdim": dim, "kv_rank": d // 4, "scale": dim ** -0.5}
    mixers = {"channel_delta": rule, "attention": att, "latent_attention": lat}
    return {"architecture": "Sisadra", "vocab": vocab, "width": d, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "embedding": {"scale": 8.0, "bigram": {"buckets": 65521, "mul_prev": 1000003, "mul_cur": 999983}},
            "layers": [{"type": k, "mixer": mixers[k], "mlp": {"kind": "dense", "ff": 4 * d}}
                       for k in ["channel_delta", "attention", "channel_delta", "latent_attention"] * 2]}


def _guvetar(wide: bool) -> dict:
    d, vocab = (2048, 65536) if wide else (1024, 32768)
    scan = {"inner": 2 * d, "state": 16, "dt_rank": d // 16, "conv": 4}
    memory = {"heads": 16 if wide else 8, "dim": 128 if wide else 64, "vdim": 128, "gate_cap": 15.0}
    left = {"heads": d // 128, "kv_heads": d // 512, "dim": 64, "vdim": 64, "scale": 0.125, "q_temp": {"coef": 0.5, "every": 1024}}
    right = {"heads": 8, "dim": d // 16, "vdim": d // 16}
    both = {"left": left, "right": right, "left_scale": 0.7, "right_scale": 0.8}
    four = [("mamba1", scan), ("parallel", both), ("mamba1", scan), ("mlstm", memory)]
    return {"architecture": "Guvetar", "vocab": vocab, "width": d, "streams": 4, "norm": {"eps": 1e-6},
            "layers": [{"type": k, "mixer": m, "mlp": {"kind": "dense", "ff": 4 * d}} for k, m in four * 2]}


MODELS = {
    "lfm2-tiny-a": _lfm2(hidden_size=64, num_hidden_layers=4, num_attention_heads=4, num_key_value_heads=2, head_dim=16,
                         vocab_size=512, intermediate_size=192, block_auto_adjust_ff_dim=False, full_attn_idxs=[1, 3],
                         rope_theta=10000.0, max_position_embeddings=64),
    "lfm2-tiny-b": _lfm2(hidden_size=96, num_hidden_layers=6, num_attention_heads=3, num_key_value_heads=1, head_dim=32,
                         vocab_size=1000, intermediate_size=384, block_multiple_of=64, conv_L_cache=4, conv_bias=True,
                         attention_bias=True, full_attn_idxs=[0, 2, 5], norm_eps=1e-6, tie_embedding=False,
                         max_position_embeddings=512),
    "lfm2-700m": _lfm2(hidden_size=1536, num_attention_heads=24, intermediate_size=10240),
    "lfm2-1.2b": _lfm2(),
    "lfm2-2.6b": _lfm2(num_hidden_layers=30, full_attn_idxs=[2, 6, 10, 14, 18, 22, 25, 28], intermediate_size=10752),
    "potivik-1k": _potivik(False), "potivik-2k": _potivik(True),
    "petelix-1k": _petelix(False), "petelix-2k": _petelix(True),
    "sisadra-1k": _sisadra(False), "sisadra-2k": _sisadra(True),
    "guvetar-1k": _guvetar(False), "guvetar-2k": _guvetar(True),
}


def _config(model: str):
    raw = MODELS[model]
    return Lfm2Config.from_dict(raw) if "hidden_size" in raw else parse_config(raw)


@functools.lru_cache(maxsize=None)
def _shapes(model: str) -> tuple:
    """((tensor name, shape, whether it is a matrix), ...) of a checkpoint."""
    return tuple((n, tuple(d.shapes[-1]), d.role == "matrix") for n, d in expected_tensors(_config(model).plan()).items())


# ---------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------

def _case(name, model, requests, shortest, longest, new, budget=16384, dtype="bfloat16", generate=False) -> dict:
    """``requests`` prompts of ``shortest`` to ``longest`` tokens, ``new`` tokens behind each, at most
    ``budget`` tokens a step."""
    return {"name": name, "model": model, "dtype": dtype, "requests": requests, "shortest": shortest, "longest": longest,
            "new": new, "budget": budget, "generate": generate}


def listed() -> list:
    return [
        # The smallest calls: three short prompts and a dozen greedy tokens each on a model of a few hundred thousand
        # weights, all 32-bit, through the generator with its scheduler and sampler; every kernel is a launch, not work.
        _case("tiny-generate", "lfm2-tiny-b", 3, 1, 40, 12, budget=2048, dtype="float32", generate=True),
        # One user in a chat: a prompt of a paragraph and an answer, token by token; bound by the weights' stream.
        _case("chat-1", "lfm2-1.2b", 1, 93, 93, 40),
        # The benchmark's batch: eight users with prompts from a question to a long document.
        _case("chat-8", "lfm2-1.2b", 8, 160, 2048, 48),
        # A busy server: 64 requests with prompts of very different length, decoded together.
        _case("chat-64", "lfm2-1.2b", 64, 17, 400, 32),
        # A document read in one step for one answer (scoring, classification): the benchmark's prompt.
        _case("prompt-2048", "lfm2-1.2b", 1, 2048, 2048, 0),
        # Continuous batching with chunked prompts: portions of at most 512 tokens a step, decoded tokens among them.
        _case("mixed-512", "lfm2-700m", 16, 16, 2048, 24, budget=512),
        # The long context: a prompt of 8,000 tokens and the first tokens behind it.
        _case("long-8000", "lfm2-2.6b", 1, 8000, 8000, 16),
        # The 32-bit path in earnest: a model's exact twin, short prompts and a few tokens each.
        _case("float32-700m", "lfm2-700m", 2, 75, 150, 8, dtype="float32"),
        # State-space scan, windowed latent attention, experts: two requests, one twice as long as the other.
        _case("potivik-2k", "potivik-2k", 2, 333, 1801, 12),
        # Grouped attention with a sink, shared keys and values, routed experts.
        _case("petelix-2k", "petelix-2k", 2, 333, 1801, 16),
        # Delta rule with a decay per channel, differential and latent attention.
        _case("sisadra-2k", "sisadra-2k", 2, 333, 1801, 16),
        # Selective scan, sigmoid attention beside a linear recurrence, matrix memory, four residual streams.
        _case("guvetar-2k", "guvetar-2k", 2, 333, 1801, 16),
    ]


def _lengths(case) -> list:
    """Prompt lengths, the longest first, the others spread over the range out of order."""
    lo, hi = case["shortest"], case["longest"]
    return [hi - round((hi - lo) * ((0.618034 * i) % 1.0)) for i in range(case["requests"])]


def _steps(case) -> list:
    """[[(request, first, last + 1), ...], ...]: what each step runs of each request's tokens."""
    lengths, budget = _lengths(case), case["budget"]
    done, out = [0] * len(lengths), []
    while True:
        step, left = [], budget
        for r, n in enumerate(lengths):
            if n <= done[r] < n + case["new"]:
                step.append((r, done[r], done[r] + 1))
                left -= 1
        for r, n in enumerate(lengths):
            if done[r] < n and left > 0:
                take = min(left, n - done[r])
                step.append((r, done[r], done[r] + take))
                left -= take
        if not step:
            return out
        step.sort()
        for r, _, hi in step:
            done[r] = hi
        out.append(step)


def _wanted(case, r: int, hi: int) -> bool:
    """Whether the logits of the last of a step's tokens of a request are wanted (a next token would be picked)."""
    return hi >= _lengths(case)[r]


def _pairs(lo: int, hi: int, layer_window) -> int:
    """Visible (position, earlier position) pairs of positions lo..hi-1."""
    w = layer_window or (1 << 30)
    return sum(min(t + 1, w) for t in range(lo, hi))


def work(case) -> dict:
    """Every step reads its weights (of the experts, those its tokens can reach) and the cache rows its positions see
    once and writes its own cache rows and logits."""
    shapes, raw = _shapes(case["model"]), MODELS[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    tied = not any(n in ("head", "lm_head.weight") for n, _, _ in shapes)
    vocab = raw.get("vocab") or raw["vocab_size"]
    dense = experts = head = 0
    for n, shape, matrix in shapes:
        if not matrix:
            continue
        k = math.prod(shape)
        if n in ("embed", "bigram", "side.embed", "model.embed_tokens.weight"):
            head += k if tied and n in ("embed", "model.embed_tokens.weight") else 0
        elif n in ("head", "lm_head.weight"):
            head += k
        elif ".mlp.e" in n:
            experts += k
        else:
            dense += k
    router = next((l["mlp"]["router"] for l in raw.get("layers", []) if (l.get("mlp") or {}).get("kind") == "moe"), None)
    attends = _attention(raw)
    nbytes = flops = 0
    if case["generate"]:
        steps = max(1, case["new"])
        tokens = sum(_lengths(case)) + case["requests"] * (case["new"] - 1)
        again = tokens + case["requests"]
        return {"bytes": float((steps + 1) * (dense + head) * size + 4 * vocab * case["requests"]),
                "flops": float(2 * dense * (tokens + again) + 2 * head * case["requests"] * (case["new"] + 1))}
    for step in _steps(case):
        tokens = sum(hi - lo for _, lo, hi in step)
        rows = sum(_wanted(case, r, hi) for r, _, hi in step)
        share = min(1.0, tokens * router["top"] / router["experts"]) if router else 0.0
        nbytes += (dense + share * experts + (head if rows else 0)) * size + rows * vocab * 4
        flops += 2 * (dense + (experts * router["top"] / router["experts"] if router else 0)) * tokens + 2 * head * rows
        for window, width, per_pair in attends:
            for _, lo, hi in step:
                nbytes += width * size * (min(lo, window or lo) + 2 * (hi - lo))
                flops += per_pair * _pairs(lo, hi, window)
    return {"bytes": float(nbytes), "flops": float(flops)}


def _attention(raw) -> list:
    """(window, cached values a position, flops a visible pair) of every attention layer."""
    if "hidden_size" in raw:
        h, g, hd = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
        return [(None, 2 * g * hd, 4 * h * hd)] * len(raw["full_attn_idxs"])
    out = []
    for layer in raw["layers"]:
        m = layer["mixer"].get("left") or layer["mixer"]
        window = (m.get("mask") or {}).get("size")
        if layer["type"] == "latent_attention":
            out.append((window, m["kv_rank"] + m.get("rot_dim", 0), 2 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])))
        elif layer["type"] in ("attention", "parallel"):
            maps = 2 if "diff" in m else 1
            out.append((window, m["kv_heads"] * (maps * m["dim"] + m["vdim"]), 2 * maps * m["heads"] * (m["dim"] + m["vdim"])))
    return out


def _cost(case) -> float:
    """Rough seconds of a pass, to keep drawn cases below the largest listed one."""
    w = work(case)
    bf16 = case["dtype"] == "bfloat16"
    lfm2 = case["model"].startswith("lfm2")
    rate = (4e14 if lfm2 else 4e13) if bf16 else 1.2e13
    return w["bytes"] / 2.5e12 + w["flops"] / rate + 2e-4 * len(_steps(case))


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["chat", "chat", "prompt", "mixed", "float32", "tiny", "potivik", "petelix", "sisadra", "guvetar"])
        if kind == "tiny":
            lo, hi = sorted((log_int(1, 40), log_int(1, 40)))
            c = _case("", rng.choice(["lfm2-tiny-a", "lfm2-tiny-b"]), log_int(1, 8), lo, hi, rng.randint(4, 20), budget=2048,
                      dtype="float32", generate=True)
        elif kind == "float32":
            lo, hi = sorted((log_int(8, 200), log_int(8, 200)))
            c = _case("", "lfm2-700m", log_int(1, 8), lo, hi, rng.randint(0, 8), dtype="float32")
        elif kind in ("chat", "prompt", "mixed"):
            model = rng.choice(["lfm2-700m", "lfm2-1.2b", "lfm2-2.6b"])
            if kind == "prompt":
                n = log_int(24, 8000)
                c = _case("", model, 1, n, n, rng.choice([0, 0, 1, 3]))
            else:
                lo, hi = sorted((log_int(16, 2048), log_int(16, 2048)))
                c = _case("", model, log_int(1, 64), lo, hi, log_int(8, 48),
                          budget=rng.choice([256, 512, 1024, 2048]) if kind == "mixed" else 16384)
        else:
            lo, hi = sorted((log_int(16, 2048), log_int(16, 2048)))
            c = _case("", f"{kind}-{rng.choice(['1k', '2k'])}", log_int(1, 8), lo, hi, rng.randint(0, 16))
        if sum(_lengths(c)) <= c["budget"] or c["budget"] < 16384:
            if _cost(c) <= most:
                del c["name"]
                return c


# ---------------------------------------------------------------------------------------------------
# weights
# ---------------------------------------------------------------------------------------------------

def _generator(seed: int, name: str, device: str = "cuda") -> torch.Generator:
    return torch.Generator(device=device).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & ((1 << 62) - 1))


def _vector(raw, name: str, shape, normal, uniform):
    """Values of the vectors, of the size that trained ones have: (mean, spread) or the values."""
    last = "." + name
    arch = raw.get("architecture", "Lfm2")
    if last.endswith("hc1.mix") or last.endswith("hc2.mix"):
        n = shape[0]
        return 0.8 * torch.eye(n, device="cuda") + 0.25 / math.sqrt(n) * normal()
    if last.endswith(("hc1.in", "hc2.in")):
        return 1.0 / shape[0] + 0.2 * normal()
    if last.endswith(("hc1.out", "hc2.out")):
        return 0.8 + 0.2 * normal()
    if last.endswith("A_log"):
        if arch == "Guvetar":
            return torch.log(torch.linspace(0.05, 4.0, shape[1], device="cuda"))[None, :] + 0.3 * normal()
        if arch == "Sisadra":
            return torch.linspace(-2.5, 0.7, shape[0], device="cuda") + 0.1 * normal()
        return torch.log(0.3 + 3.0 * uniform())
    if last.endswith("dt_bias"):
        return (-1.5 if arch == "Potivik" else -0.5) + 0.8 * normal()
    if last.endswith("dt.b"):
        return -2.0 + normal()
    if last.endswith(".D"):
        return 1.0 + 0.2 * normal()
    if last.endswith("lower"):
        return 0.9 * uniform()
    if last.endswith(".pb"):
        return -3.0 + normal()
    if last.endswith(".sink"):
        return 0.5 + normal()
    if last.endswith(".i.b"):
        return -1.0 + normal()
    if last.endswith(".f.b"):
        return (1.5 if "right" in last else 3.0) + normal()
    if last.endswith(("lq1", "lk1", "lq2", "lk2")):
        return 0.5 / math.sqrt(shape[0]) * normal()
    if last.endswith("correction"):
        return 0.01 / shape[0] * normal()
    if last.endswith(("norm1b", "norm2b", "side.norm")):
        # norms behind a sublayer: what a sublayer adds is small beside the stream
        return 0.2 * (1.0 + 0.1 * normal())
    if "norm" in last:
        return 1.0 + 0.1 * normal()
    if "conv" in last and not last.endswith((".b", "bias")):
        return 0.3 + 0.4 * normal()
    return 0.1 * normal()                                    # biases


def _weights(case, seed: int) -> dict:
    """Random tensors of the model, on the GPU: matrices that keep the size of what passes through them, outputs of
    sublayers smaller than the stream, vectors as ``_vector`` says.  Experts are chosen as by a trained router, clearly:
    every token's embedding has a part along the router rows of the experts it goes to, so that rounding moves no choice."""
    raw, out = MODELS[case["model"]], {}
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    for name, shape, matrix in _shapes(case["model"]):
        g = _generator(seed, name)
        normal = lambda: torch.randn(shape, generator=g, device="cuda")             # noqa: E731
        uniform = lambda: torch.rand(shape, generator=g, device="cuda")             # noqa: E731
        if not matrix:
            out[name] = _vector(raw, name, shape, normal, uniform)
            continue
        std = 1.0 / math.sqrt(shape[-1])
        if name.endswith((".o", ".down", "out_proj.weight", "w2.weight")):
            std *= 0.3
        if name in ("embed", "bigram", "side.embed", "model.embed_tokens.weight"):
            std = 1.0 / float((raw.get("embedding") or {}).get("scale", 1.0))
        out[name] = torch.empty(shape, device="cuda", dtype=dtype).normal_(0.0, std, generator=g)
    _mark_experts(raw, seed, out)
    return out


def _mark_experts(raw, seed: int, tensors: dict) -> None:
    routed = [i for i, l in enumerate(raw.get("layers", [])) if (l.get("mlp") or {}).get("kind") == "moe"]
    if not routed:
        return
    embed = tensors["embed"].float()
    scale = float((raw.get("embedding") or {}).get("scale", 1.0))
    for i in routed:
        r = raw["layers"][i]["mlp"]["router"]
        n, count = r["experts"] + r.get("identity", 0), (r.get("groups") or {}).get("count", 1)
        keep = (r.get("groups") or {}).get("keep", count)
        g = _generator(seed, f"choice {i}")
        rows = torch.randn(n, embed.shape[1], generator=g, device="cuda")
        rows /= rows.norm(dim=1, keepdim=True)
        tensors[f"l{i}.mlp.router"] = (rows * (1.0 if raw["architecture"] == "Petelix" else 0.3)).to(tensors["embed"].dtype)
        score = torch.rand(embed.shape[0], count, n // count, generator=g, device="cuda")
        kept = torch.rand(embed.shape[0], count, generator=g, device="cuda").topk(keep, dim=1).indices
        mark = torch.zeros_like(score)
        mark.scatter_(2, score.topk(r["top"] // keep, dim=2).indices, 1.0)
        mark *= torch.zeros(embed.shape[0], count, device="cuda").scatter_(1, kept, 1.0)[:, :, None]
        embed += (mark * (9.0 + 2.0 * score)).reshape(-1, n) @ rows / scale
    tensors["embed"] = embed.to(tensors["embed"].dtype)


# ---------------------------------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------------------------------

def _tokens(case, seed: int) -> list:
    """Each request's prompt and the tokens behind it, uniform over the vocabulary."""
    raw = MODELS[case["model"]]
    vocab = raw.get("vocab") or raw["vocab_size"]
    g = _generator(seed, "tokens", "cpu")
    return [torch.randint(0, vocab, (n + case["new"],), generator=g).tolist() for n in _lengths(case)]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = dict(case)
    config = _config(case["model"])
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    model = build_model(config.plan(), TensorDict(_weights(case, seed)), dtype, "cuda:0")
    model.config = config
    tokens, longest = _tokens(case, seed), max(_lengths(case)) + case["new"]
    ctx = 16 * PAGE * (-(-longest // (16 * PAGE)))
    pages = sum(-(-(n + case["new"]) // PAGE) + 1 for n in _lengths(case)) + 1
    if case["generate"]:
        s.prompts = [t[:n] for t, n in zip(tokens, _lengths(case))]
        s.params = SamplingParams(temperature=0.0, max_new_tokens=case["new"])
        s.generator = Generator(model, dtype=case["dtype"], ctx=min(ctx, config.plan().max_context), page_size=PAGE,
                                n_pages=2 * pages, max_running=case["requests"], max_batch_tokens=case["budget"])
    else:
        steps = _steps(case)
        s.requests = list(range(case["requests"]))
        s.steps = [[StepEntry(r, tokens[r][lo:hi], (hi - lo - 1,) if _wanted(case, r, hi) else ()) for r, lo, hi in step]
                   for step in steps]
        s.ends = [[r for r, _, hi in step if hi == len(tokens[r])] for step in steps]
        rows = sum(len(e.want) for step in s.steps for e in step)
        s.logits = torch.empty((rows, model.vocab_size), dtype=torch.float32, device="cuda")
        s.engine = Engine(model, n_pages=pages, page_size=PAGE, max_requests=case["requests"],
                          max_step_tokens=max(sum(len(e.tokens) for e in step) for step in s.steps), max_context=ctx)
    run(s)           # a server has answered before: its decode graphs exist
    return s


def run(s):
    if s.case["generate"]:
        return _generate(s)
    row = 0
    for r in s.requests:
        s.engine.open(r)
    for entries, ends in zip(s.steps, s.ends):
        logits = s.engine.step(entries)
        if logits is not None:
            # (the next decode step writes into the same logits)
            s.logits[row:row + logits.shape[0]].copy_(logits)
            row += logits.shape[0]
        for r in ends:
            s.engine.close(r)
    return s.logits


def _generate(s):
    """The tokens, and the logits that a scoring step over prompt and answer gives for what would come next."""
    ids = s.generator.generate(s.prompts, s.params, stop_at_eos=False)
    eng = s.generator.engine
    for r in range(len(ids)):
        eng.open(("score", r))
    logits = eng.step([StepEntry(("score", r), p + a, (len(p) + len(a) - 1,)) for r, (p, a) in enumerate(zip(s.prompts, ids))])
    for r in range(len(ids)):
        eng.close(("score", r))
    return {"tokens": torch.tensor(ids), "logits": logits}


def tolerance(case):
    """About three times what this engine is off 64-bit arithmetic (0.002 to 0.008 in bfloat16, whose products and caches
    are rounded to 8 bits; 4e-7 to 2e-6 in 32-bit): sums in another order round differently everywhere."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.02, "max": 0.4}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------

def exact(case, seed):
    raw, tensors, tokens = MODELS[case["model"]], _weights(case, seed), _tokens(case, seed)
    tensors = {k: v.cpu() if v.numel() > (1 << 28) else v for k, v in tensors.items()}
    lengths = _lengths(case)
    forward = _forward_lfm2 if "hidden_size" in raw else _forward_layers
    if case["generate"]:
        ids = [t[:n] for t, n in zip(tokens, lengths)]
        for _ in range(case["new"]):
            z = forward(raw, tensors, ids, [[len(t) - 1] for t in ids])
            ids = [t + [int(zi[0].argmax())] for t, zi in zip(ids, z)]
        z = forward(raw, tensors, ids, [[len(t) - 1] for t in ids])
        return {"tokens": torch.tensor([t[n:] for t, n in zip(ids, lengths)]), "logits": torch.cat(z)}
    z = forward(raw, tensors, tokens, [list(range(n - 1, n + case["new"])) for n in lengths])
    at = [0] * len(tokens)
    out = []
    for step in _steps(case):
        for r, _, hi in step:
            if _wanted(case, r, hi):
                out.append(z[r][at[r]])
                at[r] += 1
    return torch.stack(out)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, gain, eps):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, freq, pairs: str):
    """x [T, heads, dim]: the first 2 len(freq) entries turned by position * freq (the angle formed in 32-bit, as the
    designs do), entries (2i, 2i + 1) or (i, i + n) together."""
    n = freq.numel()
    ang = (torch.arange(x.shape[0], device=x.device).float()[:, None] * freq.to(x.device).float()[None, :]).to(F64)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    out = x.clone()
    a, b = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if pairs == "adjacent" else (slice(0, n), slice(n, 2 * n))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _frequencies(base, dims, scaling=None):
    f = torch.pow(torch.tensor(float(base), dtype=F64), -2.0 * torch.arange(dims // 2, dtype=F64) / dims)
    if scaling:
        factor, low, high, orig = (float(scaling[k]) for k in ("factor", "low", "high", "original"))
        wave = 2.0 * math.pi / f
        s = ((orig / wave - low) / (high - low)).clamp(0.0, 1.0)
        f = (1.0 - s) * f / factor + s * f
    return f


def _seen(T, device, window=None, block=None):
    i = torch.arange(T, device=device)
    seen = i[None, :] <= i[:, None]
    if window:
        seen &= i[:, None] - i[None, :] < window
    if block:
        seen &= torch.div(i, block, rounding_mode="floor")[:, None] == torch.div(i, block, rounding_mode="floor")[None, :]
    return seen


def _softmax(s, seen, sink=None):
    """Softmax over what is seen; ``sink``: a score that joins the denominator only."""
    s = s.masked_fill(~seen, -math.inf)
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        m = m.clamp(min=float(sink))
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(sink - m) if sink is not None else 0.0))


def _conv(x, taps, bias=0.0):
    """x [T, C], taps [C, K]: the last tap on the current token, zeros before the start."""
    T, K = x.shape[0], taps.shape[1]
    padded = torch.cat([torch.zeros(K - 1, x.shape[1], dtype=F64, device=x.device), x])
    return sum(padded[n:n + T] * taps[:, n] for n in range(K)) + bias


def _each(fn, lengths, *rows):
    """``fn`` on every request's rows, the results one behind the other."""
    return torch.cat([fn(*parts) for parts in zip(*(r.split(lengths) for r in rows))])


def _forward_lfm2(raw, tensors, tokens, rows):
    eps, hd = raw["norm_eps"], raw["head_dim"]
    lengths = [len(t) for t in tokens]
    ids = torch.tensor([i for t in tokens for i in t], device="cuda")
    W = lambda n: tensors[n].to(device="cuda", dtype=F64)                                          # noqa: E731
    B = lambda n: W(n) if n in tensors else 0.0                                                    # noqa: E731
    x = tensors["model.embed_tokens.weight"].to("cuda")[ids].to(F64)
    j = torch.arange(hd // 2, dtype=torch.float32)
    freq = 1.0 / torch.pow(torch.tensor(float(raw["rope_theta"])), 2.0 * j / hd)

    def attend(q, k, v):
        q, k = _turn(q, freq, "halves"), _turn(k, freq, "halves")
        out, seen, per = torch.empty_like(q), _seen(q.shape[0], q.device), q.shape[1] // k.shape[1]
        for h in range(q.shape[1]):
            out[:, h] = _softmax(q[:, h] @ k[:, h // per].T / math.sqrt(hd), seen) @ v[:, h // per]
        return out

    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W(p + "operator_norm.weight")
        if i in raw["full_attn_idxs"]:
            q, k, v = ((h @ W(p + f"self_attn.{n}_proj.weight").T + B(p + f"self_attn.{n}_proj.bias")).reshape(len(ids), -1, hd)
                       for n in "qkv")
            q = _rms(q, eps) * W(p + "self_attn.q_layernorm.weight")
            k = _rms(k, eps) * W(p + "self_attn.k_layernorm.weight")
            o = _each(attend, lengths, q, k, v).reshape(len(ids), -1)
            x = x + o @ W(p + "self_attn.out_proj.weight").T + B(p + "self_attn.out_proj.bias")
        else:
            b, c, u = (h @ W(p + "conv.in_proj.weight").T + B(p + "conv.in_proj.bias")).chunk(3, dim=-1)
            taps, bias = W(p + "conv.conv.weight" if p + "conv.conv.weight" in tensors else p + "conv.weight"), B(p + "conv.conv.bias")
            y = c * _each(lambda z: _conv(z, taps.reshape(raw["hidden_size"], -1), bias), lengths, b * u)
            x = x + y @ W(p + "conv.out_proj.weight").T + B(p + "conv.out_proj.bias")
        h = _rms(x, eps) * W(p + "ffn_norm.weight")
        f = p + "feed_forward."
        x = x + (_silu(h @ W(f + "w1.weight").T) * (h @ W(f + "w3.weight").T)) @ W(f + "w2.weight").T
    z = torch.cat([part[r] for part, r in zip(x.split(lengths), rows)])
    head = "lm_head.weight" if "lm_head.weight" in tensors else "model.embed_tokens.weight"
    z = (_rms(z, eps) * W("model.embedding_norm.weight")) @ W(head).T
    return list(z.split([len(r) for r in rows]))


def _windowed_latent(h, w, m, eps, lengths):
    """Latent attention with a rotated key part, a window and a gate per head (or neither, with a sink per head)."""
    T, H, dn, dr, dv, r = h.shape[0], m["heads"], m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"]
    q = (h @ w["q"].T).reshape(T, H, dn + dr)
    both = h @ w["dkv"].T
    c = _rms(both[:, :r], eps) * w["dkv.norm"]
    k, v = (c @ w["uk"].T).reshape(T, H, dn), (c @ w["uv"].T).reshape(T, H, dv)

    def attend(q, k, v, part):
        seen = _seen(q.shape[0], q.device, window=(m.get("mask") or {}).get("size"))
        if dr:
            f = _frequencies(m["rot"]["base"], m["rot"]["dims"])
            q = torch.cat([q[..., :dn], _turn(q[..., dn:], f, "adjacent")], -1)
            k = torch.cat([k, _turn(part[:, None], f, "adjacent").expand(-1, H, -1)], -1)
        return torch.stack([_softmax(q[:, n] @ k[:, n].T * m["scale"], seen, w["sink"][n] if "sink" in w else None) @ v[:, n]
                            for n in range(H)], 1)

    o = _each(attend, lengths, q, k, v, both[:, r:])
    if "g" in w:
        o = o * torch.sigmoid(h @ w["g"].T)[:, :, None]
    return o.reshape(T, -1) @ w["o"].T


def _mamba2(h, w, m, eps, lengths):
    T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    u = h @ w["in"].T
    z, xbc, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])

    def scan(xbc, dt):
        xbc = _silu(_conv(xbc, w["conv"], w["conv.b"]))
        x = xbc[:, :inner].reshape(-1, H, P)
        B, C = (xbc[:, a:a + G * N].reshape(-1, G, N).repeat_interleave(H // G, 1) for a in (inner, inner + G * N))
        decay = torch.exp(-torch.exp(w["A_log"]) * dt)
        S, out = torch.zeros(H, N, P, dtype=F64, device=h.device), torch.empty_like(x)
        xd = x * dt[:, :, None]
        for t in range(x.shape[0]):
            S = decay[t][:, None, None] * S + B[t][:, :, None] * xd[t][:, None, :]
            out[t] = (S * C[t][:, :, None]).sum(1)
        return (out + w["D"][None, :, None] * x).reshape(-1, inner)

    y = _each(scan, lengths, xbc, dt) * _silu(z)
    y = _rms(y.reshape(T, m["norm_groups"], -1), eps).reshape(T, inner) * w["norm"]
    return y @ w["o"].T


def _sink_attention(h, w, m, eps, lengths, kv):
    T, H, G, dim, vdim = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    f = _frequencies(m["rot"]["base"], m["rot"]["dims"])
    turn = lambda x: _turn(x, f, "adjacent")                                                       # noqa: E731
    q = _each(turn, lengths, (_rms(h @ w["q"].T, eps) * w["q.norm"]).reshape(T, H, dim))
    if kv is None:
        kv = (_each(turn, lengths, (_rms(h @ w["k"].T, eps) * w["k.norm"]).reshape(T, G, dim)), (h @ w["v"].T).reshape(T, G, vdim))

    def attend(q, k, v):
        seen, zero = _seen(q.shape[0], q.device, window=m["mask"]["size"]), torch.zeros((), dtype=F64, device=q.device)
        out = []
        for n in range(H):
            s = m["softcap"] * torch.tanh(q[:, n] @ k[:, n * G // H].T * m["scale"] / m["softcap"])
            out.append(_softmax(s, seen, zero) @ v[:, n * G // H])
        return torch.stack(out, 1)

    o = _each(attend, lengths, q, *kv).reshape(T, -1) * torch.sigmoid(h @ w["g"].T)
    return o @ w["o"].T, kv


def _differential(h, w, m, eps, lengths):
    T, H, G, dim, vdim = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q = _rms((h @ w["q"].T + w["q.b"]).reshape(T, 2 * H, dim), eps) * w["q.norm"]
    k = _rms((h @ w["k"].T + w["k.b"]).reshape(T, 2 * G, dim), eps) * w["k.norm"]
    v = (h @ w["v"].T + w["v.b"]).reshape(T, G, vdim)
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + m["diff"]
    f = _frequencies(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])

    def attend(q, k, v):
        q, k, seen = _turn(q, f, "halves"), _turn(k, f, "halves"), _seen(q.shape[0], q.device, block=m["mask"]["size"])
        out = []
        for n in range(H):
            g = n * G // H
            a, b = (_softmax(q[:, 2 * n + e] @ k[:, 2 * g + e].T * m["scale"], seen) @ v[:, g] for e in (0, 1))
            out.append(_rms(a - lam * b, eps) * (1.0 - m["diff"]))
        return torch.stack(out, 1)

    return _each(attend, lengths, q, k, v).reshape(T, -1) @ w["o"].T + w["o.b"]


def _channel_delta(h, w, m, eps, lengths):
    T, H, G, dim, vdim = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)                          # noqa: E731
    q, k, v = (_each(lambda z: _silu(_conv(z, w[n + ".conv"])), lengths, h @ w[n].T) for n in "qkv")
    q = (unit(q.reshape(T, G, dim)) * dim ** -0.5).repeat_interleave(H // G, 1)
    k, v = unit(k.reshape(T, G, dim)).repeat_interleave(H // G, 1), v.reshape(T, H, vdim)
    beta = torch.sigmoid(h @ w["b"].T)
    a = torch.nn.functional.softplus((h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).reshape(T, H, dim)
    decay = torch.exp(-torch.exp(w["A_log"])[None, :, None] * a)

    def rule(q, k, v, beta, decay):
        S, out = torch.zeros(H, dim, vdim, dtype=F64, device=h.device), torch.empty_like(v)
        for t in range(q.shape[0]):
            S = decay[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[t] = (S * q[t][:, :, None]).sum(1)
        return out

    o = _rms(_each(rule, lengths, q, k, v, beta, decay), eps) * w["norm"]
    gate = torch.sigmoid((h @ w["g1"].T) @ w["g2"].T)
    return (o.reshape(T, -1) * gate) @ w["o"].T


def _mamba1(h, w, m, eps, lengths):
    inner, rank, n = m["inner"], m["dt_rank"], m["state"]
    x, z = (h @ w["in"].T).split(inner, -1)
    x = _each(lambda v: _silu(_conv(v, w["conv"], w["conv.b"])), lengths, x)
    p = x @ w["x"].T
    dt = torch.nn.functional.softplus(p[:, :rank] @ w["dt"].T + w["dt.b"])
    A = -torch.exp(w["A_log"])

    def scan(x, dt, B, C):
        S, y = torch.zeros_like(A), torch.empty_like(x)
        for t in range(x.shape[0]):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * x[t])[:, None] * B[t][None, :]
            y[t] = S @ C[t] + w["D"] * x[t]
        return y

    return (_each(scan, lengths, x, dt, p[:, rank:rank + n], p[:, rank + n:]) * _silu(z)) @ w["o"].T


def _sigmoid_attention(h, w, m, eps, lengths):
    T, H, G, dim = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    q = _rms((h @ w["q"].T).reshape(T, H, dim), eps) * w["q.norm"]
    k = _rms((h @ w["k"].T).reshape(T, G, dim), eps) * w["k.norm"]
    v = (h @ w["v"].T).reshape(T, G, m["vdim"])
    t = m["q_temp"]

    def attend(q, k, v):
        p = torch.arange(q.shape[0], dtype=F64, device=q.device)
        q = q * (1.0 + t["coef"] * torch.log(torch.floor((p + 1.0) / t["every"]) + 1.0))[:, None, None]
        seen = _seen(q.shape[0], q.device)
        return torch.stack([(torch.sigmoid(q[:, n] @ k[:, n * G // H].T * m["scale"] + w["pb"][n]) * seen) @ v[:, n * G // H]
                            for n in range(H)], 1)

    return _each(attend, lengths, q, k, v).reshape(T, -1) @ w["o"].T


def _gated_write(h, w, m, eps, lengths):
    T, H, dim, vdim = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q = _silu(h @ w["q"].T).reshape(T, H, dim)
    f = (w["lower"] + (1.0 - w["lower"]) * torch.sigmoid(h @ w["f"].T + w["f.b"])).reshape(T, H, dim)
    v = (h @ w["v"].T).reshape(T, H, vdim)

    def rule(q, f, v):
        S, out = torch.zeros(H, dim, vdim, dtype=F64, device=h.device), torch.empty_like(v)
        for t in range(q.shape[0]):
            S = f[t][:, :, None] * S + (1.0 - f[t])[:, :, None] * v[t][:, None, :]
            out[t] = (S * q[t][:, :, None]).sum(1)
        return out

    return (_rms(_each(rule, lengths, q, f, v), eps) * w["norm"]).reshape(T, -1) @ w["o"].T


def _both(h, w, m, eps, lengths):
    left = _sigmoid_attention(h, _sub(w, "left."), m["left"], eps, lengths)
    return m["left_scale"] * left + m["right_scale"] * _gated_write(h, _sub(w, "right."), m["right"], eps, lengths)


def _matrix_memory(h, w, m, eps, lengths):
    T, H, dim, vdim, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], float(m["gate_cap"])
    q, k, v = ((h @ w[n].T).reshape(T, H, -1) for n in "qkv")
    q = q * dim ** -0.5
    i = cap * torch.tanh((h @ w["i"].T + w["i.b"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w["f"].T + w["f.b"]) / cap))

    def rule(q, k, v, i, f):
        S, n = torch.zeros(H, dim, vdim, dtype=F64, device=h.device), torch.zeros(H, dim, dtype=F64, device=h.device)
        top, out = torch.zeros(H, dtype=F64, device=h.device), torch.empty_like(v)
        for t in range(q.shape[0]):
            new = torch.maximum(f[t] + top, i[t])
            keep, write = torch.exp(f[t] + top - new)[:, None], torch.exp(i[t] - new)[:, None]
            kw, top = write * k[t], new
            S = keep[:, :, None] * S + kw[:, :, None] * v[t][:, None, :]
            n = keep * n + kw
            den = torch.maximum((n * q[t]).sum(1).abs(), torch.exp(-top)) + 1e-6
            out[t] = (S * q[t][:, :, None]).sum(1) / den[:, None]
        return out

    o = _rms(_each(rule, lengths, q, k, v, i, f), eps).reshape(T, -1) * w["norm"]
    return (o * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _feed_forward(arch, h, w, f):
    if f["kind"] == "moe":
        return _experts(arch, h, w, f)
    if arch == "Potivik":
        return _clamped(h, w["gate"], w["up"], w["down"], f["limit"])
    z = h @ w["up"].T
    z = torch.relu(z) ** 2 if arch == "Guvetar" else 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))
    return z @ w["down"].T


def _clamped(h, gate, up, down, limit):
    g, u = (h @ gate.T).clamp(max=limit), (h @ up.T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down.T


def _experts(arch, h, w, f):
    r, z, out = f["router"], h @ w["router"].T, torch.zeros_like(h)
    if arch == "Potivik":
        score = torch.sigmoid(z)
        pick = score
    else:
        score = torch.softmax(z, -1)
        pick, count = score + w["correction"], r["groups"]["count"]
        best = pick.reshape(-1, count, pick.shape[1] // count).amax(-1).topk(r["groups"]["keep"], dim=-1).indices
        open_ = torch.zeros(len(h), count, dtype=torch.bool, device=h.device).scatter_(1, best, True)
        pick = pick.masked_fill(~open_.repeat_interleave(pick.shape[1] // count, 1), -math.inf)
    chosen = torch.zeros_like(score, dtype=torch.bool).scatter_(1, pick.topk(r["top"], dim=-1).indices, True)
    for e in range(score.shape[1]):
        t = chosen[:, e].nonzero().flatten()
        if not t.numel():
            continue
        s = score[t, e][:, None]
        if e >= r["experts"]:
            out[t] += s * h[t]
        elif arch == "Potivik":
            out[t] += _clamped(s * h[t], w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"], f["expert"]["limit"])
        else:
            out[t] += s * ((_silu(h[t] @ w[f"e{e}.gate"].T) * (h[t] @ w[f"e{e}.up"].T)) @ w[f"e{e}.down"].T)
    if f.get("shared"):
        both = _clamped(h, w["shared.gate"], w["shared.up"], w["shared.down"], f["shared"]["limit"])
        out = out + torch.sigmoid(h @ w["shared.sg"].T) * both
    return out


class _Sub(dict):
    """Tensors under a prefix, widened when they are read."""

    def __getitem__(self, k):
        return super().__getitem__(k).to(device="cuda", dtype=F64)


def _sub(tensors, prefix):
    return _Sub({k[len(prefix):]: dict.__getitem__(tensors, k) for k in tensors if k.startswith(prefix)})


_MIXERS = {"mamba2": _mamba2, "channel_delta": _channel_delta, "mamba1": _mamba1, "parallel": _both, "mlstm": _matrix_memory,
           "latent_attention": _windowed_latent}


def _forward_layers(raw, tensors, tokens, rows):
    """Potivik, Petelix, Sisadra and Guvetar: logits at the given rows of each sequence."""
    arch, eps, T = raw["architecture"], raw["norm"]["eps"], _Sub(tensors)
    lengths, ids = [len(t) for t in tokens], torch.tensor([i for t in tokens for i in t], device="cuda")
    x = tensors["embed"].to("cuda")[ids].to(F64) * float((raw.get("embedding") or {}).get("scale", 1.0))
    pair = (raw.get("embedding") or {}).get("bigram")
    if pair:
        at = [torch.cat([t.new_tensor([pair["buckets"]]), (t[:-1] * pair["mul_prev"] + t[1:] * pair["mul_cur"]) % pair["buckets"]])
              for t in ids.split(lengths)]
        x = x + tensors["bigram"].to("cuda")[torch.cat(at)].to(F64)
    norm = (lambda v, n: _layer_norm(v, T[n], eps)) if arch in ("Potivik", "Sisadra") else (lambda v, n: _rms(v, eps) * T[n])
    if arch == "Guvetar":
        e = torch.arange(raw["width"], device="cuda")
        f = torch.pow(torch.tensor(10000.0, dtype=F64, device="cuda"), -(2 * (e // 2)).to(F64) / raw["width"])
        ang = torch.cat([torch.arange(n, device="cuda") for n in lengths]).float()[:, None] * f.float()[None, :]
        x = x + torch.where(e % 2 == 0, torch.sin(ang.to(F64)), torch.cos(ang.to(F64)))
        x = x[None].repeat(raw["streams"], 1, 1)
    kept = {}
    for i, layer in enumerate(raw["layers"]):
        p, m = f"l{i}.", layer["mixer"]

        def mix(h):
            if layer["type"] != "attention":
                return _MIXERS[layer["type"]](h, _sub(tensors, p + "mix."), m, eps, lengths)
            if arch == "Sisadra":
                return _differential(h, _sub(tensors, p + "mix."), m, eps, lengths)
            y, kept[i] = _sink_attention(h, _sub(tensors, p + "mix."), m, eps, lengths, kept.get(m.get("kv_from")))
            return y

        for n, fn in (("1", mix), ("2", lambda h: _feed_forward(arch, h, _sub(tensors, p + "mlp."), layer["mlp"]))):
            if arch == "Guvetar":
                y = fn(norm(torch.einsum("s,std->td", T[p + f"hc{n}.in"], x), p + "norm" + n))
                x = torch.einsum("sn,std->ntd", T[p + f"hc{n}.mix"], x) + T[p + f"hc{n}.out"][:, None, None] * y[None]
            else:
                y = fn(norm(x, p + "norm" + n))
                x = x + (norm(y, p + f"norm{n}b") if arch == "Potivik" else y)
        if raw.get("token_side"):
            d = raw["token_side"]["dim"]
            g = torch.nn.functional.gelu(x @ T[p + "side.gate"].T, approximate="tanh")
            g = g * tensors["side.embed"].to("cuda")[:, i * d:(i + 1) * d][ids].to(F64)
            x = x + _rms(g @ T[p + "side.proj"].T, eps) * T[p + "side.norm"]
    if arch == "Guvetar":
        x = x.sum(0)
    z = torch.cat([part[r] for part, r in zip(x.split(lengths), rows)])
    z = norm(z, "final.norm") @ T["embed" if arch == "Guvetar" else "head"].T
    cap = raw.get("logit_softcap")
    return list((cap * torch.tanh(z / cap) if cap else z).split([len(r) for r in rows]))

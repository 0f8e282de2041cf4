"""The Petelix design on the GPU against the plain implementation
(tests/plain_petelix.py): every mechanism alone, then whole models through the
engine's step function, cut and batched in every way, then greedy generation
through the scheduler.

Where both compute dtypes run: float32 must match every row; in bfloat16 a
router choice at a near tie may flip under the rounding of the router's
input, which changes that token's row (and, faintly, later ones), so whole
models are held to "nearly all rows" there.  Mechanisms alone are given inputs
without such ties and are held to every row in both.
"""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import plain_petelix as plain
from helpers import run_trace_on_engine, trace_mixed, trace_portions, trace_tail_decoded, trace_whole
from petelix_helpers import (CFG_A, CFG_B, CFG_C, CFG_D, CONFIGS, attention_params, build, make_weights, random_config,
                             routed_params)
from potivik_helpers import PartHarness, ids_for, make_part, rel_rows

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-4, "bfloat16": 4e-2}
DEV = "cuda:0"
F64 = torch.float64


def gen(seed):
    return torch.Generator().manual_seed(seed)


def bf(t):
    return t.to(torch.bfloat16).to(torch.float32)


def dbl(W):
    return {k: v.double() for k, v in W.items()}


def check_rows(got, want, dtype: str, strict: bool = True, what: str = ""):
    e = rel_rows(got, want)
    if strict or dtype == "float32":
        assert e.max() <= TOL[dtype], f"{what}: row {int(e.argmax())} differs by {e.max():.3g} (tolerance {TOL[dtype]})"
    else:
        frac = float((e > TOL[dtype]).mean())
        assert frac <= 0.45 and np.median(e) <= 0.75 * TOL[dtype], \
            f"{what}: {frac:.1%} of the rows differ by more than {TOL[dtype]} (median {np.median(e):.3g})"


# ---------------------------------------------------------------------------
# mechanisms alone
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("scale", [1.0, 0.37, 12.0])
def test_embedding_with_a_scale(dtype, scale):
    from gibbs_b200.engine.step import StepState
    g = gen(1)
    V, d = 77, 52
    table = bf(torch.randn(V, d, generator=g))
    part = make_part("embedding", "token_embedding", {"vocab": V, "dim": d, "scale": scale}, {"weight": table}, DTYPES[dtype])
    ids = torch.randint(0, V, (33,), generator=g)
    out = part.forward(ids.to(DEV, torch.int32)).cpu()
    assert out.dtype == torch.float32
    assert rel_rows(out, table[ids].double() * scale).max() < 1e-6


def _plain_mixer(h, W, m, eps):
    pos = torch.arange(h.shape[0])
    return plain.attention_mixer(h.double(), dbl(W), m, eps, pos, None)[0]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg,layer", [(CFG_A, 0), (CFG_A, 2), (CFG_B, 0), (CFG_B, 1), (CFG_C, 0), (CFG_C, 1),
                                       (CFG_D, 0), (CFG_D, 2), (CFG_D, 3), (CFG_D, 4)])
def test_attention_alone_whole_cut_and_decoded(cfg, layer, dtype):
    m, d, eps = cfg["layers"][layer]["mixer"], cfg["width"], cfg["norm"]["eps"]
    W = plain.sub(make_weights(cfg, 5), f"l{layer}.mix.")
    part = make_part("mixer", "gated_attention", attention_params(m, d, eps), W, DTYPES[dtype])
    T = 150
    h = bf(torch.randn(T, d, generator=gen(6)))
    want = _plain_mixer(h, W, m, eps)
    # the sink shows: the first tokens see few keys, and their weights do not add up to one
    no_sink = _attention_without_sink(h, W, m, eps)
    assert rel_rows(no_sink[:3], want[:3]).max() > 0.05
    hz = PartHarness(part, n_pages=12, page_size=16, fill=0.0)      # 12 pages: 192 positions, pages come back and go out again
    for rid, cuts in (("whole", [T]), ("cut", [2, 3, 17, 2, 31, 16, 1, 5, 64, 7]), ("decoded", [T - 45, 1])):
        got = hz.run_cut(rid, h, cuts)
        check_rows(got, want, dtype, what=f"attention, {rid}")
        hz.close(rid)


def _attention_without_sink(h, W, m, eps):
    """The same mixer with an ordinary softmax, to show that a test's inputs tell the two apart."""
    Wd, pos = dbl(W), torch.arange(h.shape[0])
    H, dim = m["heads"], m["dim"]
    rot = m.get("rot") or {}
    q = plain.rotate_pairs(plain.rms_norm(h.double() @ Wd["q"].T, Wd["q.norm"], eps).reshape(-1, H, dim), pos,
                           rot.get("base", 1.0), int(rot.get("dims", 0)))
    k, v = plain.keys_and_values(h.double(), Wd, m, eps, pos)
    T, G = h.shape[0], m["kv_heads"]
    out = torch.zeros(T, H, m["vdim"], dtype=F64)
    w = (m.get("mask") or {}).get("size")
    for hd in range(H):
        s = (q[:, hd] @ k[:, hd // (H // G)].T) * m["scale"]
        if m.get("softcap"):
            s = m["softcap"] * torch.tanh(s / m["softcap"])
        i, j = torch.arange(T)[:, None], torch.arange(T)[None, :]
        seen = (j <= i) & ((i - j < w) if w else True)
        out[:, hd] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, hd // (H // G)]
    o = out.reshape(T, -1) * torch.sigmoid(h.double() @ Wd["g"].T)
    return o @ Wd["o"].T


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_norm_is_over_the_whole_projection_and_the_cap_bends_large_scores(dtype):
    """Heads of very unequal size and scores far beyond the cap: a norm per head, or no cap, gives other rows."""
    d, eps = 48, 1e-5
    m = {"heads": 4, "kv_heads": 2, "dim": 8, "vdim": 8, "scale": 2.0, "softcap": 3.0, "mask": {"size": 50},
         "rot": {"base": 100.0, "dims": 4}}
    g = gen(31)
    W = {"q": torch.randn(32, d, generator=g) / 7, "k": torch.randn(16, d, generator=g) / 7, "v": torch.randn(16, d, generator=g) / 5,
         "q.norm": 1 + 0.2 * torch.randn(32, generator=g), "k.norm": 1 + 0.2 * torch.randn(16, generator=g),
         "g": torch.randn(32, d, generator=g) / 5, "o": torch.randn(d, 32, generator=g) / 6}
    W["q"][:8] *= 9.0                                          # head 0 carries nearly all of the projection's mean square
    W["k"][8:] *= 5.0
    W = {k: bf(v) for k, v in W.items()}
    h = bf(torch.randn(70, d, generator=g))
    want = _plain_mixer(h, W, m, eps)
    uncapped = _plain_mixer(h, W, {**m, "softcap": None}, eps)
    assert np.median(rel_rows(uncapped, want)) > 0.05
    q = h.double() @ W["q"].double().T
    per_head = plain.rms_norm(q.reshape(-1, 4, 8), 1.0, eps).reshape(-1, 32)
    assert rel_rows(per_head, plain.rms_norm(q, 1.0, eps)).max() > 0.5
    part = make_part("mixer", "gated_attention", attention_params(m, d, eps), W, DTYPES[dtype])
    hz = PartHarness(part, fill=0.0)
    check_rows(hz.run_cut("a", h, [33, 2, 1]), want, dtype, what="unequal heads, capped scores")


def _pointed_attention(window, T, hot_key, query, vdim=8, seed=7):
    """Weights and inputs for which the query position's score against ``hot_key`` stands far above all
    others (when that key is visible), and whose values tell keys apart.  Keys read the input's first 64
    entries, queries its last 64: the query token's own key is an ordinary one."""
    d, H, G, dim = 128, 2, 1, 64
    m = {"heads": H, "kv_heads": G, "dim": dim, "vdim": vdim, "scale": 1.0, "softcap": 100.0}
    if window:
        m["mask"] = {"size": window}
    g = gen(seed)
    W = {"q": torch.zeros(H * dim, d), "k": torch.zeros(G * dim, d), "v": bf(torch.randn(G * vdim, d, generator=g) / 8),
         "q.norm": torch.ones(H * dim), "k.norm": torch.ones(G * dim), "g": torch.zeros(H * vdim, d),
         "o": bf(torch.randn(d, H * vdim, generator=g) / 4)}
    for i in range(dim):
        W["k"][i, i] = 1.0
        for hh in range(H):
            W["q"][hh * dim + i, 64 + i] = 1.0
    h = bf(torch.randn(T, d, generator=g))
    h[query, 64:] = h[hot_key, :64]          # q of the query token points along the hot key: score 64 against about +-8
    return m, W, h


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("decoded", [False, True])
@pytest.mark.parametrize("vdim", [8, 32])                     # 32: in bfloat16 the tensor-core kernel runs
@pytest.mark.parametrize("window,T,hot,query", [
    (40, 120, 60, 99),        # the oldest key the window keeps (99 - 60 = 39)
    (40, 120, 59, 99),        # the first one it has dropped
    (40, 120, 0, 39),         # the first token of the sequence, just inside
    (40, 120, 0, 40),         # ... and just outside
    (16, 120, 80, 95),        # a window of one page: its edge is a page's edge
    (16, 120, 79, 95),
    (32, 120, 64, 95),        # a window of one key tile
    (32, 120, 63, 95),
    (64, 200, 128, 191),      # ... of the tensor-core kernel's key tile
    (64, 200, 127, 191),
    (None, 400, 3, 399),      # no window: a key hundreds of positions back
    (None, 400, 16, 399),     # ... at a page's first row
    (None, 400, 31, 399),     # ... at a key tile's last row
    (300, 400, 100, 399),     # a long window: far but inside
    (300, 400, 99, 399),      # ... and outside
])
def test_attention_finds_the_one_key_that_matters(window, T, hot, query, vdim, decoded, dtype):
    m, W, h = _pointed_attention(window, T, hot, query, vdim)
    part = make_part("mixer", "gated_attention", attention_params(m, h.shape[1], 1e-5), W, DTYPES[dtype])
    want = _plain_mixer(h, W, m, 1e-5)
    visible = window is None or query - hot < window
    hz = PartHarness(part, n_pages=32, page_size=16, fill=0.0)
    got = hz.run_cut("r", h, [query - 10, 1] if decoded else [T])
    e = rel_rows(got, want)
    assert e[query] <= TOL[dtype], f"query row differs by {e[query]:.3g}"
    # (the other rows' scores are eight times as wide as a model's: in bfloat16 the rounding of keys and queries
    # shows in their sharp softmax)
    assert e.max() <= (TOL[dtype] if dtype == "float32" else 0.1)
    # the hot key's value dominates the output exactly when it is visible (gate logits are zero: sigmoid = 1/2)
    v_hot = (W["v"].double() @ h[hot].double()) * 0.5
    out_hot = W["o"].double() @ torch.cat([v_hot, v_hot])
    close = float((got[query].double() - out_hot).norm() / out_hot.norm())
    assert (close < 0.2) == visible, f"hot key visible={visible}, distance to its value {close:.3g}"


def _without_ties(h, W, f, margin=0.02):
    """The rows of h whose choice of experts and of groups does not hang on the last bits."""
    r = f["router"]
    s = torch.softmax(h.double() @ W["router"].double().T, -1)
    c = s + W["correction"].double()
    g = r.get("groups") or {}
    count, keep_g = g.get("count", 1), g.get("keep", g.get("count", 1))
    ok = torch.ones(h.shape[0], dtype=torch.bool)
    if count > 1 and keep_g < count:
        marks = torch.sort(c.reshape(h.shape[0], count, -1).max(-1).values, dim=1, descending=True).values
        ok &= (marks[:, keep_g - 1] - marks[:, keep_g]) > margin * marks[:, 0].abs().clamp(min=0.05)
    open_ = torch.ones_like(c, dtype=torch.bool)
    if count > 1 and keep_g < count:
        best = c.reshape(h.shape[0], count, -1).max(-1).values
        kept = torch.topk(best, keep_g, dim=-1).indices
        allowed = torch.zeros(h.shape[0], count, dtype=torch.bool).scatter_(1, kept, True)
        open_ = allowed[:, :, None].expand(-1, -1, c.shape[1] // count).reshape(h.shape[0], -1)
    cc = torch.where(open_, c, torch.full_like(c, -math.inf))
    srt = torch.sort(cc, dim=1, descending=True).values
    top = r["top"]
    if top < int(open_[0].sum()):
        ok &= (srt[:, top - 1] - srt[:, top]) > margin * 0.1
    return ok


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg,layer", [(CFG_A, 0), (CFG_A, 2), (CFG_A, 3), (CFG_B, 0), (CFG_B, 1), (CFG_C, 0), (CFG_C, 2)])
def test_routed_experts_alone(cfg, layer, dtype):
    f, d = cfg["layers"][layer]["mlp"], cfg["width"]
    W = plain.sub(make_weights(cfg, 13), f"l{layer}.mlp.")
    part = make_part("feed_forward", "routed_glu", routed_params(f, d), W, DTYPES[dtype])
    h = bf(torch.randn(160, d, generator=gen(15)))
    h = h[_without_ties(h, W, f)]
    assert h.shape[0] > 60
    want = plain.routed_experts(h.double(), dbl(W), f)
    hz = PartHarness(part)
    got = hz.feed("a", h)
    check_rows(got, want, dtype, what="routed experts")
    # one token at a time gives the same rows as the batch
    single = torch.cat([hz.feed("b", h[t:t + 1]) for t in range(6)], 0)
    assert rel_rows(single, got[:6]).max() <= (1e-5 if dtype == "float32" else 2e-2)


def test_the_routers_rule_shows():
    """Inputs made so that every clause of the rule decides something: the best output lies in a group that
    a correction closes; choice scores are negative, so a closed output (minus infinity) must not beat them;
    the weights are the scores without the correction and do not add up to one; an identity output is chosen."""
    d = 16
    r = {"experts": 4, "identity": 2, "top": 2, "groups": {"count": 3, "keep": 1}}
    f = {"kind": "moe", "router": r, "expert": {"ff": 8}}
    g = gen(41)
    W = {"router": torch.zeros(6, d), "correction": torch.tensor([-0.9, -0.9, -2.0, -2.0, -0.6, -0.7])}
    # logits: input entry e is output e's logit
    for e in range(6):
        W["router"][e, e] = 1.0
    for e in range(4):
        W[f"e{e}.gate"], W[f"e{e}.up"] = bf(torch.randn(8, d, generator=g)), bf(torch.randn(8, d, generator=g))
        W[f"e{e}.down"] = bf(torch.randn(d, 8, generator=g))
    h = torch.zeros(3, d)
    h[0, :6] = torch.tensor([0.0, 0.0, 3.0, 0.0, 1.0, 1.5])    # output 2 has the largest score, its group is closed
    h[1, :6] = torch.tensor([2.0, 1.0, 0.0, 0.0, 0.0, 0.0])    # group 0 wins: two real experts
    h[2, :6] = torch.tensor([0.0, 0.0, 0.0, 0.0, 0.0, 4.0])    # an identity output and its neighbour
    h[:, 6:] = bf(torch.randn(3, d - 6, generator=g))
    choice, weight = plain.route(h.double(), dbl(W), r)
    assert sorted(choice[0].tolist()) == [4, 5] and sorted(choice[1].tolist()) == [0, 1] and sorted(choice[2].tolist()) == [4, 5]
    assert float(weight.sum(-1).max()) < 0.999
    part = make_part("feed_forward", "routed_glu", routed_params(f, d), W, torch.float32)
    got = PartHarness(part).feed("a", h)
    want = plain.routed_experts(h.double(), dbl(W), f)
    assert rel_rows(got, want).max() < 1e-5
    # rows 0 and 2 use identity experts only: the output is the input times the two scores
    s = torch.softmax(h[2, :6].double(), -1)
    assert rel_rows(got[2:3], (s[4] + s[5]) * h[2:3].double()).max() < 1e-5


# ---------------------------------------------------------------------------
# whole models through the engine
# ---------------------------------------------------------------------------

_CACHE: dict = {}


def model_and_truth(name: str, dtype: str, lengths=(1, 2, 23, 61, 130)):
    """A model, some requests, and the plain implementation's logits for them."""
    key = (name, dtype)
    if key not in _CACHE:
        cfg, seed = CONFIGS[name]
        W, model = build(cfg, seed, dtype)
        reqs = {f"r{n}": ids_for(cfg, 100 + n, n) for n in lengths}
        tkey = ("truth", name)
        if tkey not in _CACHE:
            _CACHE[tkey] = {rid: plain.forward(cfg, W, ids).numpy() for rid, ids in reqs.items()}
        _CACHE[key] = (cfg, model, reqs, _CACHE[tkey])
    return _CACHE[key]


def engine_for(model, n_pages=64, page_size=16, max_requests=4, cap=512, **kw):
    from gibbs_b200 import Engine
    return Engine(model, n_pages=n_pages, page_size=page_size, max_requests=max_requests, max_step_tokens=cap,
                  max_context=cap, guard_cache=True, **kw)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_whole_decoded_and_cut_prompts_match_the_plain_implementation(name, dtype):
    cfg, model, reqs, truth = model_and_truth(name, dtype)
    eng = engine_for(model)
    assert eng.plan is not None, eng.plan_refusal
    for what, steps in (("whole", trace_whole(reqs)), ("decoded", trace_tail_decoded(reqs, tail=40)),
                        ("cut", trace_portions(reqs)), ("cut in twos", trace_portions(reqs, sizes=(2,)))):
        got = run_trace_on_engine(eng, steps)
        for rid in reqs:
            check_rows(got[rid], truth[rid], dtype, strict=False, what=f"{name} {what} {rid}")


@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_layer_by_layer_in_float32(name):
    """The residual stream after every layer, through the parts' forward methods."""
    cfg, model, reqs, _ = model_and_truth(name, "float32")
    W = make_weights(cfg, CONFIGS[name][1])
    ids = reqs["r61"]
    layers = []
    plain.forward(cfg, W, ids, layers_out=layers)
    eng = engine_for(model, use_plan=False, use_graphs=False)
    seen = []
    originals = [b.forward for b in model.blocks]
    try:
        for b, orig in zip(model.blocks, originals):
            def fw(x, step, caches, orig=orig):
                orig(x, step, caches)
                seen.append(x.tensor().clone())
            b.forward = fw
        from gibbs_b200 import StepEntry
        eng.open("x")
        eng.step([StepEntry("x", ids, [len(ids) - 1])])
        eng.close("x")
    finally:
        for b in model.blocks:
            del b.forward
    assert len(seen) == len(cfg["layers"])
    for i, x in enumerate(seen):
        assert rel_rows(x.cpu(), layers[i]).max() <= 1e-4, f"layer {i}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "D"])
def test_plan_and_forward_methods_give_the_same_bits(name, dtype):
    cfg, model, reqs, _ = model_and_truth(name, dtype)
    steps = trace_mixed(reqs, capacity_tokens=320, seed=3)
    a = run_trace_on_engine(engine_for(model, n_pages=20), steps)
    b = run_trace_on_engine(engine_for(model, n_pages=20, use_plan=False, use_graphs=False), steps)
    for rid in reqs:
        assert np.array_equal(a[rid], b[rid]), rid


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C", "D"])
def test_mixed_batches_with_pages_used_again(name, dtype):
    """Up to three live requests in a pool that holds little more than the live ones, portions beside
    single tokens: against the plain implementation, and against each request run alone."""
    cfg, model, reqs, truth = model_and_truth(name, dtype)
    more = dict(reqs)
    for k in range(4):                                        # the same lengths again: pages go round
        more[f"again{k}"] = ids_for(cfg, 500 + k, 40 + 17 * k)
    for seed in (0, 1):
        eng = engine_for(model, n_pages=20, max_requests=3)   # 320 tokens of pages
        got = run_trace_on_engine(eng, trace_mixed(more, capacity_tokens=320, max_live=3, seed=seed))
        assert eng.cache.free_pages() == [20] * len(eng.cache.groups)
        for rid in reqs:
            check_rows(got[rid], truth[rid], dtype, strict=False, what=f"{name} mixed {rid}")
        alone = run_trace_on_engine(engine_for(model), trace_whole(more))
        for rid in more:
            e = rel_rows(got[rid], alone[rid])
            lim = 1e-4 if dtype == "float32" else TOL[dtype]
            assert (e > lim).mean() <= (0.0 if dtype == "float32" else 0.45), f"{rid}: batch against alone {e.max():.3g}"


@pytest.mark.parametrize("seed", [2, 5, 8, 13, 21, 34, 55])
def test_random_configurations_in_float32(seed):
    """Sizes, options and the order of layers drawn at random (one to five layers; layers that read another
    layer's keys through a window of their own; windows of one token and none; one expert, all outputs chosen;
    groups; identity experts), whole, cut, decoded and in mixed batches.  Held to the plain implementation in
    float64, with room for a choice of experts that hangs on the last bits of a 32-bit softmax."""
    from gibbs_b200.config import parse_config
    from gibbs_b200.parts.model import build_model
    from gibbs_b200.weights import TensorDict
    cfg = random_config(seed)
    W = make_weights(cfg, seed)
    model = build_model(parse_config(cfg).plan(), TensorDict({k: v.to(torch.bfloat16) for k, v in W.items()}),
                        torch.float32, DEV)
    reqs = {f"r{n}": ids_for(cfg, seed * 7 + n, n) for n in (1, 2, 37, 90)}
    truth = {rid: plain.forward(cfg, W, ids).numpy() for rid, ids in reqs.items()}
    for what, steps in (("whole", trace_whole(reqs)), ("cut", trace_portions(reqs)),
                        ("decoded", trace_tail_decoded(reqs, tail=30)),
                        ("mixed", trace_mixed(reqs, capacity_tokens=256, max_live=3, seed=seed))):
        eng = engine_for(model, n_pages=16, max_requests=3, cap=256)
        got = run_trace_on_engine(eng, steps)
        for rid in reqs:
            e = rel_rows(got[rid], truth[rid])
            assert (e > 3e-4).mean() <= 0.02, f"{what} {rid}: {e.max():.3g} at row {int(e.argmax())}"


def test_long_decoding_past_windows_and_pages():
    """260 tokens decoded one by one after a two-token prompt: every window edge and page edge is passed
    by single tokens."""
    cfg, model, _, _ = model_and_truth("A", "float32")
    W = make_weights(cfg, CONFIGS["A"][1])
    ids = ids_for(cfg, 77, 262)
    truth = plain.forward(cfg, W, ids).numpy()
    eng = engine_for(model, n_pages=20)
    got = run_trace_on_engine(eng, trace_tail_decoded({"long": ids}, tail=260))
    e = rel_rows(got["long"], truth)
    assert e.max() <= TOL["float32"], f"first wrong position {int(np.nonzero(e > TOL['float32'])[0][0])}"
    assert min(eng.cache.free_pages()) == 20


def test_greedy_generation_through_the_scheduler():
    """Generator -> Scheduler -> Engine.step -> sampler: the tokens are those the plain implementation
    picks, fed back one by one; several prompts of unequal length at once."""
    from gibbs_b200 import Generator, SamplingParams
    cfg, model, _, _ = model_and_truth("B", "float32")
    W = make_weights(cfg, CONFIGS["B"][1])
    gen_ = Generator(model, ctx=256, page_size=16, n_pages=40, max_running=4, max_batch_tokens=48)
    prompts = [ids_for(cfg, 900 + k, n) for k, n in enumerate((3, 50, 19))]
    outs = gen_.generate(prompts, SamplingParams(max_new_tokens=12, temperature=0.0), stop_at_eos=False)
    for p, out in zip(prompts, outs):
        seq = list(p)
        for tok in out:
            logits = plain.forward(cfg, W, seq)[-1]
            top2 = torch.topk(logits, 2).values
            if float(top2[0] - top2[1]) > 1e-3:               # (no verdict on a tie)
                assert int(logits.argmax()) == tok, f"after {len(seq)} tokens"
            seq.append(tok)
        assert len(out) == 12


def test_command_line_from_a_configuration_to_tokens(tmp_path, capsys):
    """config.json -> random weights on disk -> --arch-dump, --probe-top5 and a greedy continuation, all
    through the command line's own entry point."""
    import json
    from gibbs_b200.engine.cli import main
    cfg_path = tmp_path / "cfg.json"
    cfg_path.write_text(json.dumps(CFG_A))
    folder = tmp_path / "model"
    assert main(["--random", str(cfg_path), "--save", str(folder), "--seed", "3", "--dtype", "float32"]) == 0
    capsys.readouterr()
    assert main(["-m", str(folder), "--arch-dump"]) == 0
    dump = json.loads(capsys.readouterr().out)
    assert dump["architecture"] == "Petelix"
    prompt = ids_for(CFG_A, 5, 9)
    ids = ",".join(map(str, prompt))
    assert main(["-m", str(folder), "--dtype", "float32", "--probe-top5", ids, "--ctx", "128"]) == 0
    top = json.loads(capsys.readouterr().out)
    from gibbs_b200.weights import Checkpoint
    ck = Checkpoint(folder)
    W = {n: ck.tensor(n) for n in ck.names()}
    logits = plain.forward(CFG_A, W, prompt)[-1]
    assert top["ids"][0] == int(logits.argmax())
    assert abs(top["logits"][0] - float(logits.max())) < 1e-3
    assert main(["-m", str(folder), "--dtype", "float32", "--prompt-ids", ids, "--max-tokens", "5", "--temperature", "0",
                 "--ctx", "128"]) == 0
    out = capsys.readouterr().out
    generated = [int(t) for t in out.split("Output:\n")[1].splitlines()[0].split(",")]
    assert len(generated) == 5 and generated[0] == top["ids"][0]


# launches of 48 tiles of 64 rows (the smallest on tcgen05) and of many: windows within a key tile and across tiles, groups that do not divide 128, pages of 8 to
# 64, a single token beside portions, two maps, the edges of 64 keys, blocks of positions, no softmax
@pytest.mark.parametrize("heads,kvh,maps,vdim,ps,window,cap,sink,gate,sig,starts,lens,blocked", [
    (16, 4, 1, 64, 16, 0, 30.0, True, True, False, [0, 63], [1000, 230], False),
    (32, 8, 1, 64, 16, 100, 30.0, True, False, False, [0, 1000, 64], [433, 1, 260], False),
    (24, 8, 1, 128, 8, 64, 0.0, False, False, False, [127, 65], [800, 7], False),
    (20, 4, 2, 128, 64, 1, 0.0, True, False, False, [0, 5], [300, 300], False),
    (16, 4, 2, 128, 32, 193, 0.0, False, False, False, [1000], [677], False),
    (16, 4, 1, 64, 16, 0, 0.0, False, False, True, [3, 0], [640, 700], False),
    (8, 8, 1, 64, 16, 40, 5.0, False, True, True, [0], [2500], False),
    (16, 4, 2, 128, 16, 100, 0.0, False, False, False, [150, 0], [500, 230], True), (32, 8, 1, 64, 16, 64, 20.0, True, True, False, [37], [700], True),
    (16, 4, 2, 128, 32, 1024, 0.0, False, False, False, [0, 1000], [300, 377], True),
    (16, 4, 1, 64, 16, 0, 30.0, True, True, False, [0], [176], False), (32, 8, 1, 128, 16, 0, 0.0, False, False, False, [0, 0], [65, 1], False),
    (8, 8, 1, 64, 16, 0, 0.0, False, False, True, [70], [321], False),
])
def test_tensor_core_attention_of_portions(heads, kvh, maps, vdim, ps, window, cap, sink, gate, sig, starts, lens, blocked):
    _portions_against_float64(heads, kvh, maps, vdim, ps, window, cap, sink, gate, sig, starts, lens, blocked)


# more requests than a warp has lanes, short portions beside long ones
@pytest.mark.parametrize("heads,kvh,vdim,window,sig,starts,lens", [
    (16, 4, 64, 0, False, [40 * (r % 5) for r in range(70)], [1 + 7 * r % 50 for r in range(70)]),
    (8, 8, 128, 30, False, [r for r in range(33)], [130 - 4 * r for r in range(32)] + [1]),
    (32, 8, 64, 0, True, [0] * 32 + [500], [40] * 32 + [77]),
])
def test_tensor_core_attention_of_many_portions(heads, kvh, vdim, window, sig, starts, lens):
    _portions_against_float64(heads, kvh, 1, vdim, 16, window, 0.0, False, False, sig, starts, lens, False)


class _Pages:
    """One request's keys and values on shuffled pages, and the attention of its last ``n`` tokens (or of some of them)."""

    def __init__(self, heads, kvh, vdim, start, n, one_sign=False):
        self.heads, self.kvh, self.vdim, self.start, self.n, self.ps, ctx = heads, kvh, vdim, start, n, 16, start + n
        self.n_pages = -(-ctx // self.ps) + 2
        self.table = torch.randperm(self.n_pages)[:self.n_pages - 2].int().cuda()[None].contiguous()
        self.q = (torch.randn(n, heads * 64, device="cuda") * 0.5).bfloat16()
        self.k = torch.randn(self.n_pages, kvh, self.ps, 64, device="cuda").bfloat16()
        v = torch.randn(self.n_pages, kvh, self.ps, vdim, device="cuda")
        self.v = (1 + v.abs() if one_sign else v).bfloat16()

    def at(self, positions):
        """(pages, rows) of positions."""
        i = torch.as_tensor(positions, device="cuda")
        return self.table[0].long()[i // self.ps], i % self.ps

    def attend(self, window=0, sig=False, blocked=False, first=0, n=None, v=None, cap=0.0):
        from gibbs_b200.ops import hybrid
        n, v = self.n - first if n is None else n, self.v if v is None else v
        i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
        out = torch.empty(n, self.heads * self.vdim, device="cuda")
        q, bias = self.q[first:first + n].contiguous(), torch.zeros(self.heads, device="cuda")
        req, pos, at = i32([0] * n), i32(list(range(self.start + first, self.start + first + n))), i32([0])
        hybrid.call("sigmoid_attention_tc" if sig else "sink_attention_tc",
                    [q.data_ptr(), self.k.data_ptr(), v.data_ptr(), self.table.data_ptr(), self.table.shape[1], self.ps, self.n_pages, req.data_ptr(),
                     pos.data_ptr(), 0, 0, out.data_ptr(), out.stride(0), n, self.heads, self.kvh, 64, self.vdim, window, self.start + self.n, 0, 1,
                     at.data_ptr(), bias.data_ptr() if sig else 0], [0.125, cap, 1.0 if sig else 0.0], flags=2 | (4 if blocked else 0) | 1 << 8)
        return out.reshape(n, self.heads, self.vdim)


# portions whose own later tokens, and positions that a window has passed for some rows, have values that are not finite
@pytest.mark.parametrize("vdim,start,n,window,sig,blocked,odd", [
    (64, 0, 400, 0, False, False, [17, 63, 64, 200, 399]), (128, 100, 300, 0, True, False, [130, 131, 250]), (64, 5, 500, 70, False, False, [3, 40, 300]),
    (128, 5, 500, 200, False, False, [150, 504]), (64, 0, 400, 128, True, True, [130, 255, 256]), (64, 4500, 300, 0, False, False, [4490, 4600, 4700]),
])
def test_values_that_are_not_finite_stay_with_the_rows_that_see_them(vdim, start, n, window, sig, blocked, odd):
    torch.manual_seed(vdim + n)
    a = _Pages(16, 4, vdim, start, n)
    want = a.attend(window, sig, blocked)
    v = a.v.clone()
    what = [float("inf"), float("nan"), float("-inf")]
    for i, pos in enumerate(odd):
        page, row = a.at(pos)
        v[page, i % 4, row, 7 * i % vdim] = what[i % 3]
    got = a.attend(window, sig, blocked, v=v)
    pos = torch.arange(start, start + n, device="cuda")
    first = pos * 0 if not window else pos // window * window if blocked else pos - window + 1
    touched = torch.zeros(n, 16, vdim, dtype=torch.bool, device="cuda")
    for i, o in enumerate(odd):
        touched[(pos >= o) & (first <= o), 4 * (i % 4):4 * (i % 4) + 4, 7 * i % vdim] = True
    assert not torch.isfinite(got[touched]).any()
    # (rows that met such a value are worked out again, in 32-bit and in another order: what the weights' 16 bits and the sums allow twice)
    size = a.attend(window, sig, blocked, v=a.v.abs())
    assert ((got - want).abs() <= 2.0 ** -14.5 * size + 1e-6)[~touched].all()


# contexts of thousands of keys, values of one sign, so that truncated sums show: no further off than the kernel of 64-row tiles, which fewer tokens
# at a time bring into play
@pytest.mark.parametrize("vdim,sig,cap", [(64, False, 0.0), (128, False, 20.0), (64, True, 0.0), (128, True, 0.0)])
@pytest.mark.parametrize("ctx", [2048, 4096, 8192, 16300])
def test_long_contexts_lose_no_precision(vdim, sig, cap, ctx):
    torch.manual_seed(ctx + vdim)
    n = 256
    a = _Pages(16, 4, vdim, ctx - n, n, one_sign=True)
    got, other = a.attend(0, sig, cap=cap), torch.cat([a.attend(0, sig, first=t, n=64, cap=cap) for t in range(0, n, 64)])
    err = [0.0, 0.0]
    page, row = a.at(list(range(ctx)))
    k, v = (x[page, :, row].double().repeat_interleave(4, 1) for x in (a.k, a.v))
    for t in range(0, n, 64):
        s = torch.einsum("thd,khd->thk", a.q[t:t + 64].double().reshape(64, 16, 64), k) * 0.125
        s = cap * torch.tanh(s / cap) if cap else s
        seen = torch.arange(ctx, device="cuda")[None] <= torch.arange(ctx - n + t, ctx - n + t + 64, device="cuda")[:, None]
        w = torch.sigmoid(s).masked_fill(~seen[:, None], 0.0) if sig else torch.softmax(s.masked_fill(~seen[:, None], -math.inf), 2)
        want = torch.einsum("thk,khd->thd", w, v)
        for i, x in enumerate((got, other)):
            err[i] += ((x[t:t + 64].double() - want) / want).pow(2).mean().item() / (n // 64)
    err = [e ** 0.5 for e in err]
    assert err[0] <= 1.001 * err[1] and err[0] < 2e-5, err


def _portions_against_float64(heads, kvh, maps, vdim, ps, window, cap, sink, gate, sig, starts, lens, blocked):
    from gibbs_b200.ops import hybrid
    torch.manual_seed(heads * 1000 + window)
    dk, n, group = 64, sum(lens), heads // kvh
    need = [(a + b + ps - 1) // ps for a, b in zip(starts, lens)]
    n_pages, first = sum(need) + 3, [sum(lens[:r]) for r in range(len(lens))]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    perm = torch.randperm(n_pages).tolist()
    bt = torch.zeros(len(lens), max(need), dtype=torch.int32)
    for r, k in enumerate(need):
        bt[r, :k] = torch.tensor(perm[sum(need[:r]):sum(need[:r]) + k])
    q = torch.randn(n, heads * maps * dk, device="cuda").bfloat16()
    kp, vp = torch.randn(n_pages, kvh, ps, maps * dk, device="cuda").bfloat16(), torch.randn(n_pages, kvh, ps, vdim, device="cuda").bfloat16()
    # what no row sees is not finite: the rest of every last page, and what lies in front of a window
    for r, (a, b) in enumerate(zip(starts, lens)):
        at = torch.arange(need[r] * ps)
        at = at[(at >= a + b) | (at < (a // window * window if blocked else a - window + 1 if window else 0))]
        vp[bt[r][at // ps].long().cuda(), :, (at % ps).cuda()] = float("nan")
        kp[bt[r][at // ps].long().cuda(), :, (at % ps).cuda()] = float("inf")
    logits = torch.randn(n, heads * vdim, device="cuda") if gate else None
    score, scale, factor = torch.randn(heads, device="cuda"), 0.3, 1.5
    out = torch.full((n, heads * maps * vdim + 8), 7.0, device="cuda")
    tables, tok_req, starts_, pos = (bt.cuda(), i32([r for r, b in enumerate(lens) for _ in range(b)]), i32(first),
                                     i32([a + i for a, b in zip(starts, lens) for i in range(b)]))
    hybrid.call("sigmoid_attention_tc" if sig else "sink_attention_tc",
                [q.data_ptr(), kp.data_ptr(), vp.data_ptr(), tables.data_ptr(), bt.shape[1], ps, n_pages, tok_req.data_ptr(), pos.data_ptr(),
                 logits.data_ptr() if gate else 0, logits.stride(0) if gate else 0, out.data_ptr(), out.stride(0), n, heads, kvh, dk, vdim, window,
                 max(a + b for a, b in zip(starts, lens)), 0, len(lens), starts_.data_ptr(), score.data_ptr() if sink or sig else 0],
                [scale, cap, factor if sig else 0.0], flags=(1 if sink else 0) | 2 | (4 if blocked else 0) | maps << 8)
    assert (out[:, heads * maps * vdim:] == 7.0).all()
    got = out[:, :heads * maps * vdim].reshape(n, heads, maps, vdim).double()
    for r, (a, b) in enumerate(zip(starts, lens)):
        rows, idx, at = slice(first[r], first[r] + b), torch.arange(a + b, device="cuda"), torch.arange(a, a + b, device="cuda")
        pages = tables[r].long()[idx // ps]
        seen = idx[None] <= at[:, None]
        if window:
            seen &= idx[None] >= (at // window * window if blocked else at - window + 1)[:, None]
        k = kp[pages, :, idx % ps].double().reshape(a + b, kvh, maps, dk).repeat_interleave(group, 1)
        v = vp[pages, :, idx % ps].double().repeat_interleave(group, 1)
        v = torch.where(seen.any(0)[:, None, None], v, torch.zeros_like(v))
        s = torch.einsum("thmd,khmd->thmk", q[rows].double().reshape(b, heads, maps, dk), k) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if sig:
            w = torch.sigmoid(s + score.double()[None, :, None, None]).masked_fill(~seen[:, None, None], 0.0) * factor
        else:
            s = s.masked_fill(~seen[:, None, None], -math.inf)
            z = score.double()[None, :, None, None].expand(b, heads, maps, 1)
            w = torch.softmax(torch.cat([s, z], 3), 3)[..., :-1] if sink else torch.softmax(s, 3)
        want, size = torch.einsum("thmk,khd->thmd", w, v), torch.einsum("thmk,khd->thmd", w, v.abs())
        if gate:
            o = torch.sigmoid(logits[rows].double()).reshape(b, heads, 1, vdim)
            want, size = want * o, size * o
        # weights of 16 bits (2^-17), scores of up to 30 formed and rounded in 32-bit a few times (2^-16 of a weight at most), sums
        # that the tensor core truncates (160 terms of 2^-24)
        assert ((got[rows] - want).abs() <= 2.0 ** -14.5 * size + 1e-6).all(), r


# experts of many rows on CTA pairs (edges of 32 and 256 rows, empty experts, weight rows that are no whole tiles, as many experts as
# the kernel takes) and of few
@pytest.mark.parametrize("E,K,out,mode,counts", [
    (4, 64, 64, 0, [256, 257, 0, 33]), (3, 136, 448, 0, [1, 512, 700]), (5, 512, 256, 0, [129, 128, 127, 300, 31]),
    (4, 64, 130, 1, [256, 257, 0, 33]), (3, 136, 448, 1, [1, 512, 700]), (2, 1024, 2048, 1, [300, 96]),
    (3, 200, 320, 2, [64, 300, 200]), (1, 64, 64, 1, [2500]), (128, 64, 64, 0, [64] * 127 + [200]),
    (5, 512, 256, 0, [1, 0, 3, 16, 17]), (40, 512, 256, 1, [0] * 38 + [2, 1]), (3, 136, 448, 0, [60, 0, 64]),
])
def test_routed_experts_products_of_many_rows_and_of_few(E, K, out, mode, counts):
    _routed_experts_product(E, K, out, mode, counts)


# CTA pairs with tiles cut to 32, 64 and 128 rows because there are few, and whole ones on the other side of a round of 74; a function's outputs
# stored two at a time and, where their number or stride is odd, one at a time; plain outputs at the line from which pairs take them and below it
@pytest.mark.parametrize("E,K,out,mode,counts", [
    (1, 64, 64, 0, [40]), (2, 72, 64, 0, [300, 1]), (8, 64, 128, 0, [0, 0, 700, 0, 0, 0, 0, 1]), (37, 64, 128, 0, [64] * 37), (38, 64, 256, 0, [70] * 38),
    (3, 200, 321, 2, [64, 300, 200]), (1, 64, 2, 2, [33]), (5, 136, 130, 2, [31, 32, 33, 0, 257]), (4, 64, 1024, 2, [1000, 3, 0, 200]),
    (128, 512, 130, 1, [128] * 126 + [129, 127]), (128, 512, 130, 1, [128] * 126 + [128, 127]), (64, 512, 448, 1, [0, 257] * 32),
    (16, 1024, 512, 1, [960] * 16),
])
def test_routed_experts_products_at_the_edges_of_their_dispatch(E, K, out, mode, counts):
    _routed_experts_product(E, K, out, mode, counts)


def _routed_experts_product(E, K, out, mode, counts):
    from gibbs_b200.ops import hybrid
    torch.manual_seed(K + out)
    rows, per = sum(counts), (2 * out if mode == 0 else out)
    room = rows + 5
    x = torch.randn(room, K, device="cuda").bfloat16()
    x[rows:] = float("nan")                                    # rows behind the last expert's
    w = (torch.randn(E, per, K, device="cuda") / K ** 0.5).bfloat16()
    off = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device="cuda")
    y = torch.full((room, out + 8), 7.0, device="cuda", dtype=torch.float32 if mode == 1 else torch.bfloat16)
    hybrid.call("moe_experts_tc", [x.data_ptr(), K, room, w.data_ptr(), 0, off.data_ptr(), E, y.data_ptr(), y.stride(0), rows, out, K, mode, 1, 4],
                [1.702, 7.0, 1.0] if mode == 0 else [0.0, 0.0, 0.0])
    assert (y[:, out:] == 7.0).all() and (y[rows:] == 7.0).all()
    at = 0
    for e, c in enumerate(counts):
        if c == 0:
            continue
        z, size = x[at:at + c].double() @ w[e].double().T, x[at:at + c].double().abs() @ w[e].double().abs().T
        ulp = K * 2.0 ** -24                                   # (of every term of a sum that is truncated K times at most)
        if mode == 0:
            z, size = z.reshape(c, -1, 2, 64), size.reshape(c, -1, 2, 64)
            g, u = z[:, :, 0].reshape(c, -1).clamp(max=7.0), z[:, :, 1].reshape(c, -1).clamp(-7.0, 7.0)
            want = g * torch.sigmoid(1.702 * g) * (u + 1.0)
            # (the unit grows by at most 8 x 1.1 times what g does, and by 7 times what u does)
            tol = 9 * ulp * size.sum(2).reshape(c, -1) + 2.0 ** -8 * want.abs()
        elif mode == 2:
            want = z.clamp(min=0.0) ** 2
            tol = 2 * z.abs() * ulp * size + (ulp * size) ** 2 + 2.0 ** -8 * want
        else:
            want, tol = z, ulp * size
        err = (y[at:at + c, :out].double() - want).abs()
        assert (err <= tol + 1e-9).all(), (e, (err - tol).max().item())
        at += c


@pytest.mark.parametrize("cfg,layer", [(CFG_D, 0), (CFG_D, 2), (CFG_D, 3), (CFG_D, 4)])
def test_tensor_core_attention_against_the_generic_kernel(cfg, layer, monkeypatch):
    """In bfloat16 the two kernels read the same pages; they differ by the rounding of the queries and of
    the weights' second term only.  A long request, cut so that tiles hold a few rows and many."""
    from gibbs_b200.parts import gated_attention as ga
    m, d, eps = cfg["layers"][layer]["mixer"], cfg["width"], cfg["norm"]["eps"]
    W = plain.sub(make_weights(cfg, 5), f"l{layer}.mix.")
    T = 330
    h = bf(torch.randn(T, d, generator=gen(8)))
    want = _plain_mixer(h, W, m, eps)
    outs = {}
    for on in (True, False):
        monkeypatch.setattr(ga, "USE_TENSOR_CORES", on)
        part = make_part("mixer", "gated_attention", attention_params(m, d, eps), W, torch.bfloat16)
        hz = PartHarness(part, n_pages=24, page_size=16, fill=0.0)
        outs[on] = hz.run_cut("r", h, [150, 3, 1, 1, 90, 1, 64, 2, 1])
        check_rows(outs[on], want, "bfloat16", what=f"tensor cores {on}")
    assert rel_rows(outs[True], outs[False]).max() < 1.5e-2


@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("longest,vdim", [(300, 40), (4100, 33), (20000, 64), (20000, 256)])
def test_chunks_of_keys_are_merged_whatever_their_number(longest, vdim, sink):
    """Contexts that fill one chunk, some or nearly all of 2 to 79 (an upper bound on the context decides), the others
    empty, against 64 bits: a score is off by (dim + 4) 2^-24 scale |q|.|k| at most, a weight by exp of twice that and
    2^-20, the sums by (keys + chunks + 64) 2^-24."""
    from gibbs_b200.ops import hybrid, library
    torch.manual_seed(longest + vdim)
    H, G, dim, ps, pos = 4, 2, 16, 16, [0, 299, 255 if longest == 300 else 2500]
    n, blocks = len(pos), max(pos) // 16 + 1
    kp, vp = torch.randn(n * blocks, G, ps, dim), torch.randn(n * blocks, G, ps, vdim)
    table = torch.randperm(n * blocks).reshape(n, blocks)
    q, gate = torch.randn(n, H * dim), torch.randn(n, H * vdim)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lib = library("hybrid")
    ws = torch.full((lib.gb_sink_attention_workspace_rows(), vdim + 2), float("nan"), device=DEV)
    dev = [t.to(DEV) for t in (q, kp, vp, gate)]
    ints = [i32(table.tolist()), i32(list(range(n))), i32(pos)]
    out = torch.full((n, H * vdim), float("nan"), device=DEV)
    scale = dim ** -0.5
    launched = hybrid.call("sink_attention", [dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), ints[0].data_ptr(), blocks, ps,
                                              n * blocks, ints[1].data_ptr(), ints[2].data_ptr(), dev[3].data_ptr(), H * vdim,
                                              out.data_ptr(), H * vdim, n, H, G, dim, vdim, 0, longest, ws.data_ptr()],
                           [scale, 0.0, 0.0], flags=1 if sink else 0)
    assert launched == 2                                 # (the attention and the merge)
    for t in range(n):
        j = torch.arange(pos[t] + 1)
        for h in range(H):
            k, v = kp[table[t][j // ps], h // 2, j % ps].double(), vp[table[t][j // ps], h // 2, j % ps].double()
            qh = q[t, h * dim:(h + 1) * dim].double()
            sc = k @ qh * scale
            w = torch.softmax(torch.cat([sc, torch.zeros(1, dtype=F64)]) if sink else sc, 0)[:len(j)]
            f = torch.sigmoid(gate[t, h * vdim:(h + 1) * vdim].double())
            d = (dim + 4) * 2.0 ** -24 * scale * float((k.abs() @ qh.abs()).max())
            tol = (2 * (2 * d + 2.0 ** -20) + (len(j) + 79 + 64) * 2.0 ** -24) * (w @ v.abs()) * f
            err = (out[t, h * vdim:(h + 1) * vdim].double().cpu() - (w @ v) * f).abs()
            assert (err <= tol).all(), (t, h)


def test_a_chunk_whose_factor_is_zero_still_counts_where_its_sum_is_no_number():
    """The last key's score is 200 above all others, so the first chunks' factors are 0 in 32 bits; a value that is no
    number (or infinite) in one of them makes its column none, as in one chunk and in 64 bits."""
    from gibbs_b200.ops import hybrid, library
    H, G, dim, vdim, ps, L = 4, 2, 16, 40, 16, 4100
    blocks = L // ps + 1
    q = torch.zeros(1, H * dim, device=DEV)
    q[:, ::dim] = 20.0
    kp, vp = torch.randn(blocks, G, ps, dim, device=DEV), torch.randn(blocks, G, ps, vdim, device=DEV)
    kp[..., 0] = 0.0
    kp[(L - 1) // ps, :, (L - 1) % ps, 0] = 10.0
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lib = library("hybrid")
    ws = torch.empty(lib.gb_sink_attention_workspace_rows(), vdim + 2, device=DEV)
    table, req, pos = i32([list(range(blocks))]), i32([0]), i32([L - 1])
    for value in (float("nan"), float("inf")):
        vp[3, :, 5, 7] = value
        out = torch.zeros(1, H * vdim, device=DEV)
        launched = hybrid.call("sink_attention", [q.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(), blocks, ps, blocks, req.data_ptr(),
                                                  pos.data_ptr(), 0, 0, out.data_ptr(), H * vdim, 1, H, G, dim, vdim, 0, L, ws.data_ptr()],
                               [1.0, 0.0, 0.0])
        assert launched == 2
        bad = out.view(H, vdim).isnan()
        assert bad[:, 7].all() and int(bad.sum()) == H


@pytest.mark.parametrize("splits,vdim", [(2, 8), (3, 33), (4, 128), (6, 200)])
@pytest.mark.parametrize("sink", [0, 1])
def test_merge_by_a_block_and_by_a_warp_a_row_has_the_same_bits(splits, vdim, sink):
    """Steps on both sides of the number of rows (128 a chunk) from which a warp takes a row; contexts that leave chunks empty."""
    from gibbs_b200.ops import hybrid, library
    torch.manual_seed(vdim)
    H, G, dim, ps, longest = 16, 2, 16, 16, 256 * splits
    n, blocks = 8 * splits, longest // 16
    q, gate = torch.randn(n, H * dim, device=DEV), torch.randn(n, H * vdim, device=DEV)
    kp, vp = torch.randn(blocks, G, ps, dim, device=DEV), torch.randn(blocks, G, ps, vdim, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lib = library("hybrid")
    import ctypes
    chunk, got = ctypes.c_int(0), {}
    ws = torch.empty(lib.gb_sink_attention_workspace_rows(), vdim + 2, device=DEV)
    for k in (n - 1, n):                                     # n * H = 128 * splits is the first launch by warps
        assert lib.gb_sink_attention_chunks(k, H, G, 0, longest, ctypes.byref(chunk)) == splits
        table, req, pos = i32([list(range(blocks))] * k), i32(list(range(k))), i32([(97 * i) % longest for i in range(k)])
        out = torch.full((k, H * vdim), float("nan"), device=DEV)
        launched = hybrid.call("sink_attention", [q.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(), blocks, ps, blocks, req.data_ptr(), pos.data_ptr(),
                                                  gate.data_ptr(), H * vdim, out.data_ptr(), H * vdim, k, H, G, dim, vdim, 0, longest, ws.data_ptr()],
                               [dim ** -0.5, 0.0, 0.0], flags=sink)
        assert launched == 2
        got[k] = out
    assert not got[n].isnan().any() and torch.equal(got[n - 1], got[n][:n - 1])


@pytest.mark.parametrize("H,G,dim,vdim,maps", [(1, 1, 16, 8, 1), (4, 2, 40, 24, 1), (32, 8, 64, 64, 1), (9, 3, 64, 96, 2), (70, 7, 32, 32, 1), (8, 8, 300, 64, 1)])
@pytest.mark.parametrize("flags", [0, 1, 8, 8 | 16, 32])
def test_queries_and_keys_have_the_same_bits_in_a_step_of_few_tokens_and_of_many(H, G, dim, vdim, maps, flags):
    """One token, 64 (the last step with several blocks a token and a table of angles) and 65: queries, keys and values, with
    every norm and both ways of pairing; more angles than the table holds; and the first token against 64 bits."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(dim + flags)
    ps, ld = 16, (H + G) * maps * dim + G * vdim
    rot = dim // 2 * 2
    x, qg, kg = torch.randn(65, ld, device=DEV), torch.randn(H * maps * dim, device=DEV), torch.randn(G * maps * dim, device=DEV)
    inv = torch.rand(rot // 2 + 1, device=DEV)
    inv[-1] = 1.25
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table, pos, whole = i32([[i] for i in range(65)]), [(7 * i + 3) % ps for i in range(65)], None
    for n in (65, 64, 1):
        kp, vp = torch.zeros(65, G, ps, maps * dim, device=DEV), torch.zeros(65, G, ps, vdim, device=DEV)
        out, req, at = torch.empty(n, H * maps * dim, device=DEV), i32(list(range(n))), i32(pos[:n])
        hybrid.call("qk_prep", [x.data_ptr(), ld, H * maps * dim, (H + G) * maps * dim, qg.data_ptr(), kg.data_ptr(), inv.data_ptr(), rot,
                                req.data_ptr(), at.data_ptr(), table.data_ptr(), 1, ps, kp.data_ptr(), vp.data_ptr(), 65, n, H, G, dim, vdim,
                                out.data_ptr(), maps], [1e-5, 0.0, 0.0], flags=flags)
        got = torch.cat([out, kp[:n].flatten(1), vp[:n].flatten(1)], 1)
        whole = got if whole is None else whole
        assert torch.equal(got, whole[:n]), n
    v = x[0, :H * maps * dim].double().view(H * maps, dim)
    if flags & 1:
        v = (v / (v.pow(2).mean() + 1e-5).sqrt()) * qg.double().view_as(v)
    if flags & 8:
        v = v / (v.pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * qg[:dim].double()
    ang = (pos[0] * inv[:-1]).double()                       # (the angle is formed in 32 bits)
    c, s = torch.cos(ang) * 1.25, torch.sin(ang) * 1.25
    a, b = (v[:, :rot // 2], v[:, rot // 2:rot]) if flags & 16 else (v[:, 0:rot:2], v[:, 1:rot:2])
    u, w = a * c - b * s, b * c + a * s
    turned = torch.cat([u, w], 1) if flags & 16 else torch.stack([u, w], 2).flatten(1)
    turned = torch.cat([turned, v[:, rot:]], 1)
    if flags & 32:
        turned = turned / (turned.pow(2).mean(1, keepdim=True) + 1e-5).sqrt()
    assert rel_rows(whole[0, :H * maps * dim].double().view(H * maps, dim).cpu(), turned.cpu()).max() < 2e-6

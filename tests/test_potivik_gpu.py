"""The Potivik design on the GPU against the plain implementation
(tests/plain_potivik.py): every mechanism alone, then whole models through the
engine's step function, cut and batched in every way, then greedy generation
through the scheduler.

Where both compute dtypes run: float32 must match every row; in bfloat16 a
router choice at a near tie may flip under the rounding of the router's
input, which changes that token's row (and, faintly, later ones), so whole
models with routed experts are held to "nearly all rows" there.  Mechanisms
alone have no such ties and are held to every row in both.
"""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import plain_potivik as plain
from helpers import run_trace_on_engine, trace_mixed, trace_portions, trace_tail_decoded, trace_whole
from potivik_helpers import CFG_A, CFG_B, CONFIGS, PartHarness, build, ids_for, make_part, make_weights, rel_rows

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-4, "bfloat16": 4e-2}
DEV = "cuda:0"


def gen(seed):
    return torch.Generator().manual_seed(seed)


def bf(t):
    return t.to(torch.bfloat16).to(torch.float32)


def check_rows(got, want, dtype: str, strict: bool = True, what: str = ""):
    e = rel_rows(got, want)
    if strict or dtype == "float32":
        assert e.max() <= TOL[dtype], f"{what}: row {int(e.argmax())} differs by {e.max():.3g} (tolerance {TOL[dtype]})"
    else:
        # (measured: a flipped choice shows in up to a third of a short request's rows; the median stays at 1.4e-2)
        frac = float((e > TOL[dtype]).mean())
        assert frac <= 0.45 and np.median(e) <= 0.75 * TOL[dtype], \
            f"{what}: {frac:.1%} of the rows differ by more than {TOL[dtype]} (median {np.median(e):.3g})"


# ---------------------------------------------------------------------------
# mechanisms alone
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kind,ref", [("layernorm", plain.layer_norm), ("rmsnorm_rows", plain.rms_norm)])
def test_norm_in_front_and_behind(kind, ref, dtype):
    g = gen(1)
    dim = 200
    x = torch.randn(37, dim, generator=g) * 3 + 1.5          # a mean far from zero: the variance is of deviations
    y = torch.randn(37, dim, generator=g) * 0.01 + 4.0
    w = 1 + 0.2 * torch.randn(dim, generator=g)
    part = make_part("norm", kind, {"dim": dim, "eps": 1e-5}, {"weight": w}, DTYPES[dtype])
    xd = x.to(DEV)
    out = part.forward(xd).float().cpu()
    check_rows(out, ref(x.double(), w.double(), 1e-5), dtype, what="norm")
    rows = torch.tensor([5, 0, 36, 5], dtype=torch.int32, device=DEV)
    out = part.forward(xd, rows=rows).float().cpu()
    check_rows(out, ref(x.double(), w.double(), 1e-5)[[5, 0, 36, 5]], dtype, what="gathered rows")
    # behind a sublayer: x += norm(y) * w, always in 32-bit
    from gibbs_b200.engine.step import StepState
    from gibbs_b200.parts.runner import Eager
    z = torch.zeros(1, dtype=torch.int32, device=DEV)
    step = StepState(37, 1, 0, z, z, z, z, z, z, z, z, z)
    part.add_normed(Eager(part.rt, step), xd, y.to(DEV))
    want = x.double() + ref(y.double(), w.double(), 1e-5)
    assert rel_rows(xd.cpu(), want).max() < 2e-5


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("f", [40, 128])      # 128: in bfloat16 the unit runs in the epilogue of the gate/up product
def test_clamped_unit_alone(dtype, f):
    g = gen(2)
    d, limit = 64, 0.7
    W = {k: bf(torch.randn(*s, generator=g) * 0.3) for k, s in (("gate", (f, d)), ("up", (f, d)), ("down", (d, f)))}
    part = make_part("feed_forward", "clamped_glu", {"hidden": d, "inner": f, "limit": limit}, W, DTYPES[dtype])
    h = bf(torch.randn(50, d, generator=g) * 2)               # many pre-activations beyond the clamps, on both sides
    hz = PartHarness(part)
    got = hz.feed("a", h)
    want = plain.clamped_glu(h.double(), W["gate"].double(), W["up"].double(), W["down"].double(), limit)
    check_rows(got, want, dtype, what="clamped unit")
    assert (h @ W["gate"].T > limit).any() and (h @ W["up"].T < -limit).any()


def _attention_params(m, d):
    return {"hidden": d, "heads": m["heads"], "dim": m["dim"], "rot_dim": m["rot_dim"], "vdim": m["vdim"],
            "kv_rank": m["kv_rank"], "scale": m["scale"], "window": (m.get("mask") or {}).get("size"),
            "rot_base": m["rot"]["base"], "rot_dims": m["rot"].get("dims", m["rot_dim"]), "eps": 1e-5}


def _mixer_weights(cfg, layer, seed):
    W = make_weights(cfg, seed)
    return plain.sub(W, f"l{layer}.mix.")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg,layer", [(CFG_A, 0), (CFG_A, 3), (CFG_B, 1)])
def test_latent_attention_alone_whole_cut_and_decoded(cfg, layer, dtype):
    m, d = cfg["layers"][layer]["mixer"], cfg["width"]
    W = _mixer_weights(cfg, layer, 5)
    part = make_part("mixer", "latent_attention", _attention_params(m, d), W, DTYPES[dtype])
    T = 150
    h = bf(torch.randn(T, d, generator=gen(6)))
    want = plain.latent_attention(h.double(), m, {k: v.double() for k, v in W.items()}, 1e-5)
    hz = PartHarness(part, n_pages=12, page_size=16)          # 12 pages: 192 positions, pages come back and go out again
    for rid, cuts in (("whole", [T]), ("cut", [2, 3, 17, 2, 31, 16, 1, 5, 64, 7]), ("decoded", [T - 45, 1])):
        got = hz.run_cut(rid, h, cuts)
        check_rows(got, want, dtype, what=f"latent attention, {rid}")
        hz.close(rid)


@pytest.mark.parametrize("H,r,dr", [(1, 8, 0), (3, 24, 8), (8, 64, 40), (5, 136, 8), (16, 256, 32), (33, 320, 0), (16, 512, 64)])
@pytest.mark.parametrize("window", [0, 1, 31, 33, 200])
def test_latent_attention_with_whole_weights_is_as_exact_as_the_generic_kernel(H, r, dr, window):
    """The tensor-core kernel for windows and single tokens against 64-bit arithmetic on the same pages: portions that
    end inside row tiles, key tiles and pages, single tokens, both in one step, chunked and not.  A score is off by at
    most d = (r + dr + 16) 2^-24 scale |q|.|c| (its sum is cut into terms of three sizes and four quarters), a weight
    by exp(2 d + 2^-20), the weighted sum by (keys + 64) 2^-24."""
    from gibbs_b200.ops import hybrid, library
    torch.manual_seed(r + window)
    Dk, ps, R = r + dr, 16, 3
    n_pages = 64
    pages = torch.randn(n_pages, ps, Dk).to(torch.bfloat16)
    perm = torch.randperm(n_pages)[:60].reshape(3, 20)
    scale, sink = 0.7 * Dk ** -0.5, torch.randn(H)
    lens_of = {"portions": [(0, 70), (30, 33), (250, 1)], "single": [(299, 1), (31, 1), (0, 1)], "mixed": [(100, 1), (0, 40), (200, 17)]}
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    rows = library("hybrid").gb_latent_attention_workspace_rows()
    ws = torch.full((rows, r + 2), float("nan"), device=DEV)
    for what, spans in lens_of.items():
        tok_req = [i for i, (p, k) in enumerate(spans) for _ in range(k)]
        tok_pos = [p + j for p, k in spans for j in range(k)]
        n = len(tok_req)
        if window == 0 and n >= 8 * R and n * H >= 256:
            continue                                        # (such steps run on the kernel without windows)
        starts = [sum(k for _, k in spans[:i]) for i in range(R)]
        q, gate = torch.randn(n, H, Dk), torch.randn(n, H)
        dev = {k: v.to(DEV).contiguous() for k, v in dict(q=q, pages=pages, gate=gate, sink=sink).items()}
        table, tr, tp, qs = i32(perm.tolist()), i32(tok_req), i32(tok_pos), i32(starts)
        got = {}
        for tc in (True, False):
            out = torch.full((n, H * r), float("nan"), device=DEV)
            hybrid.call("latent_attention", [dev["q"].data_ptr(), dev["pages"].data_ptr(), 1, table.data_ptr(), 20, ps, n_pages,
                                             tr.data_ptr(), tp.data_ptr(), dev["gate"].data_ptr(), H, out.data_ptr(), H * r, n, H,
                                             r, dr, window, 320, ws.data_ptr(), dev["sink"].data_ptr(), R if tc else 0,
                                             qs.data_ptr() if tc else 0], [scale])
            got[tc] = out.double().cpu().reshape(n, H, r)
        off = {True: 0.0, False: 0.0}
        for t in range(n):
            lo = max(0, tok_pos[t] - window + 1) if window else 0
            j = torch.arange(lo, tok_pos[t] + 1)
            c = pages[perm[tok_req[t]][j // ps], j % ps].double()
            sc = q[t].double() @ c.T * scale
            w = torch.softmax(torch.cat([sc, sink.double()[:, None]], 1), 1)[:, :-1]
            f = torch.sigmoid(gate[t].double())[:, None]
            want, size = (w @ c[:, :r]) * f, (w @ c[:, :r].abs()) * f
            d = (Dk + 16) * 2.0 ** -24 * scale * (q[t].double().abs() @ c.T.abs()).amax(1)
            tol = (2 * d[:, None] + 2.0 ** -20 + (len(j) + 64) * 2.0 ** -24) * size + 2.0 ** -22 * want.abs()
            assert ((got[True][t] - want).abs() <= tol).all(), (what, t)
            for tc in off:
                off[tc] += float((got[tc][t] - want).pow(2).sum())
        # (two kernels did run; a window of one key runs on the generic kernel)
        assert window == 1 or not torch.equal(got[True], got[False])
        if what != "single":                                # (rows enough for the two errors to be compared: measured 0.55 to 1)
            assert off[True] <= off[False], (off[True] / off[False]) ** 0.5


@pytest.mark.parametrize("H,r,dr", [(1, 32, 0), (2, 64, 0), (4, 64, 16), (16, 128, 0), (16, 128, 32), (8, 256, 32), (16, 512, 0), (16, 512, 64)])
def test_latent_attention_with_whole_weights_is_no_further_off_than_the_generic_kernel(H, r, dr):
    """Single tokens at short and long contexts and a short portion, with and without a window, on both kernels against
    64 bits: the root of the summed squares of all errors."""
    from gibbs_b200.ops import hybrid, library
    torch.manual_seed(r + dr)
    Dk, ps, blocks = r + dr, 16, 128
    pages = torch.randn(3 * blocks, ps, Dk, device=DEV).to(torch.bfloat16)
    table = torch.randperm(3 * blocks, device=DEV).reshape(3, blocks)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    ws = torch.empty(library("hybrid").gb_latent_attention_workspace_rows(), r + 2, device=DEV)
    scale, bt, off = 0.7 * Dk ** -0.5, table.to(torch.int32), {True: 0.0, False: 0.0}
    for spans in ([(2000, 1), (900, 1), (299, 1)], [(0, 7), (300, 9), (1500, 5)]):
        tok_req = [i for i, (p, k) in enumerate(spans) for _ in range(k)]
        tok_pos = [p + j for p, k in spans for j in range(k)]
        n = len(tok_req)
        starts = i32([sum(k for _, k in spans[:i]) for i in range(3)])
        tr, tp = i32(tok_req), i32(tok_pos)
        for window in (0, 128, 1024):
            for _ in range(4 if H < 8 else 1):
                q, gate, sink = (torch.randn(*s, device=DEV) for s in ((n, H, Dk), (n, H), (H,)))
                got = {}
                for tc in (True, False):
                    got[tc] = torch.empty(n, H * r, device=DEV)
                    hybrid.call("latent_attention", [q.data_ptr(), pages.data_ptr(), 1, bt.data_ptr(), blocks, ps, 3 * blocks,
                                                     tr.data_ptr(), tp.data_ptr(), gate.data_ptr(), H, got[tc].data_ptr(), H * r, n,
                                                     H, r, dr, window, 2001, ws.data_ptr(), sink.data_ptr(), 3 if tc else 0,
                                                     starts.data_ptr() if tc else 0], [scale])
                assert not torch.equal(got[True], got[False])                # (two kernels did run)
                for t in range(n):
                    j = torch.arange(max(0, tok_pos[t] - window + 1) if window else 0, tok_pos[t] + 1, device=DEV)
                    c = pages[table[tok_req[t]][j // ps], j % ps].double()
                    sc = torch.cat([q[t].double() @ c.T * scale, sink.double()[:, None]], 1)
                    want = (torch.softmax(sc, 1)[:, :-1] @ c[:, :r]) * torch.sigmoid(gate[t].double())[:, None]
                    for tc in off:
                        off[tc] += float((got[tc][t].double().view(H, r) - want).pow(2).sum() / want.pow(2).sum())
    assert off[True] <= off[False], (off[True] / off[False]) ** 0.5


class LatentCalls:
    """Single calls of the latent attention on bfloat16 pages of random rows."""
    def __init__(self, H, r, dr, blocks=64, ps=16, seed=0):
        from gibbs_b200.ops import library
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.H, self.r, self.dr, self.blocks, self.ps = H, r, dr, blocks, ps
        self.pages = torch.randn(blocks, ps, r + dr, generator=g, device=DEV).to(torch.bfloat16)
        self.table = torch.randperm(blocks, generator=g, device=DEV).to(torch.int32)
        self.rows = library("hybrid").gb_latent_attention_workspace_rows()
        self.ws = torch.full((self.rows, r + 2), float("nan"), device=DEV)

    def __call__(self, q, gate, sink, spans, window, longest, chunks=True):
        """q [tokens, H, r + dr], gate [tokens, H]; spans: (first position, tokens) of each request (all read the same
        pages); `chunks` False: no workspace, one chunk."""
        from gibbs_b200.ops import hybrid
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        R, n = len(spans), sum(k for _, k in spans)
        req, pos = i32([i for i, (p, k) in enumerate(spans) for _ in range(k)]), i32([p + j for p, k in spans for j in range(k)])
        start, bt = i32([sum(k for _, k in spans[:i]) for i in range(R)]), self.table.expand(R, -1).contiguous()
        out = torch.full((n, self.H * self.r), float("nan"), device=DEV)
        q, gate = q.contiguous(), gate.contiguous()
        hybrid.call("latent_attention", [q.data_ptr(), self.pages.data_ptr(), 1, bt.data_ptr(), self.blocks, self.ps, self.blocks,
                                         req.data_ptr(), pos.data_ptr(), gate.data_ptr(), self.H, out.data_ptr(), self.H * self.r, n,
                                         self.H, self.r, self.dr, window, longest, self.ws.data_ptr() if chunks else 0,
                                         0 if sink is None else sink.data_ptr(), R, start.data_ptr()], [(self.r + self.dr) ** -0.5])
        return out


@pytest.mark.parametrize("H,r,dr", [(3, 40, 8), (5, 128, 0), (16, 256, 32)])
@pytest.mark.parametrize("window", [32, 33, 200])
def test_latent_attention_with_whole_weights_does_not_depend_on_the_rows_beside_a_token(H, r, dr, window):
    """A token's bits are the same however the portion is cut, alone and beside another request, with one chunk and with
    chunks of the same length (as many tokens in the step), and where a request brings no token."""
    call = LatentCalls(H, r, dr)
    torch.manual_seed(window)
    n, first = 37, 250
    q, gate, sink = (torch.randn(*s, device=DEV) for s in ((n, H, r + dr), (n, H), (H,)))
    whole = call(q, gate, sink, [(first, n)], window, 300, chunks=False)
    for cuts in ([0, 1, n], [0, 16, 18, n], [0, 5, 7, 30, n]):
        for a, b in zip(cuts, cuts[1:]):
            assert torch.equal(call(q[a:b], gate[a:b], sink, [(first + a, b - a)], window, 300, chunks=False), whole[a:b]), (a, b)
    some = call(q[:6], gate[:6], sink, [(first, 6)], window, 300)
    for spans in ([(first, 1), (first + 1, 5)], [(first, 3), (first + 3, 0), (first + 3, 3)], [(first, 6)] + [(0, 0)] * 5,
                  [(first + i, 1) for i in range(6)]):
        assert torch.equal(call(q[:6], gate[:6], sink, spans, window, 300), some), spans
    sc = torch.einsum("nhd,ld->nhl", q[:6].double(), call.pages[call.table.long()].reshape(-1, r + dr).double()) * (r + dr) ** -0.5
    i, j = torch.arange(first, first + 6, device=DEV)[:, None], torch.arange(sc.shape[2], device=DEV)
    sc.masked_fill_(~((j <= i) & (j > i - window))[:, None], -math.inf)
    w = torch.softmax(torch.cat([sc, sink.double()[None, :, None].expand(6, H, 1)], 2), 2)[:, :, :-1]
    want = (w @ call.pages[call.table.long()].reshape(-1, r + dr)[:, :r].double()) * torch.sigmoid(gate[:6].double())[..., None]
    assert rel_rows(some.cpu(), want.reshape(6, -1).cpu()).max() < 2e-6


@pytest.mark.parametrize("H,r,dr,window", [(3, 40, 8, 0), (16, 256, 32, 0), (16, 512, 64, 0), (16, 512, 64, 40), (5, 128, 0, 512)])
@pytest.mark.parametrize("with_sink", [False, True])
def test_latent_attention_with_whole_weights_has_the_same_bits_in_one_chunk_and_in_several(H, r, dr, window, with_sink):
    """Contexts that fit one chunk: without a workspace, with an upper bound that gives one chunk, and with one that gives
    many, all others empty."""
    call = LatentCalls(H, r, dr)
    torch.manual_seed(r + window)
    spans = [(20, 1), (5, 1), (31, 1)]
    q, gate = torch.randn(3, H, r + dr, device=DEV), torch.randn(3, H, device=DEV)
    sink = torch.randn(H, device=DEV) if with_sink else None
    one = call(q, gate, sink, spans, window, 64, chunks=False)
    assert not one.isnan().any()
    for longest in (33, 64, 300, 1000):
        assert torch.equal(call(q, gate, sink, spans, window, longest), one), longest


@pytest.mark.parametrize("H,r,dr", [(3, 40, 8), (16, 320, 0), (16, 512, 64)])
@pytest.mark.parametrize("window", [0, 40])
def test_latent_attention_with_whole_weights_keeps_what_is_not_finite_to_the_rows_that_see_it(H, r, dr, window):
    """Cached rows that hold no numbers or infinite ones (one behind some tokens, one in front of some windows), a query
    that does: what is no number is what is none in 64 bits, all else as there, and rows that do not see it as without it."""
    call = LatentCalls(H, r, dr)
    torch.manual_seed(r)
    spans, n = [(98, 7), (50, 1), (70, 1)], 9
    q, gate, sink = (torch.randn(*s, device=DEV) for s in ((n, H, r + dr), (n, H), (H,)))
    clean, pos, tok = call(q, gate, sink, spans, window, 128), [98 + i for i in range(7)] + [50, 70], torch.arange(n)

    def exact(q):
        out = []
        for t in range(n):
            c = call.pages[call.table.long()].reshape(-1, r + dr)[max(0, pos[t] - window + 1) if window else 0:pos[t] + 1].double()
            sc = torch.cat([q[t].double() @ c.T * (r + dr) ** -0.5, sink.double()[:, None]], 1)
            w = torch.softmax(sc, 1)[:, :-1]
            out.append(((w[:, :, None] * c[None, :, :r]).sum(1) * torch.sigmoid(gate[t].double())[:, None]).reshape(-1))
        return torch.stack(out).cpu()

    def same(got, want, what):
        assert torch.equal(got.isnan().cpu(), want.isnan()), what
        assert rel_rows(got.nan_to_num(0.0).cpu() + 1e-30, want.nan_to_num(0.0) + 1e-30).max() < 1e-5, what

    sound = call.pages.clone()
    for value in (float("nan"), float("inf"), -float("inf")):
        for at, entry in ((102, 3), (61, r - 1), (61, 0)):
            call.pages.copy_(sound)
            call.pages[call.table[at // 16].long(), at % 16, entry] = value
            got = call(q, gate, sink, spans, window, 128)
            same(got, exact(q), (value, at, entry))
            blind = [t for t in tok.tolist() if at > pos[t] or (window and at <= pos[t] - window)]
            assert blind and len(blind) < n
            assert rel_rows(got[blind].cpu(), clean[blind].cpu()).max() < 1e-5
            assert got[[t for t in range(n) if t not in blind]].isnan().any()
        call.pages.copy_(sound)
        bad = q.clone()
        bad[2, H - 1, 5] = value
        got = call(bad, gate, sink, spans, window, 128)
        same(got, exact(bad), value)
        assert torch.equal(got.isnan().any(1).cpu(), tok == 2)


@pytest.mark.parametrize("splits,r", [(2, 8), (2, 512), (3, 264), (5, 40), (8, 512)])
def test_latent_merge_has_the_same_bits_by_a_block_and_by_a_warp_a_row(splits, r):
    """Steps of single tokens on both sides of the number of rows (128 a chunk) from which a warp takes a row: the first
    tokens are the same, and so are their bits."""
    H, n = 16, 8 * splits                                    # (n * H = 128 * splits is the first launch by warps)
    call = LatentCalls(H, r, 0)
    torch.manual_seed(r)
    gate, sink = torch.randn(n, H, device=DEV), torch.randn(H, device=DEV)
    by_blocks, by_warps = (_merge_alone(call, k, H, r, splits, sink, gate) for k in (n - 1, n))
    assert torch.equal(by_blocks, by_warps[:n - 1])


def _merge_alone(call, n, H, r, splits, sink, gate):
    """The generic kernel on 32-bit pages of one chunk of 64 keys after the other: `splits` of them by the context."""
    from gibbs_b200.ops import hybrid
    g = torch.Generator(device=DEV).manual_seed(7)
    blocks, ps, longest = 4 * splits, 16, 64 * splits
    pages = torch.randn(blocks, ps, r, generator=g, device=DEV)
    q = torch.randn(n, H, r, generator=g, device=DEV)
    bt = torch.arange(blocks, dtype=torch.int32, device=DEV)[None].expand(n, -1).contiguous()
    req = torch.arange(n, dtype=torch.int32, device=DEV)
    pos = (torch.arange(n, device=DEV) * 37 % longest).to(torch.int32)
    out = torch.full((n, H * r), float("nan"), device=DEV)
    launched = hybrid.call("latent_attention", [q.data_ptr(), pages.data_ptr(), 0, bt.data_ptr(), blocks, ps, blocks, req.data_ptr(),
                                                pos.data_ptr(), gate.data_ptr(), H, out.data_ptr(), H * r, n, H, r, 0, 0, longest,
                                                call.ws.data_ptr(), sink.data_ptr(), 0, 0], [r ** -0.5])
    assert launched == 2 and not out.isnan().any()
    return out


@pytest.mark.parametrize("d", [40, 64, 300, 2048, 2049, 4096])
@pytest.mark.parametrize("kind", [0, 1])
def test_norm_behind_a_sublayer_in_steps_of_few_rows_and_of_many(d, kind):
    """296 rows (the last step whose gains are read ahead) and 297, with the next sublayer's norm and without: against 64
    bits, and the rows they share have the same bits."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(d)
    x0, y, gain, then = torch.randn(297, d), torch.randn(297, d), torch.randn(d), torch.randn(d)
    dev = [t.to(DEV) for t in (y, gain, then)]
    def norm(v, g):
        v = v.double() - (v.double().mean(1, keepdim=True) if kind == 0 else 0.0)
        return v / (v.pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * g.double()
    new = x0.double() + norm(y, gain)
    for second in (False, True):
        got = {}
        for n in (297, 296):
            x, h = x0[:n].to(DEV), torch.zeros(n, d, device=DEV)
            hybrid.call("norm_add", [x.data_ptr(), d, dev[0].data_ptr(), d, dev[1].data_ptr(), n, d, kind, 0, dev[2].data_ptr() if second else 0,
                                     h.data_ptr() if second else 0, 0, kind], [1e-5, 1e-5])
            got[n] = torch.cat([x, h], 1)
        assert torch.equal(got[296], got[297][:296])
        assert rel_rows(got[297][:, :d].cpu(), new).max() < 1e-6
        if second:
            assert rel_rows(got[297][:, d:].cpu(), norm(new, then)).max() < 2e-6


@pytest.mark.parametrize("H,P,N,G", [(2, 4, 4, 1), (3, 32, 32, 3), (4, 68, 36, 2), (2, 64, 64, 2), (64, 64, 128, 8), (5, 36, 124, 1)])
def test_state_space_scan_at_the_edges_of_its_groups_of_tokens(H, P, N, G):
    """Lengths around the groups of 2 to 8 tokens and the chunks of 16, widths that fill a block's columns and lanes or
    do not, against the recurrence in 64 bits.  The state is a sum of decayed products whose errors decay with it: each
    token adds 4 roundings to what is kept and exp and softplus a few units in the last place; the read-out adds N
    terms.  With decays of at most exp(-0.5) per token the kept errors add up to less than 2.6 tokens' worth."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(N)
    for lens in ([1, 2, 7], [8, 9, 15], [16, 17, 33, 1, 130]):
        R, n = len(lens), sum(lens)
        ld = H * P + 2 * G * N
        xbc, dt = torch.randn(n, ld), torch.rand(n, H)
        bias, alog, D = torch.rand(H), torch.rand(H), torch.randn(H)
        slot, S0 = H * P * N, torch.randn(R + 2, H, N, P)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        ids, starts = list(range(R, 0, -1)), [sum(lens[:i]) for i in range(R)]
        dev = [t.to(DEV) for t in (xbc, dt, bias, alog, D)]
        state, y = S0.clone().to(DEV), torch.full((n, H * P), float("nan"), device=DEV)
        i = [i32(ids), i32(starts), i32(lens)]
        p = [t.data_ptr() for t in dev]
        hybrid.call("ssm_scan", [p[0], ld, p[1], H, p[2], p[3], p[4], state.data_ptr(), slot, i[0].data_ptr(), i[1].data_ptr(),
                                 i[2].data_ptr(), y.data_ptr(), H * P, R, H, P, N, G])
        step = torch.nn.functional.softplus(dt.double() + bias.double())
        decay = torch.exp(-torch.exp(alog.double()) * step)
        assert decay.max() <= math.exp(-0.5)
        x, B, C = xbc[:, :H * P].double().reshape(n, H, P), xbc[:, H * P:H * P + G * N].double(), xbc[:, H * P + G * N:].double()
        B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        for r in range(R):
            S, size = S0[ids[r]].double(), S0[ids[r]].double().abs()
            for t in range(starts[r], starts[r] + lens[r]):
                add = B[t][:, :, None] * (step[t][:, None] * x[t])[:, None]
                S, size = decay[t][:, None, None] * S + add, decay[t][:, None, None] * size + add.abs()
                want = (S * C[t][:, :, None]).sum(1) + D.double()[:, None] * x[t]
                bound = (size * C[t].abs()[:, :, None]).sum(1) + (D.double()[:, None] * x[t]).abs()
                err = (y[t].double().cpu().reshape(H, P) - want).abs()
                assert (err <= (N / 4 + 40) * 2.0 ** -24 * bound).all(), (lens, r, t - starts[r])
            assert ((state[ids[r]].double().cpu() - S).abs() <= 40 * 2.0 ** -24 * size).all()
        assert torch.equal(state[0].cpu(), S0[0]) and torch.equal(state[R + 1].cpu(), S0[R + 1])


@pytest.mark.parametrize("H,P,N,R", [(3, 36, 32, 2), (3, 36, 36, 2), (2, 64, 64, 2), (16, 64, 128, 2), (64, 64, 128, 6), (8, 16, 128, 3)])
def test_state_space_scan_has_the_same_bits_however_states_lie_and_portions_are_cut(H, P, N, R):
    """States on 4-byte boundaries beside 8-byte ones; portions whole, cut in two and token by token, alone and together (few
    blocks and many: the two forms of the kernel for 128 values)."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(N)
    G, n = 1, 19
    ld = H * P + 2 * G * N
    xbc, dt = torch.randn(R * n, ld, device=DEV), torch.rand(R * n, H, device=DEV)
    bias, alog, D, S0 = torch.rand(H, device=DEV), torch.rand(H, device=DEV), torch.randn(H, device=DEV), torch.randn(R, H * N * P, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def run(cuts, together, pad):
        store = torch.zeros(R * (H * N * P + pad) + pad, device=DEV)
        state = store[pad:].as_strided((R, H * N * P), (H * N * P + pad, 1))
        state.copy_(S0)
        y = torch.full((R * n, H * P), float("nan"), device=DEV)
        for a, b in zip(cuts, cuts[1:]):
            for who in ([list(range(R))] if together else [[r] for r in range(R)]):
                ids, at, ln = i32(who), i32([r * n + a for r in who]), i32([b - a] * len(who))
                hybrid.call("ssm_scan", [xbc.data_ptr(), ld, dt.data_ptr(), H, bias.data_ptr(), alog.data_ptr(), D.data_ptr(), state.data_ptr(),
                                         H * N * P + pad, ids.data_ptr(), at.data_ptr(), ln.data_ptr(), y.data_ptr(), H * P, len(who), H, P, N, G])
        return torch.cat([y.flatten(), state.flatten()])

    want = run([0, n], True, 0)
    assert not want.isnan().any()
    for cuts, together, pad in (([0, n], True, 1), ([0, n], False, 0), ([0, 7, n], True, 3), (list(range(n + 1)), True, 0), (list(range(n + 1)), False, 1)):
        assert torch.equal(run(cuts, together, pad), want), (cuts, together, pad)


@pytest.mark.parametrize("H,r,dr,spans,window,longest,generic", [
    (16, 128, 32, [(0, 7)], 0, 8, True), (16, 128, 32, [(0, 7)], 0, 16, True), (16, 128, 32, [(0, 7)], 0, 17, False),
    (16, 512, 64, [(0, 7)], 0, 8, True), (16, 512, 64, [(0, 7)], 0, 9, False), (16, 512, 0, [(300, 2)] * 2, 16, 320, False),
    (16, 256, 32, [(300, 2)] * 2, 16, 320, True), (16, 256, 32, [(300, 2)] * 2, 17, 320, False),
    (8, 128, 32, [(300, 1)] * 16, 0, 1024, True), (8, 128, 32, [(300, 1)] * 16, 0, 1023, False), (8, 128, 32, [(300, 1)] * 15, 0, 1024, False),
    (9, 128, 32, [(300, 1)] * 16, 0, 1024, False), (8, 136, 32, [(300, 1)] * 16, 0, 1024, False), (8, 136, 32, [(300, 1)] * 64, 256, 1024, True),
    (8, 136, 32, [(300, 1)] * 64, 264, 1024, False), (16, 128, 32, [(300, 1)] * 64, 128, 1024, True), (16, 128, 32, [(300, 1)] * 63, 128, 1024, False),
    (16, 128, 32, [(300, 1)] * 64, 129, 1024, False), (2, 64, 0, [(300, 1)] * 15 + [(300, 2)], 0, 1024, False)])
def test_latent_attention_takes_the_kernel_that_pays(H, r, dr, spans, window, longest, generic):
    """Both sides of every line of the rule: the generic kernel's bits or not, and 64 bits either way."""
    call = LatentCalls(H, r, dr)
    torch.manual_seed(longest)
    n = sum(k for _, k in spans)
    q, gate, sink = (torch.randn(*s, device=DEV) for s in ((n, H, r + dr), (n, H), (H,)))
    got, pos = call(q, gate, sink, spans, window, longest), [p + j for p, k in spans for j in range(k)]
    assert torch.equal(got, _generic_latent(call, q, gate, sink, spans, window, longest)) == generic
    rows = call.pages[call.table.long()].reshape(-1, r + dr).double()
    for t in (0, n - 1):
        c = rows[max(0, pos[t] - window + 1) if window else 0:pos[t] + 1]
        sc = torch.cat([q[t].double() @ c.T * (r + dr) ** -0.5, sink.double()[:, None]], 1)
        want = (torch.softmax(sc, 1)[:, :-1] @ c[:, :r]) * torch.sigmoid(gate[t].double())[:, None]
        assert rel_rows(got[t].view(H, r).cpu(), want.cpu()).max() < 2e-6


def _generic_latent(call, q, gate, sink, spans, window, longest):
    """The same call on the generic kernel (no row starts per request)."""
    from gibbs_b200.ops import hybrid
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    R, n = len(spans), sum(k for _, k in spans)
    req, pos = i32([i for i, (p, k) in enumerate(spans) for _ in range(k)]), i32([p + j for p, k in spans for j in range(k)])
    out, bt = torch.full((n, call.H * call.r), float("nan"), device=DEV), call.table.expand(R, -1).contiguous()
    hybrid.call("latent_attention", [q.data_ptr(), call.pages.data_ptr(), 1, bt.data_ptr(), call.blocks, call.ps, call.blocks,
                                     req.data_ptr(), pos.data_ptr(), gate.data_ptr(), call.H, out.data_ptr(), call.H * call.r, n,
                                     call.H, call.r, call.dr, window, longest, call.ws.data_ptr(), sink.data_ptr(), 0, 0],
                [(call.r + call.dr) ** -0.5])
    return out


@pytest.mark.parametrize("weights,result", [("float32", "float32"), ("bfloat16", "float32"), ("bfloat16", "bfloat16")])
@pytest.mark.parametrize("H,O,I", [(1, 1, 8), (3, 5, 24), (16, 128, 512), (2, 17, 1024), (2, 18, 1032), (4, 512, 128), (2, 9, 20)])
def test_head_products_of_a_few_rows(H, O, I, weights, result):
    """Rows 1 to 17 (the few-rows kernel ends at 16), outputs that do not fill a warp's four, inputs at and beyond what
    its registers hold and no whole pieces (the other kernels): a lane adds I / 32 + 8 products, then five levels.
    From 64 rows on bfloat16 weights round their inputs; these stay below."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(I)
    W = torch.randn(H, O, I).to(DTYPES[weights])
    Wd = W.to(DEV)
    for n in (1, 2, 3, 16, 17):
        x, gate = torch.randn(n, H * I + 4), torch.randn(n, H * O)
        xd, gd = x.to(DEV), gate.to(DEV)
        for gated in (False, True):
            out = torch.full((n, H * O), float("nan"), dtype=DTYPES[result], device=DEV)
            hybrid.call("head_linear", [xd.data_ptr(), H * I + 4, I, Wd.data_ptr(), 1 if weights == "bfloat16" else 0, out.data_ptr(),
                                        1 if result == "bfloat16" else 0, H * O, O, n, H, O, I] +
                        ([gd.data_ptr(), H * O] if gated else []))
            xs = x[:, :H * I].double().reshape(n, H, I)
            f = torch.sigmoid(gate.double()).reshape(n, H, O) if gated else torch.ones(n, H, O, dtype=torch.float64)
            want = torch.einsum("nhi,hoi->nho", xs, W.double()) * f
            size = torch.einsum("nhi,hoi->nho", xs.abs(), W.double().abs()) * f
            tol = (I / 8 + 24) * 2.0 ** -24 * size + (2.0 ** -8 * want.abs() if result == "bfloat16" else 0)
            assert ((out.double().cpu().reshape(n, H, O) - want).abs() <= tol).all(), (n, gated)


@pytest.mark.parametrize("weights", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,O,I", [(16, 16, 32), (16, 64, 64), (16, 128, 128), (16, 64, 256), (4, 64, 512), (2, 64, 1024)])
def test_head_products_of_a_few_rows_are_no_further_off_than_the_other_kernel(H, O, I, weights):
    """Rows from 1 to 16 on both kernels (inputs that are not 16-byte aligned run on the other) against 64 bits, the bits
    of a row whatever the rows beside it."""
    from gibbs_b200.ops import hybrid
    torch.manual_seed(I)
    W = torch.randn(H, O, I, device=DEV).to(DTYPES[weights])
    if weights == "float32" and I > 512:
        pytest.skip("more pieces than a lane keeps: the other kernel in both cases")
    store, off, first = torch.randn(16 * H * I + 1, device=DEV), {0: 0.0, 1: 0.0}, None
    for shift in (0, 1):
        x = store[shift:shift + 16 * H * I].view(16, H * I)
        want = torch.einsum("nhi,hoi->nho", x.double().view(16, H, I), W.double())
        whole = None
        for n in (16, 9, 8, 5, 4, 3, 2, 1):
            out = torch.empty(n, H * O, device=DEV)
            hybrid.call("head_linear", [x.data_ptr(), H * I, I, W.data_ptr(), 1 if weights == "bfloat16" else 0, out.data_ptr(), 0, H * O, O,
                                        n, H, O, I])
            whole = out if whole is None else whole
            assert shift or torch.equal(out, whole[:n]), n
            off[shift] += float((out.double().view(n, H, O) - want[:n]).pow(2).sum())
    assert off[0] <= 1.05 ** 2 * off[1], (off[0] / off[1]) ** 0.5        # (other inputs: the two sums are each within 2%)


def _pointed_attention(window, T, hot_key, query, d=64, seed=7):
    """Weights and inputs for which the query position's score against ``hot_key`` stands far
    above all others (when that key is visible), and whose values tell keys apart.  The latent is
    the input's first entries, the unrotated key of head 0 is the latent's first entries, the
    query is the input scaled: q . k_j = gamma * h_q . rmsnorm(h_j)."""
    H, dn, dr, dv, r = 2, 16, 4, 8, 24
    m = {"heads": H, "dim": dn, "rot_dim": dr, "vdim": dv, "kv_rank": r, "scale": 1.0, "rot": {"base": 100.0, "dims": dr}}
    if window:
        m["mask"] = {"size": window}
    g = gen(seed)
    W = {"q": torch.zeros(H * (dn + dr), d), "dkv": torch.zeros(r + dr, d), "dkv.norm": torch.ones(r),
         "uk": torch.zeros(H * dn, r), "uv": bf(torch.randn(H * dv, r, generator=g)), "g": torch.zeros(H, d),
         "o": bf(torch.randn(d, H * dv, generator=g) / 4)}
    for i in range(r):
        W["dkv"][i, i] = 1.0
    for hh in range(H):
        for i in range(dn):
            W["uk"][hh * dn + i, i] = 1.0
            W["q"][hh * (dn + dr) + i, i] = 1.0
    h = bf(torch.randn(T, d, generator=g))
    h[:, r:] = 0
    key = h[hot_key, :dn] / h[hot_key, :r].pow(2).mean().sqrt()
    h[query] = 0
    h[query, :dn] = bf(6.0 * key / key.norm())               # score against the hot key: about 6 |k|, others a few units
    h[query, dn:r] = 30.0                                     # (a long latent: the query's own key scores low)
    return m, W, h


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("decoded", [False, True])
@pytest.mark.parametrize("window,T,hot,query", [
    (40, 120, 60, 99),        # the oldest key the window keeps (99 - 60 = 39)
    (40, 120, 59, 99),        # the first one it has dropped
    (40, 120, 0, 39),         # the first token of the sequence, just inside
    (40, 120, 0, 40),         # ... and just outside
    (16, 120, 80, 95),        # a window of one page: its edge is a page's edge
    (16, 120, 79, 95),
    (None, 400, 3, 399),      # no window: a key hundreds of positions back
    (None, 400, 16, 399),     # ... at a page's first row
    (300, 400, 100, 399),     # a long window: far but inside
    (300, 400, 99, 399),      # ... and outside
])
def test_latent_attention_finds_the_one_key_that_matters(window, T, hot, query, decoded, dtype):
    m, W, h = _pointed_attention(window, T, hot, query)
    part = make_part("mixer", "latent_attention", _attention_params(m, h.shape[1]), W, DTYPES[dtype])
    want = plain.latent_attention(h.double(), m, {k: v.double() for k, v in W.items()}, 1e-5)
    visible = window is None or query - hot < window
    hz = PartHarness(part, n_pages=32, page_size=16)
    got = hz.run_cut("r", h, [query - 10, 1] if decoded else [T])
    e = rel_rows(got, want)
    assert e[query] <= TOL[dtype], f"query row differs by {e[query]:.3g}"
    assert e.max() <= TOL[dtype]
    # the hot key's value dominates the output exactly when it is visible
    c_hot = plain.rms_norm(h[hot, :m["kv_rank"]].double(), None, 1e-5)
    v_hot = (W["uv"].double() @ c_hot) * 0.5                   # gate logits are zero: sigmoid = 1/2
    out_hot = W["o"].double() @ v_hot
    close = float((got[query].double() - out_hot).norm() / out_hot.norm())
    assert (close < 0.2) == visible, f"hot key visible={visible}, distance to its value {close:.3g}"


def _ssm_params(m, d):
    return {"hidden": d, "heads": m["heads"], "vdim": m["vdim"], "state": m["state"], "groups": m["groups"],
            "conv": m["conv"], "norm_groups": m.get("norm_groups", 1), "eps": 1e-5}


def _ssm_cfg(state, vdim, heads=2, groups=1, conv=3):
    return {"vocab": 16, "width": 48, "norm": {"eps": 1e-5}, "layers": [
        {"type": "mamba2", "mixer": {"heads": heads, "vdim": vdim, "state": state, "groups": groups, "conv": conv,
                                     "norm_groups": 1}, "mlp": None}]}


# states of 20, 64 and 128 values run with the state in registers (one, two and four lanes a column); 70 (no multiple
# of four) and 160 (more than 128) with the lanes over the state dimension; 128 x 72: more columns than a block takes
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg,layer", [(CFG_A, 1), (CFG_B, 0), (_ssm_cfg(64, 8), 0), (_ssm_cfg(128, 72, heads=4, groups=2), 0),
                                       (_ssm_cfg(160, 8), 0)])
def test_state_space_mixer_alone_whole_cut_and_decoded(cfg, layer, dtype):
    m, d = cfg["layers"][layer]["mixer"], cfg["width"]
    W = _mixer_weights(cfg, layer, 8)
    part = make_part("mixer", "state_space", _ssm_params(m, d), W, DTYPES[dtype])
    T = 90
    h = bf(torch.randn(T, d, generator=gen(9)))
    want = plain.mamba2(h.double(), m, {k: v.double() for k, v in W.items()}, 1e-5)
    hz = PartHarness(part, n_slots=2)
    for rid, cuts in (("whole", [T]), ("cut", [2, 1, 3, 17, 2, 31, 1, 1, 5]), ("decoded", [T - 40, 1])):
        got = hz.run_cut(rid, h, cuts)
        check_rows(got, want, dtype, what=f"state-space mixer, {rid}")
        hz.close(rid)                                           # the slot goes back and is taken again, zeroed


def test_state_space_state_is_carried_far_and_a_reused_slot_starts_at_zero():
    """Decay close to one and a strong first token: position 0 still shows 300 tokens later, however
    the sequence is cut; and the next request in the same slot does not see it."""
    cfg = {"heads": 2, "vdim": 8, "state": 16, "groups": 1, "conv": 3, "norm_groups": 1}
    d = 32
    W = _mixer_weights({**CFG_A, "width": d, "layers": [{"type": "mamba2", "mixer": cfg, "mlp": None}],
                        "token_side": None}, 0, 10)
    W["A_log"] = torch.full((2,), math.log(0.02))             # exp(-0.02 dt): almost no forgetting
    part = make_part("mixer", "state_space", _ssm_params(cfg, d), W, torch.float32)
    T = 300
    h = bf(torch.randn(T, d, generator=gen(11)) * 0.3)
    h2 = h.clone()
    h2[0] = bf(h[0] * 8 + 1)
    Wd = {k: v.double() for k, v in W.items()}
    want, want2 = plain.mamba2(h.double(), cfg, Wd, 1e-5), plain.mamba2(h2.double(), cfg, Wd, 1e-5)
    assert np.median(rel_rows(want[-20:], want2[-20:])) > 1e-3  # the first token matters at the end
    hz = PartHarness(part, n_slots=1)
    got2 = hz.run_cut("first", h2, [7, 2, 64, 1, 1, 100, 3])
    assert rel_rows(got2, want2).max() <= TOL["float32"]
    hz.close("first")
    got = hz.run_cut("second", h, [150, 1])                    # same slot
    assert rel_rows(got, want).max() <= TOL["float32"]


def _routed_params(f, d):
    sh = f.get("shared")
    return {"hidden": d, "experts": f["router"]["experts"], "top": f["router"]["top"], "expert_inner": f["expert"]["ff"],
            "expert_limit": f["expert"]["limit"], "shared_inner": sh["ff"] if sh else 0,
            "shared_limit": sh["limit"] if sh else 0.0}


# experts whose width is a multiple of 64: in bfloat16 their products run on the tensor cores (tiles of 64 rows
# for the batch, of 16 for single tokens), in float32 on the 32-bit tiles with the same weight layout
CFG_WIDE_EXPERTS = {"vocab": 16, "width": 64, "norm": {"eps": 1e-5}, "layers": [
    {"type": "mamba2", "mixer": {"heads": 1, "vdim": 8, "state": 8, "groups": 1, "conv": 2, "norm_groups": 1},
     "mlp": {"kind": "moe", "router": {"experts": 4, "top": 2}, "expert": {"ff": 128, "limit": 1.5}}}]}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg,layer", [(CFG_A, 0), (CFG_A, 3), (CFG_B, 0), (CFG_WIDE_EXPERTS, 0)])
def test_routed_experts_alone(cfg, layer, dtype):
    f, d = cfg["layers"][layer]["mlp"], cfg["width"]
    W = plain.sub(make_weights(cfg, 13), f"l{layer}.mlp.")
    # router rows far apart, so that no choice hangs on the rounding of the input
    E = f["router"]["experts"]
    W["router"] = bf(torch.randn(E, d, generator=gen(14)) * 0.9)
    part = make_part("feed_forward", "routed_glu", _routed_params(f, d), W, DTYPES[dtype])
    T = 140                                                    # more than one tile of rows for some expert
    h = bf(torch.randn(T, d, generator=gen(15)))
    z = h.double() @ W["router"].double().T
    top = f["router"]["top"]
    srt = torch.sort(z, dim=1, descending=True).values
    keep = (srt[:, top - 1] - srt[:, top]) > 0.15 if top < E else torch.ones(T, dtype=torch.bool)
    h = h[keep]
    want = plain.moe_ff(h.double(), f, {k: v.double() for k, v in W.items()})
    hz = PartHarness(part)
    got = hz.feed("a", h)
    check_rows(got, want, dtype, what="routed experts")
    # an expert's weight multiplies its INPUT: through the clamps that is not the same as scaling the output
    s = torch.sigmoid(z[keep])
    experts_only = plain.moe_ff(h.double(), {**f, "shared": None}, {k: v.double() for k, v in W.items()})
    other = torch.zeros_like(want)
    for t in range(h.shape[0]):
        for e in torch.topk(s[t], top).indices.tolist():
            other[t] += s[t, e] * plain.clamped_glu(h[t:t + 1].double(), W[f"e{e}.gate"].double(), W[f"e{e}.up"].double(),
                                                    W[f"e{e}.down"].double(), f["expert"]["limit"])[0]
    assert rel_rows(experts_only, other).max() > 0.05
    # one token at a time gives the same rows as the batch
    single = torch.cat([hz.feed("b", h[t:t + 1]) for t in range(6)], 0)
    assert rel_rows(single, got[:6]).max() <= (1e-5 if dtype == "float32" else 2e-2)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_token_input_alone(dtype):
    g = gen(16)
    d, dim, V, L = 48, 8, 50, 3
    W = {"table": bf(torch.randn(V, L * dim, generator=g)), "gate": bf(torch.randn(dim, d, generator=g) / 7),
         "proj": bf(torch.randn(d, dim, generator=g) / 3), "norm": 1 + 0.2 * torch.randn(d, generator=g)}
    for layer in (0, 2):
        part = make_part("token_input", "gated_token_input",
                         {"hidden": d, "dim": dim, "offset": layer * dim, "table_width": L * dim, "vocab": V, "eps": 1e-5},
                         W, DTYPES[dtype])
        x = torch.randn(20, d, generator=g)
        ids = torch.randint(0, V, (20,), generator=g)
        from gibbs_b200.engine.step import StepState
        z = torch.zeros(1, dtype=torch.int32, device=DEV)
        step = StepState(20, 1, 0, ids.to(DEV, torch.int32), z, z, z, z, z, z, z, z)
        xd = x.to(DEV)
        part.forward(xd, step)
        want = plain.token_side(x.double(), ids, W["table"].double(), layer * dim, (layer + 1) * dim,
                                {k: W[k].double() for k in ("gate", "proj", "norm")}, 1e-5)
        assert rel_rows(xd.cpu(), want).max() <= (1e-5 if dtype == "float32" else 2e-2)


# ---------------------------------------------------------------------------
# whole models through the engine
# ---------------------------------------------------------------------------

_CACHE: dict = {}


def model_and_truth(name: str, dtype: str, lengths=(1, 2, 23, 61, 130)):
    """A model, some requests, and the plain implementation's logits for them."""
    key = (name, dtype)
    if key not in _CACHE:
        cfg, W, model = build(name, dtype)
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
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_whole_decoded_and_cut_prompts_match_the_plain_implementation(name, dtype):
    cfg, model, reqs, truth = model_and_truth(name, dtype)
    eng = engine_for(model)
    assert eng.plan is not None, eng.plan_refusal
    for what, steps in (("whole", trace_whole(reqs)), ("decoded", trace_tail_decoded(reqs, tail=40)),
                        ("cut", trace_portions(reqs))):
        got = run_trace_on_engine(eng, steps)
        for rid in reqs:
            check_rows(got[rid], truth[rid], dtype, strict=False, what=f"{name} {what} {rid}")


@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_layer_by_layer_in_float32(name):
    """The residual stream after every layer, through the parts' forward methods."""
    cfg, model, reqs, _ = model_and_truth(name, "float32")
    W = make_weights(cfg, CONFIGS[name][1])
    ids = reqs["r61"]
    _, layers = plain.forward(cfg, W, ids, collect_layers=True)
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
@pytest.mark.parametrize("name", ["A", "B"])
def test_plan_and_forward_methods_give_the_same_bits(name, dtype):
    cfg, model, reqs, _ = model_and_truth(name, dtype)
    steps = trace_mixed(reqs, capacity_tokens=320, seed=3)
    a = run_trace_on_engine(engine_for(model, n_pages=20), steps)
    b = run_trace_on_engine(engine_for(model, n_pages=20, use_plan=False, use_graphs=False), steps)
    for rid in reqs:
        assert np.array_equal(a[rid], b[rid]), rid


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_mixed_batches_with_pages_and_slots_used_again(name, dtype):
    """Up to three live requests in a pool that holds little more than the live ones, portions beside
    single tokens: against the plain implementation, and against each request run alone."""
    cfg, model, reqs, truth = model_and_truth(name, dtype)
    more = dict(reqs)
    for k in range(4):                                        # the same lengths again: slots and pages go round
        more[f"again{k}"] = ids_for(cfg, 500 + k, 40 + 17 * k)
    for seed in (0, 1):
        eng = engine_for(model, n_pages=20, max_requests=3)   # 320 tokens of pages, 3 slots
        got = run_trace_on_engine(eng, trace_mixed(more, capacity_tokens=320, max_live=3, seed=seed))
        assert eng.cache.free_pages() == [20] * len(eng.cache.groups)
        for rid in reqs:
            check_rows(got[rid], truth[rid], dtype, strict=False, what=f"{name} mixed {rid}")
        alone = run_trace_on_engine(engine_for(model), trace_whole(more))
        for rid in more:
            e = rel_rows(got[rid], alone[rid])
            lim = 1e-4 if dtype == "float32" else TOL[dtype]
            assert (e > lim).mean() <= (0.0 if dtype == "float32" else 0.45), f"{rid}: batch against alone {e.max():.3g}"


@pytest.mark.parametrize("seed", [3, 9, 11, 14, 37, 74])
def test_random_configurations_in_float32(seed):
    """Sizes, options and the order of layers drawn at random (one to five layers; one to seventeen heads;
    windows of one token and none; one expert, all experts chosen; states of 1 to 132 values; ...), whole,
    cut, decoded and in mixed batches.  Held to the plain implementation in float64, or to ten times what
    the plain implementation itself loses in float32 where a configuration is ill-conditioned (a norm
    over a handful of values)."""
    from potivik_helpers import random_config
    from gibbs_b200.config import parse_config
    from gibbs_b200.parts.model import build_model
    from gibbs_b200.weights import TensorDict
    cfg = random_config(seed)
    W = make_weights(cfg, seed)
    model = build_model(parse_config(cfg).plan(), TensorDict({k: v.to(torch.bfloat16) for k, v in W.items()}),
                        torch.float32, DEV)
    reqs = {f"r{n}": ids_for(cfg, seed * 7 + n, n) for n in (1, 2, 37, 90)}
    truth = {rid: plain.forward(cfg, W, ids).numpy() for rid, ids in reqs.items()}
    own = {rid: rel_rows(plain.forward(cfg, W, ids, dtype=torch.float32).numpy(), truth[rid]).max()
           for rid, ids in reqs.items()}
    for what, steps in (("whole", trace_whole(reqs)), ("cut", trace_portions(reqs)),
                        ("decoded", trace_tail_decoded(reqs, tail=30)),
                        ("mixed", trace_mixed(reqs, capacity_tokens=256, max_live=3, seed=seed))):
        eng = engine_for(model, n_pages=16, max_requests=3, cap=256)
        got = run_trace_on_engine(eng, steps)
        for rid in reqs:
            e = rel_rows(got[rid], truth[rid]).max()
            assert e <= max(3e-4, 10 * own[rid]), f"{what} {rid}: {e:.3g} (the plain implementation in float32: {own[rid]:.3g})"


def test_long_decoding_past_windows_pages_and_chunks():
    """260 tokens decoded one by one after a two-token prompt: every window edge, page edge and slot
    state is passed by single tokens."""
    cfg, model, _, _ = model_and_truth("A", "float32")
    W = make_weights(cfg, CONFIGS["A"][1])
    ids = ids_for(cfg, 77, 262)
    truth = plain.forward(cfg, W, ids).numpy()
    eng = engine_for(model, n_pages=20)
    got = run_trace_on_engine(eng, trace_tail_decoded({"long": ids}, tail=260))
    e = rel_rows(got["long"], truth)
    assert e.max() <= TOL["float32"], f"first wrong position {int(np.nonzero(e > TOL['float32'])[0][0])}"
    # the windowed group has given back what the window passed
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
    cfg_path.write_text(json.dumps(CFG_B))
    folder = tmp_path / "model"
    assert main(["--random", str(cfg_path), "--save", str(folder), "--seed", "3", "--dtype", "float32"]) == 0
    capsys.readouterr()
    assert main(["-m", str(folder), "--arch-dump"]) == 0
    dump = json.loads(capsys.readouterr().out)
    assert dump["architecture"] == "Potivik"
    prompt = ids_for(CFG_B, 5, 9)
    ids = ",".join(map(str, prompt))
    assert main(["-m", str(folder), "--dtype", "float32", "--probe-top5", ids, "--ctx", "128"]) == 0
    top = json.loads(capsys.readouterr().out)
    from gibbs_b200.weights import Checkpoint
    ck = Checkpoint(folder)
    W = {n: ck.tensor(n) for n in ck.names()}
    logits = plain.forward(CFG_B, W, prompt)[-1]
    assert top["ids"][0] == int(logits.argmax())
    assert abs(top["logits"][0] - float(logits.max())) < 1e-3
    assert main(["-m", str(folder), "--dtype", "float32", "--prompt-ids", ids, "--max-tokens", "5", "--temperature", "0",
                 "--ctx", "128"]) == 0
    out = capsys.readouterr().out
    generated = [int(t) for t in out.split("Output:\n")[1].splitlines()[0].split(",")]
    assert len(generated) == 5 and generated[0] == top["ids"][0]


@pytest.mark.parametrize("H,r,dr,spans", [(16, 320, 32, [(3, 560)]), (4, 448, 32, [(40, 1100)]), (4, 480, 0, [(0, 640), (17, 515)]), (16, 264, 0, [(0, 300)])])
@pytest.mark.parametrize("with_sink", [False, True])
def test_portions_without_a_window_on_the_kernel_for_wide_latents(H, r, dr, spans, with_sink):
    """Key tiles whole and in two halves (portions of 512 tokens and more, few row tiles), against 64 bits."""
    call = LatentCalls(H, r, dr, blocks=96)
    torch.manual_seed(r)
    n, longest = sum(k for _, k in spans), max(p + k for p, k in spans)
    q, gate = torch.randn(n, H, r + dr, device=DEV).bfloat16().float(), torch.randn(n, H, device=DEV)
    sink = torch.randn(H, device=DEV) if with_sink else None
    one, two = (call(q, gate, sink, spans, 0, longest, chunks=c).reshape(n, H, r).double() for c in (False, True))
    rows, at = call.pages[call.table.long()].reshape(-1, r + dr).double(), 0
    for first, k in spans:
        mine = slice(at, at + k)
        at += k
        sc = torch.einsum("nhd,ld->nhl", q[mine].double(), rows[:first + k]) * (r + dr) ** -0.5
        sc.masked_fill_((torch.arange(first + k, device=DEV) > torch.arange(first, first + k, device=DEV)[:, None])[:, None], -math.inf)
        if with_sink:
            sc = torch.cat([sc, sink.double()[None, :, None].expand(k, H, 1)], 2)
        w = torch.softmax(sc, 2)[:, :, :first + k]
        gates = torch.sigmoid(gate[mine].double())[..., None]
        want, size = (w @ rows[:first + k, :r]) * gates, (w @ rows[:first + k, :r].abs()) * gates
        # weights of 16 bits (2^-17 each), scores of some units formed in 32-bit sums of up to 576 terms (2^-16 of a weight), sums that the
        # tensor core truncates
        for got in (one, two):
            assert ((got[mine] - want).abs() <= 2.0 ** -14 * size + 1e-7).all()


# the paths beside the block kernel: rows longer than 2,048 or no multiple of 4, y in wider rows, tiles added up into y first
@pytest.mark.parametrize("d,kind,second,splits,bias,pad", [(2052, 1, True, 3, True, 0), (4096, 0, True, 16, False, 8), (4096, 1, False, 0, False, 0),
                                                           (130, 0, True, 2, True, 6), (2050, 1, False, 1, False, 2), (1027, 1, True, 0, False, 1)])
def test_norm_behind_a_sublayer_of_rows_that_no_block_takes_whole(d, kind, second, splits, bias, pad):
    import ctypes

    from gibbs_b200.ops import _stream, device_status, hybrid
    torch.manual_seed(d)
    dev, many = torch.device("cuda", torch.cuda.current_device()), 299
    x0, gain, then, add = (torch.randn(*k, device=dev) for k in ((many, d), (d,), (d,), (d,)))
    part = torch.randn(max(splits, 1), many, d, device=dev)
    y0 = part[0].clone()
    for u in range(1, splits):
        y0 += part[u]
    if bias and splits:
        y0 += add

    def run(n, tiles):
        x, parts = x0[:n].clone(), part[:, :n].contiguous()
        y = torch.full((n, d + pad), float("nan"), device=dev)
        if not tiles:
            y[:, :d] = y0[:n]
        h, copy = torch.zeros(n, d, device=dev), torch.zeros(n, d, device=dev, dtype=torch.bfloat16)
        stream = _stream()
        ctx = hybrid._Ctx(stream.value if isinstance(stream, ctypes.c_void_p) else stream, device_status(dev).data_ptr(), None, 0, None, 0, None, 0, None,
                          parts.data_ptr() if tiles else None, splits if tiles else 0, add.data_ptr() if tiles and bias else None)
        a = (ctypes.c_longlong * 24)(x.data_ptr(), d, y.data_ptr(), d + pad, gain.data_ptr(), n, d, kind, copy.data_ptr(), then.data_ptr() if second else 0,
                                     h.data_ptr() if second else 0, 0, kind)
        rc = hybrid._function("norm_add")(ctypes.byref(ctx), a, (ctypes.c_double * 3)(1e-5, 1e-5), ctypes.c_int(hybrid.TAKES_PARTIALS if tiles else 0))
        assert rc == 1 + int(tiles) + int(second and d > 2048)
        torch.cuda.synchronize()
        assert torch.equal(copy, x.bfloat16()) and (y[:, d:].isnan().all())
        return x, h

    whole = run(many, False)
    for n in (1, 296, 297, many):                            # (either side of the rule for gains ahead)
        for tiles in ((False, True) if splits else (False,)):
            got = run(n, tiles)
            assert torch.equal(got[0], whole[0][:n]) and torch.equal(got[1], whole[1][:n]), (n, tiles)

    def norm(v, g):
        v = v.double() - (v.double().mean(1, keepdim=True) if kind == 0 else 0.0)
        return v / (v.pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * g.double()
    new = x0.double() + norm(y0, gain)
    assert ((whole[0].double() - new).norm(dim=1) / new.norm(dim=1)).max() < 1e-6
    if second:
        want = norm(new, then)
        assert ((whole[1].double() - want).norm(dim=1) / want.norm(dim=1)).max() < 1e-6


# rows in 16-byte pieces (blocks for few rows and for many) and value by value; no shared expert, one that is whole, and one as partial tiles
@pytest.mark.parametrize("width,top", [(1024, 2), (2048, 1), (260, 5), (130, 3), (2048, 8)])
@pytest.mark.parametrize("splits,bias", [(-1, False), (0, False), (1, True), (9, False), (3, True)])
def test_experts_outputs_are_summed_with_a_shared_expert_in_tiles(width, top, splits, bias):
    import ctypes

    from gibbs_b200.ops import _stream, device_status, hybrid
    torch.manual_seed(width + top)
    dev, many = torch.device("cuda", torch.cuda.current_device()), 700
    e, gate = torch.randn(many * top, width, device=dev), torch.rand(many, device=dev)
    part, add = torch.randn(max(splits, 1), many, width, device=dev), torch.randn(width, device=dev)
    shared = part[0].clone()
    for u in range(1, splits):
        shared += part[u]
    if splits > 0 and bias:
        shared += add
    for n in (1, 591, 592, many):
        pair = torch.randperm(n * top, device=dev).int()
        parts, whole, y = part[:, :n].contiguous(), shared[:n].clone(), torch.full((n, width + 4), 7.0, device=dev)
        if splits > 0:
            whole.fill_(float("nan"))
        stream = _stream()
        ctx = hybrid._Ctx(stream.value if isinstance(stream, ctypes.c_void_p) else stream, device_status(dev).data_ptr(), None, 0, None, 0, None, 0, None,
                          parts.data_ptr() if splits > 0 else None, max(splits, 0), add.data_ptr() if splits > 0 and bias else None)
        a = (ctypes.c_longlong * 24)(e.data_ptr(), width, pair.data_ptr(), gate.data_ptr() if splits >= 0 else 0, whole.data_ptr() if splits >= 0 else 0,
                                     width, y.data_ptr(), width + 4, n, width, top)
        assert hybrid._function("moe_combine")(ctypes.byref(ctx), a, (ctypes.c_double * 3)(), ctypes.c_int(hybrid.TAKES_PARTIALS if splits > 0 else 0)) == 1
        torch.cuda.synchronize()
        assert (y[:, width:] == 7.0).all()
        rows = e[pair.long()].reshape(n, top, width).double()
        want, size = rows.sum(1), rows.abs().sum(1)
        if splits >= 0:
            want, size = want + gate[:n, None].double() * shared[:n].double(), size + gate[:n, None].double() * shared[:n].double().abs()
        # (a rounding for every addition; the shared row's own sums are those of the reference)
        assert ((y[:, :width].double() - want).abs() <= (top + 2) * 2.0 ** -24 * size).all(), n


# a value a thread below 512 columns a group, pieces from there, rows that are not aligned
@pytest.mark.parametrize("inner,groups,pad", [(64, 1, 0), (1016, 2, 0), (1024, 2, 0), (2048, 1, 0), (2052, 1, 0), (1024, 2, 1), (3072, 4, 4)])
@pytest.mark.parametrize("bf16", [False, True])
def test_gated_group_norm(inner, groups, pad, bf16):
    from gibbs_b200.ops import hybrid
    torch.manual_seed(inner)
    n, ld = 7, inner + pad
    y, z, gain = torch.randn(n, ld, device=DEV), torch.randn(n, ld, device=DEV), torch.randn(inner, device=DEV)
    out = torch.full((n, inner + 8), 7.0, device=DEV, dtype=torch.bfloat16 if bf16 else torch.float32)
    hybrid.call("gated_group_norm", [y.data_ptr(), ld, z.data_ptr(), ld, gain.data_ptr(), out.data_ptr(), 1 if bf16 else 0, inner + 8, n, inner, groups], [1e-5])
    v = (y[:, :inner].double() * torch.nn.functional.silu(z[:, :inner].double())).reshape(n, groups, -1)
    want = (v / (v.pow(2).mean(2, keepdim=True) + 1e-5).sqrt()).reshape(n, inner) * gain.double()
    # (32-bit: expf, a sum of squares and its root; bfloat16: half a place)
    assert ((out[:, :inner].double() - want).abs() <= (2.0 ** -8 if bf16 else 2e-6) * want.abs() + 1e-7).all() and (out[:, inner:] == 7.0).all()


# heads of up to 64, 128 and 256 values
@pytest.mark.parametrize("vdim", [1, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("second,gated,whole,silu", [(False, True, False, False), (True, False, True, False), (False, False, False, False), (True, True, True, True)])
def test_head_norm(vdim, second, gated, whole, silu):
    from gibbs_b200.ops import hybrid
    torch.manual_seed(vdim)
    n, H, eps, lam, factor = 5, 3, 1e-5, 0.3, 1.5
    x, x2, gate = (torch.randn(n, H * vdim, device=DEV) for _ in range(3))
    gain, out = torch.randn(H * vdim if whole else vdim, device=DEV), torch.empty(n, H * vdim, device=DEV)
    hybrid.call("head_norm", [x.data_ptr(), H * vdim, vdim, x2.data_ptr() if second else 0, gain.data_ptr(), gate.data_ptr() if gated else 0, H * vdim,
                              out.data_ptr(), 0, H * vdim, n, H, vdim], [eps, lam, factor], flags=(1 if whole else 0) | (2 if silu else 0))
    v = (x.double() - lam * x2.double() if second else x.double()).reshape(n, H, vdim)
    want = v / (v.pow(2).mean(2, keepdim=True) + eps).sqrt() * factor * gain.double().reshape(-1, vdim)
    if gated:
        g = gate.double().reshape(n, H, vdim)
        want = want * (torch.nn.functional.silu(g) if silu else torch.sigmoid(g))
    # (lambda is a 32-bit number here; a difference of two rounded numbers, then as above)
    assert ((out.reshape(n, H, vdim).double() - want).abs() <= 4e-6 * want.abs() + 2e-6).all()

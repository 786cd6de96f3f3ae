"""Prompt attention over a latent cache on expanded keys and values (csrc/latent_attn_tc.cu) against float64, at the edges of its
tiles of 128 queries and 64 keys, with contexts of earlier steps, windows, sinks and gates, and beside the latent form through
the part that chooses between them."""
import math

import pytest
import torch

from braidinfer_b200.csrc.api import KernelError, get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dim, rot, vdim, rank", [(128, 64, 128, 512), (64, 32, 64, 256), (64, 64, 64, 40), (128, 16, 128, 72)])
@pytest.mark.parametrize("seqs, window", [([(0, 1)], None), ([(0, 64), (0, 65)], None), ([(0, 127), (63, 129), (200, 3)], None),
                                          ([(0, 300), (130, 257)], 70), ([(500, 130)], 64), ([(64, 128), (0, 0), (1, 64)], 1)])
@pytest.mark.parametrize("extras", [False, True])
def test_expanded_attention(K, dim, rot, vdim, rank, seqs, window, extras):
    H, D = 3, rank + rot
    g = torch.Generator(device=DEV).manual_seed(rank + len(seqs))
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(n for _, n in seqs)
    q_start = [sum(n for _, n in seqs[:i]) for i in range(len(seqs))]
    before, q_len = [b for b, _ in seqs], [n for _, n in seqs]
    blocks = [-(-(b + n) // 64) for b, n in seqs]
    cols = max(blocks) + 1
    order = torch.randperm(sum(blocks) + 2, generator=torch.Generator().manual_seed(1)).tolist()
    table = [[-1] * cols for _ in seqs]
    at = 0
    for i, n in enumerate(blocks):
        first = max(0, before[i] - window + 1) // 64 if window else 0      # pages that the window has passed are gone
        for b in range(first, n):
            table[i][b] = order[at]
            at += 1
    cache = torch.full((sum(blocks) + 2, 1, 1, 64, D), float("nan"), device=DEV, dtype=BF)   # stale rows must not matter
    ctx = []
    for i, (b, n) in enumerate(seqs):
        c = rnd(b + n, D).to(BF)
        ctx.append(c)
        for p in range(b + n):
            if table[i][p // 64] >= 0:
                cache[table[i][p // 64], 0, 0, p % 64] = c[p]
    proj = rnd(rows, H * (dim + rot) + 8).to(BF)
    q_u = proj[:, :H * (dim + rot)].view(rows, H, dim + rot)[:, :, :dim]
    q_lat = torch.full((rows, H, D), float("nan"), device=DEV, dtype=BF)
    q_lat[:, :, rank:] = rnd(rows, H, rot).to(BF)
    uk, uv = (rnd(H * dim, rank) * rank ** -0.5).to(BF), (rnd(H * vdim, rank) * rank ** -0.5).to(BF)
    sinks = rnd(H) if extras else None
    gate = rnd(rows, H + 2).to(BF)[:, 1:H + 1] if extras else None
    mult, scale = (0.7, (dim + rot) ** -0.5) if extras else (1.0, (dim + rot) ** -0.5)
    pages = K.latent_pages(q_len, before, window)
    t = i32(table)
    rows_c = K.latent_expand_rows(cache, t, i32(q_len), i32(before), rank, window, pages)
    at = 0
    for i, (b, n) in enumerate(seqs):                                  # the context, page by page, zeros past its end
        first = max(0, b - window + 1) // 64 * 64 if window else 0
        if n == 0:
            continue
        got = rows_c[at:at + pages[i] * 64]
        assert torch.equal(got[:b + n - first], ctx[i][first:, :rank]) and (got[b + n - first:] == 0).all()
        at += pages[i] * 64
    assert at == rows_c.shape[0]
    kv = torch.empty(rows_c.shape[0], H * (dim + vdim), device=DEV, dtype=BF)
    K.gemm_tc(rows_c, torch.cat([uk, uv]), kv)
    out = torch.full((rows, H * vdim), 9.0, device=DEV, dtype=BF)
    K.attn_latent_tc(q_u, q_lat, kv, cache, out, t, i32(q_start), i32(q_len), i32(before), len(seqs), max(q_len), vdim, rank, window,
                     scale, out_scale=mult, sinks=sinks, gate=gate)
    K.check_device_errors()
    worst = 0.0
    for i, (b, n) in enumerate(seqs):
        if n == 0:
            continue
        c = ctx[i].double()
        # keys and values as the kernel gets them: rounded to bfloat16 after the expansion
        ku = (c[:, :rank] @ uk.double().T).to(BF).double().view(b + n, H, dim)
        v = (c[:, :rank] @ uv.double().T).to(BF).double().view(b + n, H, vdim)
        q = slice(q_start[i], q_start[i] + n)
        s = torch.einsum("qhd,khd->hqk", q_u[q].double(), ku) + torch.einsum("qhr,kr->hqk", q_lat[q, :, rank:].double(), c[:, rank:])
        s = s * scale
        dist = torch.arange(b, b + n, device=DEV)[:, None] - torch.arange(b + n, device=DEV)[None]
        hidden = (dist < 0) | ((dist >= window) if window else False)
        s = s.masked_fill(hidden, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None, None].expand(H, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :b + n]
        want = torch.einsum("hqk,khd->qhd", p, v) * mult
        if gate is not None:
            want = want * torch.sigmoid(gate[q].double())[:, :, None]
        err = (out[q].double().view(n, H, vdim) - want).abs()
        # probabilities rounded to bfloat16 (2^-8 of each), keys that sit on a rounding edge (2^-8 of their score's terms), the
        # result rounded once: a few parts in 2^8 of the values' size
        size = torch.einsum("hqk,khd->qhd", p, v.abs()) * mult
        worst = max(worst, float((err / (size + 0.05)).max()))
    assert worst < 4 * 2.0 ** -8


@pytest.mark.parametrize("chunks", [[700], [300, 400], [40, 660], [690, 10]])
def test_the_part_that_chooses(monkeypatch, chunks):
    """A Bidinex model of one layer: prompts whole and in portions (the later ones expand the earlier ones' latents again), beside
    the same engine with the latent form."""
    from braidinfer_b200.engine import Engine
    import braidinfer_b200.parts.latent_attention as LA
    mixer = {"heads": 4, "dim": 64, "rot_dim": 32, "rot": {"base": 10000.0, "dims": 32}, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 4, "top": 2, "groups": {"count": 1, "keep": 1}}}
    cfg = {"architecture": "Bidinex", "vocab": 256, "width": 128, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
           "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    eng = Engine.from_random(cfg, 3, max_tokens=2048, max_slots=2, verbose=False)
    toks = torch.randint(0, 256, (sum(chunks),), generator=torch.Generator().manual_seed(2)).tolist()

    def logits():
        s, at, out = eng.open(), 0, []
        for n in chunks:
            out.append(eng.step([(s, toks[at:at + n])], want="all"))
            at += n
        eng.close(s)
        eng.check()
        return torch.cat(out).double()

    calls = []
    kernel = type(eng.kernels).attn_latent_tc
    monkeypatch.setattr(type(eng.kernels), "attn_latent_tc", lambda self, *a, **kw: (calls.append(1), kernel(self, *a, **kw)))
    got = logits()
    assert len(calls) == sum(n > 256 for n in chunks)                  # steps of up to 256 tokens keep the latent form
    monkeypatch.setattr(LA, "EXPAND_BYTES", 0)
    calls.clear()
    want = logits()
    assert not calls
    # both are bfloat16 of the same mechanism; the model's tests ask 1e-2 .. 2e-2 of either beside float64
    assert float((got - want).norm() / want.norm()) < 1e-2


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_score_factors_that_are_not_positive(K, monkeypatch, scale):
    """The kernel masks before the factor, so it refuses such a factor and prompts keep the latent form."""
    from braidinfer_b200.engine import Engine
    import braidinfer_b200.parts.latent_attention as LA
    mixer = {"heads": 4, "dim": 64, "rot_dim": 32, "rot": {"base": 10000.0, "dims": 32}, "vdim": 64, "kv_rank": 256, "scale": scale}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 4, "top": 2, "groups": {"count": 1, "keep": 1}}}
    cfg = {"architecture": "Bidinex", "vocab": 256, "width": 128, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
           "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    eng = Engine.from_random(cfg, 3, max_tokens=512, max_slots=1, verbose=False)
    toks = torch.randint(0, 256, (300,), generator=torch.Generator().manual_seed(2)).tolist()

    def logits():
        s = eng.open()
        out = eng.step([(s, toks)], want="all")
        eng.close(s)
        eng.check()
        return out

    got = logits()
    monkeypatch.setattr(LA, "EXPAND_BYTES", 0)
    assert torch.isfinite(got).all() and torch.equal(got, logits())
    z = lambda *s: torch.zeros(*s, device=DEV, dtype=BF)
    with pytest.raises(KernelError, match="positive"):
        K.attn_latent_tc(z(1, 1, 64), z(1, 1, 80), z(64, 128), z(1, 1, 1, 64, 80), z(1, 64), i32([[0]]), i32([0]), i32([1]), i32([0]), 1, 1,
                         64, 64, None, scale)


def test_gate_is_float32(K):
    """One visible key a query, so that the result is its value times the gate's sigmoid, rounded once to bfloat16 after float32 errors
    of a few units (an exponential good to two, a division, the products)."""
    H, dim, rot, vdim, rank, n = 64, 64, 16, 64, 64, 256
    g = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(BF)
    kv, gate = rnd(n, H * (dim + vdim)), -40 * torch.rand(n, H, device=DEV, generator=g).to(BF)
    out = torch.empty(n, H * vdim, device=DEV, dtype=BF)
    K.attn_latent_tc(rnd(n, H, dim), rnd(n, H, rank + rot), kv, rnd(4, 1, 1, 64, rank + rot), out, i32([[0, 1, 2, 3]]), i32([0]), i32([n]),
                     i32([0]), 1, n, vdim, rank, 1, 0.1, gate=gate)
    K.check_device_errors()
    want = (kv[:, H * dim:].double().view(n, H, vdim) * torch.sigmoid(gate.double())[:, :, None]).view(n, -1)
    half_step = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 8)
    assert ((out.double() - want).abs() <= half_step + 8 * 2.0 ** -24 * want.abs()).all()


def test_small_probabilities(K):
    """Two keys, one 2^-130 as likely as the other: bfloat16 holds that number, and its value of 2^125 shows it."""
    dim, rot, vdim, rank = 64, 16, 64, 64
    z = lambda *s: torch.zeros(*s, device=DEV, dtype=BF)
    q_u, kv, out = z(2, 1, dim), z(64, dim + vdim), z(2, vdim)
    q_u[1, 0, 0], kv[0, 0], kv[0, dim:] = 1.0, -130.0, 2.0 ** 125
    K.attn_latent_tc(q_u, z(2, 1, rank + rot), kv, z(1, 1, 1, 64, rank + rot), out, i32([[0]]), i32([0]), i32([2]), i32([0]), 1, 2, vdim, rank,
                     None, math.log(2.0))
    K.check_device_errors()
    assert ((out[1].double() - 2.0 ** -5).abs() <= 2.0 ** -5 * 2.0 ** -7).all()


def test_steps_that_graphs_hold_keep_the_latent_form(monkeypatch):
    """Whatever the engine's limit is: replays of a 300-token step behind other contexts give the bits of steps without graphs."""
    import braidinfer_b200.engine.engine as E
    mixer = {"heads": 4, "dim": 64, "rot_dim": 32, "rot": {"base": 10000.0, "dims": 32}, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 4, "top": 2, "groups": {"count": 1, "keep": 1}}}
    cfg = {"architecture": "Bidinex", "vocab": 256, "width": 128, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
           "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    monkeypatch.setattr(E, "GRAPH_PROMPT_ROWS", 512)
    toks = torch.randint(0, 256, (2000,), generator=torch.Generator().manual_seed(2)).tolist()
    res = []
    for graphs in (True, False):
        eng = E.Engine.from_random(cfg, 3, max_tokens=2048, max_slots=1, use_graphs=graphs, verbose=False)
        out = []
        for n in (0, 100, 37, 140):
            s = eng.open()
            if n:
                eng.step([(s, toks[:n])])
            out.append(eng.step([(s, toks[n:n + 300])]))
            eng.close(s)
        eng.check()
        assert (eng.graph_replays > 0) == graphs
        res.append(torch.cat(out))
    assert torch.equal(*res)


def test_sequences_below_the_least_number_of_queries_are_left_out(K):
    """Their pages are not laid out and their rows not written; the others' rows are those of a step without them."""
    H, dim, rot, vdim, rank = 2, 64, 16, 64, 64
    g = torch.Generator(device=DEV).manual_seed(9)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(BF)
    seqs = [(0, 3), (64, 70), (5, 1), (0, 129), (300, 4)]
    cache, table = rnd(16, 1, 1, 64, rank + rot), [[3, 4, 5, 6, 7], [0, 1, 2, -1, -1], [8] + [-1] * 4, [9, 10, 11, -1, -1], [12, 13, 14, 15, 3]]
    uk_uv = (rnd(H * (dim + vdim), rank).float() * rank ** -0.5).to(BF)
    n = sum(q for _, q in seqs)
    q_u, q_lat = rnd(n, H, dim), rnd(n, H, rank + rot)
    start = [sum(q for _, q in seqs[:i]) for i in range(len(seqs))]

    def run(pick, min_q):
        q_len, before = [seqs[i][1] for i in pick], [seqs[i][0] for i in pick]
        tables = i32([table[i] for i in pick]), i32(q_len), i32(before)
        pages = K.latent_pages(q_len, before, None, min_q)
        rows = K.latent_expand_rows(cache, *tables, rank, None, pages, min_q)
        kv, out = torch.empty(rows.shape[0], H * (dim + vdim), device=DEV, dtype=BF), torch.full((n, H * vdim), 9.0, device=DEV, dtype=BF)
        K.gemm_tc(rows, uk_uv, kv)
        K.attn_latent_tc(q_u, q_lat, kv, cache, out, tables[0], i32([start[i] for i in pick]), *tables[1:], len(pick), max(q_len), vdim, rank,
                         None, 0.1, min_q=min_q)
        K.check_device_errors()
        return pages, out

    pages, got = run(range(5), 4)
    assert pages == [0, 3, 0, 3, 5]
    _, want = run([1, 3, 4], 1)
    assert torch.equal(got, want) and (got[:3] == 9.0).all() and (got[73] == 9.0).all() and (got[74:] != 9.0).any()


def test_a_prompt_beside_sequences_that_decode(monkeypatch):
    """Every sequence is looked at by itself: long contexts that one query meets are not expanded because of the prompt beside them."""
    from braidinfer_b200.engine import Engine
    import braidinfer_b200.parts.latent_attention as LA
    mixer = {"heads": 4, "dim": 64, "rot_dim": 32, "rot": {"base": 10000.0, "dims": 32}, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 4, "top": 2, "groups": {"count": 1, "keep": 1}}}
    cfg = {"architecture": "Bidinex", "vocab": 256, "width": 128, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
           "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    eng = Engine.from_random(cfg, 3, max_tokens=64 * 64, max_slots=6, verbose=False)
    toks = torch.randint(0, 256, (1000,), generator=torch.Generator().manual_seed(2)).tolist()
    before, n = [600, 0, 700, 130, 0, 515], [1, 300, 1, 20, 10, 1]
    seen = []
    expand = type(eng.kernels).latent_expand_rows
    monkeypatch.setattr(LA, "EXPAND_BESIDE_FLOPS", 0)                 # however little they cost here
    monkeypatch.setattr(type(eng.kernels), "latent_expand_rows", lambda self, *a, **kw: (seen.append(list(a[6])), expand(self, *a, **kw))[1])

    def logits():
        slots = [eng.open() for _ in n]
        for s, b in zip(slots, before):
            if b:
                eng.step([(s, toks[:b])])
        seen.clear()
        out = eng.step([(s, toks[b:b + q]) for s, b, q in zip(slots, before, n)], want="all").double()
        for s in slots:
            eng.close(s)
        eng.check()
        return out

    got = logits()
    assert seen == [[0, 5, 0, 3, 0, 0]]
    monkeypatch.setattr(LA, "EXPAND_BYTES", 0)
    want = logits()
    assert not seen
    at = [sum(n[:i]) for i in range(len(n) + 1)]
    for a, b in zip(at, at[1:]):                                      # as test_the_part_that_chooses asks
        assert float((got[a:b] - want[a:b]).norm() / want[a:b].norm()) < 1e-2

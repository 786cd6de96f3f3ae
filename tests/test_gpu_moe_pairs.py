"""The experts' products on pairs of SMs (csrc/moe_tc.cu) and the plan that they walk, at the edges of their tiles: experts
without rows, with one, with a chunk of 32 slots more or less one, with more than a run of eight chunks."""
import pytest
import torch

from braidinfer_b200.csrc.api import MOE_TC_TILE, expert_halves, get_kernels, interleave_experts, interleave_gate_up

pytestmark = pytest.mark.gpu
DEV = "cuda"
# Rounding moves a number by at most half a step: 2^-24 of it in float32 (24 bits), 2^-8 in bfloat16 (8 bits); a sum that the
# tensor cores cut off instead of rounding by a whole step, 2^-23.
U = 2.0 ** -23


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def choice(counts, top, seed):
    """idx [rows, top]: expert e gets counts[e] pairs, in a shuffled order; -1 fills up the last row."""
    flat = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)])
    flat = flat[torch.randperm(flat.numel(), generator=torch.Generator().manual_seed(seed))]
    pad = -flat.numel() % top
    return torch.cat([flat, torch.full((pad,), -1)]).view(-1, top).to(torch.int32).to(DEV)


COUNTS = [[0, 1, 31, 32, 33], [255, 0, 256, 257], [300, 520, 3], [1], [40] * 70, [3000, 1]]


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("tile", [16, 32, 64])
def test_plan(K, counts, tile):
    top = 3
    idx = choice(counts, top, 1)
    rows = idx.shape[0]
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    seq[rows // 2] = -1                                              # a row of padding takes no slot
    plan = [t.cpu() if torch.is_tensor(t) else t for t in K.moe_plan(idx, seq, len(counts), tile)]
    slot_pair, pair_slot, tile_expert, meta, max_tiles = plan[:5]
    live = idx.cpu().clone()
    live[rows // 2] = -1
    real = [int((live == e).sum()) for e in range(len(counts))]
    assert meta[0] == sum(-(-n // tile) for n in real) <= max_tiles
    for pair, (e, slot) in enumerate(zip(live.view(-1).tolist(), pair_slot.tolist())):
        assert (slot < 0) == (e < 0)
        if slot >= 0:
            assert slot_pair[slot] == pair and tile_expert[slot // tile] == e
    assert int((slot_pair >= 0).sum()) == sum(real)
    if tile == MOE_TC_TILE:
        wide = plan[5].view(-1, 4)[:meta[1]].tolist()
        assert len(wide) == sum(-(-n // 256) for n in real)
        at = 0
        for w, (slot, chunks, first, runs) in enumerate(wide):       # every tile once, in order, an expert's runs alike
            e = int(tile_expert[slot // tile])
            assert slot == at and 1 <= chunks <= 8 and (tile_expert[slot // tile:slot // tile + chunks] == e).all()
            assert first <= w < first + runs and runs == -(-real[e] // 256)
            at += chunks * tile
        assert at == meta[0] * tile


# pairs for a cluster of eight CTAs, with one turn of its loops and (past 32,768) with two; as many experts as there may be
@pytest.mark.parametrize("counts", [[1400, 1400, 1399], [192] * 64, [5000, 0, 9000, 1, 11000, 8200], [e % 7 for e in range(1024)], [0] * 1023 + [40]])
@pytest.mark.parametrize("tile", [16, 32])
def test_plan_of_long_prompts(K, counts, tile):
    top, experts = 3, len(counts)
    idx = choice(counts, top, 4)
    rows = idx.shape[0]
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    seq[rows // 2] = -1                                              # a row of padding takes no slot
    plan = K.moe_plan(idx, seq, experts, tile)
    slot_pair, pair_slot, tile_expert, meta, max_tiles = plan[:5]
    live = idx.clone().long()
    live[rows // 2] = -1
    live = live.view(-1)
    real = torch.bincount(live[live >= 0], minlength=experts)
    tiles = -(-real // tile)
    assert int(meta[0]) == int(tiles.sum()) <= max_tiles
    assert torch.equal(tile_expert[:int(meta[0])].long(), torch.repeat_interleave(torch.arange(experts, device=DEV), tiles))
    assert torch.equal(pair_slot >= 0, live >= 0)
    pair = torch.nonzero(live >= 0).view(-1)
    slot = pair_slot[pair].long()
    assert torch.equal(slot_pair[slot].long(), pair) and torch.equal(tile_expert[slot // tile].long(), live[pair])
    assert int((slot_pair >= 0).sum()) == pair.numel()
    if tile == MOE_TC_TILE:
        runs = -(-tiles // 8)
        wide = plan[5].view(-1, 4)[:int(meta[1])].long()
        assert wide.shape[0] == int(runs.sum())
        owner = torch.repeat_interleave(torch.arange(experts, device=DEV), runs)
        first = torch.cumsum(runs, 0) - runs
        assert torch.equal(wide[:, 2], first[owner]) and torch.equal(wide[:, 3], runs[owner])
        assert torch.equal(wide[:, 0], (torch.cumsum(wide[:, 1], 0) - wide[:, 1]) * tile) and int(wide[:, 1].sum()) == int(meta[0])
        assert int(wide[:, 1].min()) >= 1 and int(wide[:, 1].max()) <= 8
        assert torch.equal(tile_expert[wide[:, 0] // tile].long(), owner)


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("j, k", [(8, 8), (24, 40), (64, 64), (136, 72), (264, 200), (520, 520)])
@pytest.mark.parametrize("mode", ["plain", "gated", "gated, weight on the input", "relu2"])
def test_products(K, counts, j, k, mode):
    top, experts = 2, len(counts)
    g = torch.Generator(device=DEV).manual_seed(j + k + experts)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    idx = choice(counts, top, 2)
    rows = idx.shape[0]
    x = rnd(rows, k + 8).to(torch.bfloat16)[:, :k]                    # rows further apart than they are long
    w0, w1 = [(rnd(experts, j, k) * k ** -0.5).to(torch.bfloat16) for _ in range(2)]
    wgt = torch.rand(rows, top, device=DEV, generator=g)
    plan = K.moe_plan(idx, torch.zeros(rows, dtype=torch.int32, device=DEV), experts, MOE_TC_TILE)
    xs = K.moe_gather(x, plan, top)
    out = torch.full((xs.shape[0], j), 3.0, device=DEV, dtype=torch.bfloat16)
    gated = mode.startswith("gated")
    in_wgt = wgt if "weight" in mode else None
    K.moe_gemm_tc(xs, interleave_experts(w0, w1) if gated else w0, out, plan, gated=gated, relu2=mode == "relu2", in_wgt=in_wgt)
    K.check_device_errors()
    slot_pair = plan[0].long()
    used = int(plan[3][0]) * MOE_TC_TILE
    live = slot_pair >= 0
    assert (xs[:used][~live[:used]] == 0).all() and torch.equal(xs[live], x[slot_pair[live] // top])
    expert = idx.view(-1).long()[slot_pair[live]]
    xd = xs[live].double()
    prod = lambda w: torch.einsum("nk,njk->nj", xd, w[expert].double())
    size = lambda w: torch.einsum("nk,njk->nj", xd.abs(), w[expert].double().abs())
    e0, e1 = k * U * size(w0), k * U * size(w1)                      # float32 sums in any order, off by at most this
    if gated:
        s = wgt.view(-1)[slot_pair[live]].double()[:, None] if in_wgt is not None else 1.0
        a, b, e0, e1 = prod(w0) * s, prod(w1) * s, e0 * s, e1 * s
        want = a * torch.sigmoid(a) * b
        slack = 1.1 * e0 * b.abs() + (a * torch.sigmoid(a)).abs() * e1 + 1.1 * e0 * e1
    elif mode == "relu2":
        want = prod(w0).clamp_min(0) ** 2
        slack = 2 * e0 * prod(w0).abs() + e0 * e0
    else:
        want, slack = prod(w0), e0
    # one rounding to bfloat16, and a part in 2^14 for the float32 activation
    assert ((out[live].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -14) * want.abs() + 1.01 * slack + 1e-30).all()
    if used < out.shape[0]:
        assert (out[used:] == 3.0).all()                              # nothing is written past the plan's tiles


def test_activation_is_float32(K):
    """Inputs that pick single weights, so that gate and up are exact: the result is silu(gate) * up rounded once to bfloat16 after
    float32 errors of a few units (an exponential good to two, a division, two products), down to where silu is as small as
    bfloat16's smallest normal numbers."""
    gates = torch.cat([torch.linspace(-88.0, -60.0, 64), torch.linspace(-60.0, 8.0, 192)]).to(torch.bfloat16).to(DEV)
    ups = torch.linspace(1.0, 2.0, 129)[:128].to(torch.bfloat16).to(DEV)
    w0 = torch.zeros(1, gates.numel() * 128, 8, device=DEV, dtype=torch.bfloat16)
    w1 = torch.zeros_like(w0)
    w0[0, :, 0], w1[0, :, 1] = gates.repeat_interleave(128), ups.repeat(gates.numel())
    x = torch.tensor([[1.0, 1.0] + [0.0] * 6], device=DEV, dtype=torch.bfloat16)
    zero = torch.zeros(1, dtype=torch.int32, device=DEV)
    plan = K.moe_plan(zero[None], zero, 1, MOE_TC_TILE)
    xs = K.moe_gather(x, plan, 1)
    out = torch.empty(xs.shape[0], w0.shape[1], device=DEV, dtype=torch.bfloat16)
    K.moe_gemm_tc(xs, interleave_experts(w0, w1), out, plan, gated=True)
    g, u = w0[0, :, 0].double(), w1[0, :, 1].double()
    want = g * torch.sigmoid(g) * u
    half_step = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 8)
    assert ((out[0].double() - want).abs() <= half_step + 8 * 2.0 ** -24 * want.abs()).all()


@pytest.mark.parametrize("experts, j, k", [(1, 8, 8), (5, 24, 40), (7, 33, 9), (3, 16, 72), (40, 1040, 1024)])
def test_laying_out_the_experts(experts, j, k):
    """Every expert's rows as `interleave_gate_up` lays them, with no second copy of the weights on the way."""
    g = torch.Generator(device=DEV).manual_seed(j)
    gate, up = [[torch.randn(j, k, device=DEV, generator=g).to(torch.bfloat16) for _ in range(experts)] for _ in range(2)]
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    w = interleave_experts(gate, up)
    assert torch.cuda.max_memory_allocated() - before <= w.numel() * 2 + (60 << 20)
    for e in range(experts):
        assert torch.equal(w[e], interleave_gate_up(gate[e], up[e]))


def test_views_of_the_interleaved_stack_are_the_stack(K):
    """The kernels of few rows read gate and up as blocks of 16 rows of the stack: the bits of separate tensors."""
    g = torch.Generator(device=DEV).manual_seed(0)
    experts, j, k, rows, top = 5, 40, 72, 33, 2
    w0, w1 = [torch.randn(experts, j, k, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2)]
    x = torch.randn(rows, k, device=DEV, generator=g).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(experts, generator=torch.Generator().manual_seed(r))[:top] for r in range(rows)]).int().to(DEV)
    halves = expert_halves(interleave_experts(w0, w1))
    for tile in (16, 64):
        plan = K.moe_plan(idx, torch.zeros(rows, dtype=torch.int32, device=DEV), experts, tile)
        for fn in (K.moe_gemm_mma, K.moe_gemm_simt):
            res = []
            for a, b in ((w0, w1), halves):
                out = torch.zeros(plan[4] * tile, j, device=DEV, dtype=torch.bfloat16)
                fn(x, a, b, out, plan, top, tile)
                res.append(out)
            assert torch.equal(*res)


@pytest.mark.parametrize("rows, width, top, pad", [(1, 8, 1, 0), (3, 2048, 6, 0), (5, 520, 9, 8), (4, 1001, 3, 0), (2, 516, 17, 4), (700, 40, 2, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("weighted", [True, False])
def test_weighted_sum(K, rows, width, top, pad, dtype, weighted):
    """Widths and strides that allow 16-byte loads and ones that do not, more choices than are asked for at once, pairs without a slot."""
    g = torch.Generator(device=DEV).manual_seed(rows + width)
    slots = rows * top + 5
    y = torch.randn(slots, width + pad, device=DEV, generator=g).to(dtype)[:, :width]
    h = torch.randn(rows, width, device=DEV, generator=g)
    wgt = torch.rand(rows, top, device=DEV, generator=g)
    at = torch.randperm(slots, device=DEV, generator=g)[:rows * top].int()
    at[::7] = -1
    w = (wgt if weighted else torch.ones_like(wgt)).double() * (at.view(rows, top) >= 0)
    terms = w[:, :, None] * y[at.clamp_min(0).long().view(rows, top)].double()
    want = h.double() + terms.sum(1)
    most = (top + 1) * U * (h.double().abs() + terms.abs().sum(1))
    K.moe_combine(h, y, (None, at), wgt if weighted else None, top=top)
    assert ((h.double() - want).abs() <= most).all()


def test_inputs_of_the_slots_take_no_memory_of_their_own(monkeypatch):
    """A step's peak grows by the slots' results and inner rows, not by their gathered inputs too; twice the same bits."""
    from braidinfer_b200.csrc.api import Kernels
    from braidinfer_b200.engine import Engine
    mixer = {"heads": 4, "dim": 64, "rot_dim": 32, "rot": {"base": 10000.0, "dims": 32}, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 8, "top": 4, "groups": {"count": 1, "keep": 1}}}
    cfg = {"architecture": "Bidinex", "vocab": 256, "width": 256, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
           "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    eng = Engine.from_random(cfg, 3, max_tokens=640, max_slots=1, verbose=False)
    wrote = []
    gather, product = Kernels.moe_gather, Kernels.moe_gemm_tc
    monkeypatch.setattr(Kernels, "moe_gather", lambda self, *a, **kw: (wrote.append(gather(self, *a, **kw)), wrote[-1])[1])
    monkeypatch.setattr(Kernels, "moe_gemm_tc", lambda self, xs, w, out, *a, **kw: (wrote.append(out), product(self, xs, w, out, *a, **kw))[1])
    res = []
    for _ in range(2):
        s = eng.open()
        wrote.clear()
        res.append(eng.step([(s, [(7 * i) % 256 for i in range(600)])]))
        inputs, inner, results = wrote
        assert inputs.data_ptr() == results.data_ptr() != inner.data_ptr()
        eng.close(s)
    eng.check()
    assert torch.equal(*res)

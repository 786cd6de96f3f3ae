"""The recurrence with one decay a head over chunks on the tensor cores (csrc/scan_mma.cu) beside float64 and beside the walk token
by token: sequences shorter than a chunk, at its edge and past it, portions that continue from a stored state, steep and flat decays."""
import types

import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def step(lens, slots):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(n_seqs=len(lens), max_q_len=max(lens), q_start=i32([sum(lens[:i]) for i in range(len(lens))]),
                                 q_len=i32(lens), slot_ids=i32(slots))


@pytest.mark.parametrize("heads, groups, dk, dv", [(4, 2, 128, 64), (3, 1, 64, 128), (2, 2, 64, 64)])
@pytest.mark.parametrize("lens", [[17], [64, 1], [65, 63, 128], [300, 0, 2]])
@pytest.mark.parametrize("decay", [-6.0, -1.0, 3.0])                     # from a state that hardly fades to one that a token wipes out
@pytest.mark.parametrize("with_skip", [True, False])
def test_chunks(K, heads, groups, dk, dv, lens, decay, with_skip):
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + dk)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(lens)
    q, k = (rnd(rows, groups * dk + 8).to(BF)[:, :groups * dk] for _ in range(2))
    v, gate = rnd(rows, heads * dv).to(BF), rnd(rows, heads + 1).to(BF)[:, :heads]
    bias, a_log, skip = rnd(heads).to(BF), (rnd(heads) * 0.3 + decay).to(BF), rnd(heads).to(BF) if with_skip else None
    slots = list(range(1, len(lens) + 1))
    S0 = rnd(len(lens) + 2, heads, dk, dv)
    offset = 16
    res = {}
    for chunk in (None, 0):                                             # the tensor cores' form, the walk
        state = torch.zeros(len(lens) + 2, offset + heads * dk * dv * 4, dtype=torch.uint8, device=DEV)
        state[:, offset:] = S0.reshape(S0.shape[0], -1).view(torch.uint8)
        out = torch.full((rows, heads * dv), 7.0, device=DEV)
        at = 0
        cuts = [[n - n // 3 for n in lens], [n // 3 for n in lens]] if max(lens) > 100 else [lens]
        done = [0] * len(lens)
        start = [sum(lens[:i]) for i in range(len(lens))]
        for cut in cuts:
            pick = torch.cat([torch.arange(start[i] + done[i], start[i] + done[i] + cut[i]) for i in range(len(lens))]).to(DEV)
            o = torch.full((pick.numel() + 1, heads * dv), 7.0, device=DEV)
            K.linear_scan(q[pick], k[pick], v[pick], gate[pick], bias, o[:-1], state, offset, step(cut, slots), heads, groups, dk, dv, "head",
                          q_scale=0.5, a_log=a_log, skip=skip, chunk=chunk)
            assert (o[-1] == 7.0).all()
            out[pick] = o[:-1]
            done = [a + b for a, b in zip(done, cut)]
        assert (state[:, :offset] == 0).all()
        got = state[:, offset:].contiguous().view(torch.float32).view(S0.shape)
        assert torch.equal(got[0], S0[0]) and torch.equal(got[-1], S0[-1])
        res[chunk] = out, got
    errors = {None: [], 0: []}
    of = torch.arange(heads, device=DEV) // (heads // groups)
    for i, n in enumerate(lens):
        S, at = S0[slots[i]].double(), sum(lens[:i])
        want = torch.empty(n, heads, dv, dtype=torch.float64, device=DEV)
        for t in range(n):
            dt = torch.nn.functional.softplus(gate[at + t].double() + bias.double(), threshold=50)
            kt, vt = k[at + t].double().view(groups, dk)[of], v[at + t].double().view(heads, dv)
            S = torch.exp(-torch.exp(a_log.double()) * dt)[:, None, None] * S + (dt[:, None] * kt)[:, :, None] * vt[:, None]
            want[t] = torch.einsum("hkv,hk->hv", S, q[at + t].double().view(groups, dk)[of] * 0.5)
            if skip is not None:
                want[t] += skip.double()[:, None] * vt
        for chunk, (out, state) in res.items():
            rel = lambda a, b: float((a.double() - b).norm() / b.norm())
            errors[chunk].append(max(rel(out[at:at + n].view(n, heads, dv), want) if n else 0.0, rel(state[slots[i]], S)))
    # sums of float32 numbers in another order: as far from float64 as the walk is, and never past a part in 2^19
    assert max(errors[None]) < 1.5 * max(errors[0]) + 2.0 ** -22 and max(errors[None]) < 2.0 ** -19


def scan(K, dk, tokens, spoil=None, chunk=None):
    heads, groups, dv = 2, 1, 64
    g = torch.Generator(device=DEV).manual_seed(dk)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v, gate = rnd(tokens, groups * dk).to(BF), rnd(tokens, groups * dk).to(BF), rnd(tokens, heads * dv).to(BF), rnd(tokens, heads).to(BF)
    bias, a_log, S = rnd(heads).to(BF), (rnd(heads) * 0.3 - 6.0).to(BF), rnd(1, heads, dk, dv)
    if spoil:
        spoil({"q": q, "k": k, "v": v, "gate": gate, "state": S})
    out = torch.empty(tokens, heads * dv, device=DEV)
    K.linear_scan(q, k, v, gate, bias, out, S.view(1, -1).view(torch.uint8), 0, step([tokens], [0]), heads, groups, dk, dv, "head",
                  a_log=a_log, chunk=chunk)
    return out


@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("at", [1, 9, 15, 16, 40, 79])
@pytest.mark.parametrize("what", ["q", "k", "v", "gate"])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan"), 3e38])
def test_a_token_leaves_the_tokens_before_it_alone(K, dk, at, what, bad):
    """Numbers that are not finite, or whose products are not: the bits of earlier tokens stay, a value's other columns too, and the
    results that are finite are those of the walk."""
    def spoil(t):
        t[what][at, 1] = bad

    clean, got, walk = scan(K, dk, 80), scan(K, dk, 80, spoil), scan(K, dk, 80, spoil, chunk=0)
    keep = torch.arange(80, device=DEV) != at if what == "q" else torch.arange(80, device=DEV) < at
    assert torch.equal(got[keep], clean[keep])
    if what == "v":
        assert torch.equal(got[:, 2:], clean[:, 2:]) and torch.equal(got[:, :1], clean[:, :1])
    if bad != 3e38 and not (what == "gate" and bad < 0):                # (a step that softplus makes zero: 0 times a number)
        assert torch.equal(torch.isfinite(got), torch.isfinite(walk))


@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("big", [float("inf"), float("-inf"), 3.4e38])
def test_the_largest_numbers_of_a_state(K, dk, big):
    """3.4e38 is past the largest bfloat16 number: its three parts must be finite, and an infinity's must not be NaN."""
    def spoil(t):
        t["state"][0, 1, 5, 3] = big
        t["q"] *= 2.0 ** -8

    got, walk = (scan(K, dk, 40, spoil, chunk=c) for c in (None, 0))
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(got), same(walk))
    ok = torch.isfinite(walk)
    assert float((got[ok].double() - walk[ok].double()).norm() / walk[ok].double().norm()) < 2.0 ** -18


@pytest.mark.parametrize("heads, dk, tokens, serial", [(8, 128, 300, True), (8, 128, 2048, False), (16, 128, 2048, False), (64, 128, 2048, True),
                                                       (32, 64, 700, True), (32, 64, 2048, False), (4, 64, 384, True), (4, 64, 385, False), (4, 128, 257, False)])
def test_the_form_follows_ctas_and_length(K, heads, dk, tokens, serial):
    """A long prompt on few CTAs keeps the walk whose chunks run side by side (three launches), whatever its keys' size."""
    z = lambda *s: torch.zeros(*s, device=DEV, dtype=BF)
    before = K.launches
    K.linear_scan(z(tokens, dk), z(tokens, dk), z(tokens, heads * 64), z(tokens, heads), z(heads), torch.empty(tokens, heads * 64, device=DEV),
                  torch.zeros(1, heads * dk * 64 * 4, dtype=torch.uint8, device=DEV), 0, step([tokens], [0]), heads, 1, dk, 64, "head", a_log=z(heads))
    assert (K.launches - before == 1) == serial == K.ssd_pays(tokens, tokens, heads, dk, 64)
    assert not K.ssd_pays(16, 16, 64, 128, 64)
    assert not K.ssd_pays(2048 + 192, 2048, 16, 128, 64) and K.ssd_pays(4 * 2048, 2048, 16, 128, 64)    # beside short ones, or equals


@pytest.mark.parametrize("rows, groups, group", [(90, 16, 256), (200, 8, 512), (160, 8, 520), (1190, 1, 136), (2, 16, 256)])
@pytest.mark.parametrize("gate_type", [BF, torch.float32])
@pytest.mark.parametrize("gate_first", [True, False])
def test_gated_norm_of_many_groups(K, rows, groups, group, gate_type, gate_first):
    """On either side of the warp-a-pair kernel's line: enough pairs of up to 512 columns, wider groups, few pairs."""
    g = torch.Generator(device=DEV).manual_seed(rows + group)
    width = groups * group
    y, gate = torch.randn(rows, width, device=DEV, generator=g), torch.randn(rows, width + 8, device=DEV, generator=g).to(gate_type)[:, :width]
    w = (1 + 0.1 * torch.randn(group, device=DEV, generator=g)).to(BF)
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    seq[rows // 2] = -1
    out = torch.full((rows, width), 9.0, device=DEV, dtype=BF)
    s = torch.sigmoid(gate.double())
    if gate_type == torch.float32:
        if gate_first:
            return                                                     # (the delta mixer's form norms first)
        K.delta_gated_norm(y, gate, w, out, seq, group, 1e-6)
        gated = s
    else:
        K.gated_norm(y, gate, w, out, seq, group, gate_first, 1e-6)
        gated = s * gate.double()
    u = y.double() * gated if gate_first else y.double()
    u = u.view(rows, groups, group)
    want = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-6) * w.double()).view(rows, width)
    want = want if gate_first else want * gated
    live = seq >= 0
    # one rounding to bfloat16 and a few to float32
    assert ((out[live].double() - want[live]).abs() <= (2.0 ** -8 + 2.0 ** -18) * want[live].abs() + 1e-30).all()
    assert (out[~live] == 9.0).all()


@pytest.mark.parametrize("n", [1, 8, 4095, 4096, 100003])
@pytest.mark.parametrize("start", [0, 1, 4])
def test_cast(K, n, start):
    x = torch.randn(n + start, device=DEV)[start:]
    y = torch.full((n + 1,), 9.0, device=DEV, dtype=BF)
    K.cast(x, y[:n])
    assert torch.equal(y[:n], x.to(BF)) and y[n] == 9.0
    z = torch.full((n + 1,), 9.0, device=DEV)
    K.cast(y[:n], z[:n])
    assert torch.equal(z[:n], y[:n].float()) and z[n] == 9.0

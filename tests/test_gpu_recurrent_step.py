"""The kernels of one token a sequence (csrc/scan_step.cu, delta_step_kernel, causal_conv_step_kernel) beside float64: every decay, value
sizes of one CTA and of several, the norm in the same kernel and apart, sequences that sit the step out, rows with strides."""
import types

import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
LENS = [1, 0, 1, 1]


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def step():
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(n_seqs=len(LENS), max_q_len=1, q_start=i32([0, 1, 1, 2]), q_len=i32(LENS), slot_ids=i32([4, 1, 3, 0]),
                                 token_seq=i32([0, 2, 3, -1]), rows=4)


SLOTS = [4, 3, 0]           # of the rows


def norm64(o, z, w, eps, factor, act):
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps) * w
    return (o.flatten(1) * act(z)) * factor


def check(got, want, bits):
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -bits


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("mode", ["channel", "head", "constant"])
@pytest.mark.parametrize("heads, groups, dk, dv", [(3, 3, 128, 256), (4, 2, 64, 128), (2, 1, 128, 64), (2, 2, 64, 320)])
@pytest.mark.parametrize("with_norm", [False, True])
def test_linear_scan(K, dtype, mode, heads, groups, dk, dv, with_norm):
    if with_norm and dv not in K.STEP_NORM_COLS:
        return
    g = torch.Generator(device=DEV).manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(LENS)
    q, k, v, z = (rnd(rows, n + 8).to(dtype)[:, :n] for n in (groups * dk, groups * dk, heads * dv, heads * dv))
    gate = {"channel": rnd(rows, heads * dk + 4)[:, :heads * dk], "head": rnd(rows, heads + 1).to(dtype)[:, :heads], "constant": torch.rand(heads, device=DEV)}[mode]
    bias = rnd(heads * dk if mode == "channel" else heads).to(dtype)
    a_log, skip, w = rnd(heads).to(dtype), rnd(heads).to(dtype), rnd(dv).to(dtype)
    silu = mode == "constant"
    S0 = rnd(5, heads, dk, dv)
    offset = 32
    state = torch.zeros(5, offset + heads * dk * dv * 4, dtype=torch.uint8, device=DEV)
    state[:, offset:] = S0.reshape(5, -1).view(torch.uint8)
    out = torch.full((rows + 1, heads * dv), 7.0, device=DEV)
    y = torch.full((rows + 1, heads * dv), 7.0, device=DEV, dtype=dtype)
    before = K.launches
    K.linear_scan(q, k, v, gate, None if silu else bias, None if with_norm else out[:-1], state, offset, step(), heads, groups, dk, dv, mode,
                  q_scale=0.5, inv_tau=0.25, a_log=a_log if mode == "head" else None, skip=skip if mode == "head" else None, act_silu=silu,
                  norm=(z, w, y[:-1], 1e-5, 0.7) if with_norm else None)
    assert K.launches - before == 1 and (out[-1] == 7.0).all() and (y[-1] == 7.0).all()
    of = torch.arange(heads, device=DEV) // (heads // groups)
    f = (lambda x: torch.nn.functional.silu(x.double())) if silu else (lambda x: x.double())
    q64, k64, v64 = f(q).view(rows, groups, dk)[:, of], f(k).view(rows, groups, dk)[:, of], f(v).view(rows, heads, dv)
    if mode == "channel":
        a = torch.exp(torch.nn.functional.logsigmoid(gate.double() + bias.double()) * 0.25).view(rows, heads, dk, 1)
    elif mode == "head":
        dt = torch.nn.functional.softplus(gate.double() + bias.double(), threshold=50)
        a, k64 = torch.exp(-torch.exp(a_log.double()) * dt)[:, :, None, None], k64 * dt[:, :, None]
    else:
        a = gate.double()[None, :, None, None]
    S = a * S0[SLOTS].double() + k64[..., None] * v64[:, :, None]
    o = torch.einsum("rhkv,rhk->rhv", S, q64 * 0.5)
    if mode == "head":
        o = o + skip.double()[None, :, None] * v64
    got = state[:, offset:].contiguous().view(torch.float32).view(S0.shape)
    check(got[SLOTS], S, 20)
    assert torch.equal(got[[1, 2]], S0[[1, 2]]) and (state[:, :offset] == 0).all()
    if with_norm:
        check(y[:-1], norm64(o, z.double(), w.double(), 1e-5, 0.7, torch.nn.functional.silu), 8 if dtype == BF else 19)
    else:
        check(out[:-1], o.flatten(1), 20)


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("heads, groups, dk, dv", [(3, 3, 128, 256), (4, 2, 64, 128), (2, 1, 128, 64), (2, 2, 64, 192)])
@pytest.mark.parametrize("with_norm", [False, True])
def test_delta_rule(K, dtype, heads, groups, dk, dv, with_norm):
    if with_norm and dv not in K.STEP_NORM_COLS:
        return
    g = torch.Generator(device=DEV).manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(LENS)
    unit = lambda x: (x / x.norm(dim=-1, keepdim=True)).flatten(1)
    q, k, v = unit(rnd(rows, groups, dk)), unit(rnd(rows, groups, dk)), rnd(rows, heads * dv)
    both = rnd(rows, heads * (dk + dv))
    z, gate = both[:, :heads * dk], both[:, heads * dk:]
    bias, rate, b, w = rnd(heads * dk), torch.rand(heads, device=DEV), rnd(rows, heads + 1).to(dtype)[:, :heads], rnd(dv).to(dtype)
    S0 = rnd(5, heads, dk, dv)
    state = S0.reshape(5, -1).view(torch.uint8).clone()
    out = torch.full((rows + 1, heads * dv), 7.0, device=DEV)
    y = torch.full((rows + 1, heads * dv), 7.0, device=DEV, dtype=dtype)
    before = K.launches
    K.delta_rule(q, k, v, z, bias, rate, b, None if with_norm else out[:-1], state, 0, step(), heads, groups, dk, dv, False,
                 norm=(gate, w, y[:-1], 1e-5) if with_norm else None)
    assert K.launches - before == 1 and (out[-1] == 7.0).all() and (y[-1] == 7.0).all()
    of = torch.arange(heads, device=DEV) // (heads // groups)
    q64, k64, v64 = q.double().view(rows, groups, dk)[:, of], k.double().view(rows, groups, dk)[:, of], v.double().view(rows, heads, dv)
    a = torch.exp(-rate.double()[None, :, None] * torch.nn.functional.softplus((z + bias).double().view(rows, heads, dk), threshold=50))
    S = a[..., None] * S0[SLOTS].double()
    u = torch.sigmoid(b.double())[..., None] * (v64 - torch.einsum("rhkv,rhk->rhv", S, k64))
    S = S + k64[..., None] * u[:, :, None]
    o = torch.einsum("rhkv,rhk->rhv", S, q64)
    got = state.view(torch.float32).view(S0.shape)
    check(got[SLOTS], S, 20)
    assert torch.equal(got[[1, 2]], S0[[1, 2]])
    if with_norm:
        check(y[:-1], norm64(o, gate.double(), w.double(), 1e-5, 1.0, torch.sigmoid), 8 if dtype == BF else 19)
    else:
        check(out[:-1], o.flatten(1), 19)


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels, silu", [(16, False), (520, True), (1032, True)])
def test_convolution(K, dtype, taps, channels, silu):
    g = torch.Generator(device=DEV).manual_seed(channels + taps)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(LENS)
    x, w, b = rnd(rows, channels + 8).to(dtype)[:, :channels], rnd(channels, taps).to(dtype), rnd(channels).to(dtype)
    S0 = rnd(5, taps - 1, channels)
    state = S0.reshape(5, -1).view(torch.uint8).clone()
    y = torch.full((rows + 1, channels), 7.0, device=DEV, dtype=dtype)
    before = K.launches
    K.causal_conv(x, y[:-1], w, b, state, 0, step(), silu=silu)
    assert K.launches - before == 1 and (y[-1] == 7.0).all()
    inputs = torch.cat([S0[SLOTS].double(), x.double()[:, None]], 1)
    want = b.double() + (inputs * w.double().T[None]).sum(1)
    check(y[:-1], torch.nn.functional.silu(want) if silu else want, 8 if dtype == BF else 20)
    got = state.view(torch.float32).view(S0.shape)
    assert torch.equal(got[SLOTS], inputs[:, 1:].float()) and torch.equal(got[[1, 2]], S0[[1, 2]])


@pytest.mark.parametrize("what", ["channel", "head", "constant", "chunks of one decay a head", "delta", "delta, walked", "convolution"])
def test_two_calls_on_one_state_with_nothing_between(K, what):
    """The second call starts from what the first one leaves, whether or not the host waits between them."""
    g = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    heads, dk, dv, n = 16, 128, 128, 8
    chunks = what.startswith("chunks")
    each = 20 if chunks else 1
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(n_seqs=n, max_q_len=each, q_start=i32([each * i for i in range(n)]), q_len=i32([each] * n), slot_ids=i32(list(range(n))),
                                token_seq=i32([i // each for i in range(n * each)]), rows=n * each)
    rows = n * each
    q, k, v = (rnd(rows, heads * dk).to(BF) * 0.1 for _ in range(3))
    z, bias, a_log, b = rnd(rows, heads * dk), rnd(heads * dk).to(BF), rnd(heads).to(BF), rnd(rows, heads).to(BF)
    unit = lambda x: (x.float().view(rows, heads, dk) / x.float().view(rows, heads, dk).norm(dim=-1, keepdim=True)).flatten(1)
    qu, ku, vf, taps = unit(q), unit(k), v.float(), rnd(heads * dk, 4).to(BF)
    out, y = torch.empty(rows, heads * dv, device=DEV), torch.empty(rows, heads * dk, device=DEV, dtype=BF)
    per = heads * dk * dv * 4 if what != "convolution" else 3 * heads * dk * 4

    def call(state):
        if what == "channel":
            K.linear_scan(q, k, v, z, bias, out, state, 0, ctx, heads, heads, dk, dv, "channel")
        elif what == "constant":
            K.linear_scan(q, k, v, decay, None, out, state, 0, ctx, heads, heads, dk, dv, "constant")
        elif what == "head" or chunks:
            K.linear_scan(q, k, v, b, a_log, out, state, 0, ctx, heads, heads, dk, dv, "head", a_log=a_log)
        elif what == "convolution":
            K.causal_conv(q, y, taps, None, state, 0, ctx)
        else:
            K.delta_rule(qu, ku, vf, z, zb, rate, b, out, state, 0, ctx, heads, heads, dk, dv if what == "delta" else 112, False)

    decay, zb, rate = torch.full((heads,), 0.9, device=DEV), bias.float(), torch.full((heads,), 0.5, device=DEV)
    if what == "delta, walked":
        vf, out = vf[:, :heads * 112], torch.empty(rows, heads * 112, device=DEV)
        per = heads * dk * 112 * 4
    start = rnd(n, per // 4).view(torch.uint8)
    want = start.clone()
    for _ in range(4):
        call(want)
        torch.cuda.synchronize()
    want_out = out.clone()
    for _ in range(5):
        got = start.clone()
        for _ in range(4):
            call(got)
        assert torch.equal(got, want) and torch.equal(out, want_out)


def test_the_engine_says_that_its_steps_are_settled(K, monkeypatch):
    from braidinfer_b200.engine.engine import Engine
    from loduzen_tiny import LZ_CONFIGS
    seen = []
    e = Engine.from_random(LZ_CONFIGS["A"], max_tokens=256, verbose=False)
    forward = e.model.forward
    monkeypatch.setattr(e.model, "forward", lambda ctx, *a, **kw: seen.append(ctx.settled) or forward(ctx, *a, **kw))
    s = e.open()
    e.step([(s, [1, 2, 3])])
    e.step([(s, [4])])
    e.step([(s, [4])])
    assert seen == [True] * len(seen) and len(seen) >= 2

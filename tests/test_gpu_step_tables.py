"""A step's tables fetched by a kernel from pinned buffers used in turn, and the convolution's rows whose taps all lie in the step."""
import types

import pytest
import torch

from braidinfer_b200.config import preset
from braidinfer_b200.csrc.api import KernelError, get_kernels
from braidinfer_b200.engine import Engine

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


@pytest.mark.parametrize("n", [4, 508, 512, 516, 4096])
def test_fetch(K, n):
    host = torch.empty(n, dtype=torch.int32, pin_memory=True)
    dst = torch.full((n + 4,), -1, dtype=torch.int32, device=DEV)
    for turn in range(3):                                              # the same place again: never an old line
        host.copy_(torch.arange(n, dtype=torch.int32) * (turn + 1))
        K.fetch_i32(host, dst[:n])
        torch.cuda.synchronize()
        assert torch.equal(dst[:n].cpu(), host) and (dst[n:] == -1).all()
    with pytest.raises(KernelError):
        K.fetch_i32(host[:2], dst[:2])
    with pytest.raises(KernelError):
        K.fetch_i32(torch.zeros(4, dtype=torch.int32), dst[:4])


def test_steps_that_the_host_runs_ahead_of():
    """Replayed steps whose tables lie in four buffers in turn, launched without a look at the device, beside steps without graphs."""
    res = []
    for graphs in (True, False):
        eng = Engine.from_random(preset("tiny_b"), 5, max_tokens=1024, max_slots=3, use_graphs=graphs, verbose=False)
        slots = [eng.open() for _ in range(3)]
        eng.step([(s, [1 + s, 7, 9]) for s in slots])
        out = [eng.step([(s, [(13 * t + 5 * s) % 384]) for s in slots]) for t in range(40)]
        eng.check()
        res.append(torch.cat(out))
    assert torch.equal(*res)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lens", [[1], [3, 4, 5], [30, 1, 2, 9], [7, 64]])
@pytest.mark.parametrize("taps, silu, bias", [(4, True, True), (2, False, True), (3, True, False), (4, False, False)])
def test_convolution(K, dtype, lens, taps, silu, bias):
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + taps)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows, ch = sum(lens), 72
    x, w, b = rnd(rows, ch + 8).to(dtype)[:, :ch], rnd(ch, taps).to(dtype), rnd(ch).to(dtype) if bias else None
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    start = [sum(lens[:i]) for i in range(len(lens))]
    seq = i32([i for i, n in enumerate(lens) for _ in range(n)] + [-1, -1])
    before = rnd(len(lens), taps - 1, ch)
    state = before.clone().view(len(lens), -1).view(torch.uint8)
    ctx = types.SimpleNamespace(n_seqs=len(lens), token_seq=seq, q_start=i32(start), q_len=i32(lens), slot_ids=i32(list(range(len(lens)))))
    xp = torch.cat([x, x[:2]])                                         # two rows of padding
    y = torch.full((rows + 2, ch), 9.0, device=DEV, dtype=dtype)
    K.causal_conv(xp, y, w, b, state, 0, ctx, silu=silu)
    for i, n in enumerate(lens):
        full = torch.cat([before[i].double(), x[start[i]:start[i] + n].double()])
        terms = [full[j:j + n] * w[:, j].double() for j in range(taps)]
        want, size = sum(terms), sum(t.abs() for t in terms)
        if bias:
            want, size = want + b.double(), size + b.double().abs()
        slack = (taps + 2) * 2.0 ** -23 * size
        if silu:
            want, slack = want * torch.sigmoid(want), 1.1 * slack + 2.0 ** -20 * want.abs()
        step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
        assert ((y[start[i]:start[i] + n].double() - want).abs() <= step * want.abs() + 1.01 * slack + 1e-30).all()
        assert torch.equal(state.view(torch.float32).view(before.shape)[i], full[n:].float())
    assert (y[rows:] == 9.0).all()


@pytest.mark.parametrize("lens", [[600], [2, 3, 1, 3]])
def test_activation_of_the_convolution_is_float32(K, lens):
    """One tap alone, so that the sum is one product rounded to float32: the result is its silu rounded once to bfloat16 after float32
    errors of a few units (an exponential good to two, a division, the product), down to silu's smallest normal numbers."""
    gates = torch.cat([torch.linspace(-88.0, -60.0, 64), torch.linspace(-60.0, 8.0, 192)]).to(torch.bfloat16).to(DEV)
    rows, ch, taps = sum(lens), gates.numel(), 4
    x = torch.linspace(1.0, 2.0, rows + 1)[:rows].to(torch.bfloat16).to(DEV)[:, None].repeat(1, ch)
    w = torch.zeros(ch, taps, device=DEV, dtype=torch.bfloat16)
    w[:, taps - 1] = gates
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    state = torch.zeros(len(lens), (taps - 1) * ch * 4, dtype=torch.uint8, device=DEV)
    ctx = types.SimpleNamespace(n_seqs=len(lens), token_seq=i32([i for i, n in enumerate(lens) for _ in range(n)]), q_len=i32(lens),
                                q_start=i32([sum(lens[:i]) for i in range(len(lens))]), slot_ids=i32(list(range(len(lens)))))
    y = torch.empty_like(x)
    K.causal_conv(x, y, w, None, state, 0, ctx, silu=True)
    z = (x.double() * gates.double()).float().double()
    want = z * torch.sigmoid(z)
    half_step = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -126))) - 8)
    assert ((y.double() - want).abs() <= half_step + 8 * 2.0 ** -24 * want.abs()).all()

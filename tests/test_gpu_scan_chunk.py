"""The recurrences with a decay a key channel and with a constant one a head over chunks on the tensor cores (csrc/scan_chunk.cu) beside
float64 and beside the walk token by token: sequences at a chunk's edges, portions that continue from a stored state, steep decays,
numbers that are not finite."""
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


def run(K, t, mode, lens, chunk, groups, dk, dv, silu=False, offset=16):
    """(out, states after): the step in two portions where it is long; rows of `out` past the step's stay as they were."""
    heads = t["S"].shape[1]
    slots = list(range(1, len(lens) + 1))
    state = torch.zeros(len(lens) + 2, offset + heads * dk * dv * 4, dtype=torch.uint8, device=DEV)
    state[:, offset:] = t["S"].reshape(len(lens) + 2, -1).view(torch.uint8)
    out = torch.full((sum(lens), heads * dv), 7.0, device=DEV)
    cuts = [[n - n // 3 for n in lens], [n // 3 for n in lens]] if max(lens) > 400 else [lens]
    done, start = [0] * len(lens), [sum(lens[:i]) for i in range(len(lens))]
    for cut in cuts:
        whole = len(cuts) == 1                                          # (views, with their strides)
        pick = slice(None) if whole else torch.cat([torch.arange(start[i] + done[i], start[i] + done[i] + cut[i]) for i in range(len(lens))]).to(DEV)
        o = torch.full((sum(cut) + 1, heads * dv), 7.0, device=DEV)
        gate = t["decay"] if mode == "constant" else t["z"][pick]
        K.linear_scan(t["q"][pick], t["k"][pick], t["v"][pick], gate, None if mode == "constant" else t["bias"], o[:-1], state, offset,
                      step(cut, slots), heads, groups, dk, dv, mode, q_scale=0.3, inv_tau=0.25, act_silu=silu, chunk=chunk)
        assert (o[-1] == 7.0).all()
        out[pick] = o[:-1]
        done = [a + b for a, b in zip(done, cut)]
    assert (state[:, :offset] == 0).all()
    got = state[:, offset:].contiguous().view(torch.float32).view(t["S"].shape)
    assert torch.equal(got[0], t["S"][0]) and torch.equal(got[-1], t["S"][-1])
    return out, got


def drawn(heads, groups, dk, dv, lens, logit, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(lens)
    decay = 1.0 - 2.0 ** -(1.0 + 2.0 * torch.arange(heads, device=DEV, dtype=torch.float32))
    decay[-1] = 0.02                                                    # 2^-90 over a sub-chunk
    return {"q": rnd(rows, groups * dk + 3).to(BF)[:, 3:], "k": rnd(rows, groups * dk).to(BF), "v": rnd(rows, heads * dv + 8).to(BF)[:, 8:],
            "z": (rnd(rows, heads * dk + 4) * 3 + logit)[:, :heads * dk], "bias": rnd(heads * dk).to(BF), "decay": decay,
            "S": rnd(len(lens) + 2, heads, dk, dv)}


# logits: decays near one; from near one to 2^-8 a token within a head; all channels steep
@pytest.mark.parametrize("mode, logit, silu", [("channel", 9.0, False), ("channel", -4.0, False), ("channel", -40.0, False),
                                               ("constant", 0.0, True), ("constant", 0.0, False)])
@pytest.mark.parametrize("heads, groups, dk, dv", [(3, 3, 128, 256), (4, 2, 128, 64), (2, 1, 64, 128), (2, 2, 64, 192)])
@pytest.mark.parametrize("lens", [[128], [129, 1, 64], [65, 63, 191], [530, 0, 2]])
def test_chunks(K, mode, logit, silu, heads, groups, dk, dv, lens):
    t = drawn(heads, groups, dk, dv, lens, logit, sum(lens) + dk)
    before = K.launches
    res = {c: run(K, t, mode, lens, c, groups, dk, dv, silu) for c in (None, 0)}
    assert K.launches - before in (4, 8)                                # three kernels a portion, and one of the walk
    f = (lambda x: torch.nn.functional.silu(x.double())) if silu else (lambda x: x.double())
    of = torch.arange(heads, device=DEV) // (heads // groups)
    errors = {None: [], 0: []}
    for i, n in enumerate(lens):
        S, at = t["S"][i + 1].double(), sum(lens[:i])
        want = torch.empty(n, heads, dv, dtype=torch.float64, device=DEV)
        for r in range(at, at + n):
            a = t["decay"].double()[:, None, None] if mode == "constant" else \
                torch.exp(torch.nn.functional.logsigmoid(t["z"][r].double() + t["bias"].double()) * 0.25).view(heads, dk, 1)
            S = a * S + f(t["k"][r]).view(groups, dk)[of][:, :, None] * f(t["v"][r]).view(heads, 1, dv)
            want[r - at] = torch.einsum("hkv,hk->hv", S, f(t["q"][r]).view(groups, dk)[of] * 0.3)
        rel = lambda x, y: float((x.double() - y).norm() / y.norm())
        for c, (out, state) in res.items():
            errors[c].append(max(rel(out[at:at + n].view(n, heads, dv), want) if n else 0.0, rel(state[i + 1], S)))
    # sums of float32 numbers in another order: as far from float64 as the walk is
    assert max(errors[None]) < 1.5 * max(errors[0]) + 2.0 ** -22 and max(errors[None]) < 2.0 ** -19


@pytest.mark.parametrize("mode, silu", [("channel", False), ("constant", True)])
@pytest.mark.parametrize("what", ["q", "k", "v", "z", "S"])
@pytest.mark.parametrize("at", [3, 70, 128])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan"), 3e38])
def test_numbers_that_are_not_finite(K, mode, silu, what, at, bad):
    """They do what they do in the walk, and never reach the tokens before them."""
    if what == "z" and (mode == "constant" or bad == 3e38):
        return
    lens, heads, dk, dv = [150], 2, 128, 128
    t = drawn(heads, 1, dk, dv, lens, 6.0, 5)
    t["decay"][:] = 0.9
    if bad == 3e38:                                                     # past the largest part of a split: what it meets is small, the results fit
        for other in {"q": "kS", "k": "v", "v": "k", "S": ""}[what]:
            t[other] = t[other] * 2.0 ** -9
    clean = run(K, t, mode, lens, None, 1, dk, dv, silu)[0]
    t[what] = t[what].clone()
    if what == "S":
        t["S"][1, 1, 5, 9] = bad
        t["q"] = t["q"] * 2.0 ** -9
    else:
        t[what][at, 1] = bad
    got, walk = (run(K, t, mode, lens, c, 1, dk, dv, silu)[0] for c in (None, 0))
    close = lambda x, y: float((x.double() - y.double()).norm() / y.double().norm()) < 2.0 ** -18
    if what != "S":
        assert close(got[:at], clean[:at])
    if bad == 3e38:
        assert torch.isfinite(walk).all()
    if not (what == "z" and bad < 0):
        assert torch.equal(torch.isfinite(got), torch.isfinite(walk))
        ok = torch.isfinite(walk)
        assert close(got[ok], walk[ok])


# decays of some 2^-6 a token: a sub-chunk's products lie on both sides of what its factors are split for
@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("what", ["q", "k", "v", "qk"])
@pytest.mark.parametrize("size", [0, -20, -40, -60, 30, 60])
def test_small_and_large_numbers_behind_steep_decays(K, dk, what, size):
    lens, heads, dv = [150, 129], 2, 64
    t = drawn(heads, heads, dk, dv, lens, -16.0, dk)
    for n in what:
        t[n] = t[n] * 2.0 ** size
    if "q" not in what:
        t["S"] = t["S"] * 2.0 ** size
    want = torch.empty(sum(lens), heads * dv, dtype=torch.float64, device=DEV)
    for i, n in enumerate(lens):
        S, at = t["S"][i + 1].double(), sum(lens[:i])
        for r in range(at, at + n):
            a = torch.exp(torch.nn.functional.logsigmoid(t["z"][r].double() + t["bias"].double()) * 0.25).view(heads, dk, 1)
            S = a * S + t["k"][r].double().view(heads, dk, 1) * t["v"][r].double().view(heads, 1, dv)
            want[r] = torch.einsum("hkv,hk->hv", S, t["q"][r].double().view(heads, dk) * 0.3).flatten()
    # token by token beside the size of a token's results: sums of float32 numbers in another order than the walk's
    rel = lambda x: float((x.double() - want).norm(dim=1).max() / want.pow(2).sum(1).mean().sqrt())
    chunks, walk = (rel(run(K, t, "channel", lens, c, heads, dk, dv)[0]) for c in (None, 0))
    # (2^60 is walked in the kernel, one chain of dk sums a column: a rounding of 2^-24 each, 2^-20.5 for 128 of them at random)
    assert chunks < (1.5 * walk + 2.0 ** -22 if size < 60 else 2.0 ** -20), (chunks, walk)

"""The delta rule over chunks on the tensor cores (csrc/delta_chunk.cu): numbers that are not finite, and small ones."""
import types

import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
H, DK, DV = 2, 128, 128
LENS = [150, 100]


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def drawn(dk=DK, logit=-4.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rows = sum(LENS)
    unit = lambda: (lambda x: (x / x.norm(dim=-1, keepdim=True)).flatten(1))(rnd(rows, H, dk))
    return {"q": unit(), "k": unit(), "v": rnd(rows, H * DV), "z": rnd(rows, H * dk) + logit, "b": rnd(rows, H), "S": rnd(len(LENS), H, dk, DV)}


def run(K, t, chunked, dk=DK):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(n_seqs=len(LENS), max_q_len=max(LENS), q_start=i32([0, LENS[0]]), q_len=i32(LENS), slot_ids=i32([0, 1]))
    state = t["S"].reshape(len(LENS), -1).clone().view(torch.uint8)
    out = torch.empty(sum(LENS), H * DV, device=DEV)
    K.delta_rule(t["q"], t["k"], t["v"], t["z"], torch.zeros(H * dk, device=DEV), torch.ones(H, device=DEV), t["b"], out, state, 0, ctx, H, H,
                 dk, DV, chunked)
    K.check_device_errors()
    return out.view(-1, H, DV), state.view(torch.float32).view(t["S"].shape)


@pytest.mark.parametrize("what", ["q", "k", "v", "z", "b", "S"])
@pytest.mark.parametrize("at", [3, 70, 128, 149])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_numbers_that_are_not_finite(K, what, at, bad):
    """Head 0 of the first sequence holds one.  The other head, the other sequence and the tokens of earlier blocks of 16 keep their bits;
    inside its own block it may reach back (zero times an infinity), from its token on it does what it does in the walk."""
    t = drawn()
    clean, states = run(K, t, True)
    if what == "S":
        t["S"][0, 0, 5, 9] = bad
    else:
        t[what][at, 0] = bad
    (got, S), (walk, _) = run(K, t, True), run(K, t, False)
    first = 0 if what == "S" else at // 16 * 16
    assert torch.equal(got[:, 1], clean[:, 1]) and torch.equal(got[LENS[0]:], clean[LENS[0]:]) and torch.equal(got[:first, 0], clean[:first, 0])
    assert torch.equal(S[1], states[1]) and torch.equal(S[0, 1], states[0, 1])
    since = slice(0 if what == "S" else at, LENS[0])
    assert torch.equal(torch.isfinite(got[since, 0]), torch.isfinite(walk[since, 0]))


# decays of some 2^-6 a token: a sub-chunk's products lie on both sides of what its factors are split for
@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("size", [0, -20, -40, -60])
def test_small_queries_behind_steep_decays(K, dk, size):
    t = drawn(dk, logit=4.1, seed=dk)
    t["q"] *= 2.0 ** size
    d = lambda n, w: t[n].double().view(-1, H, w)
    decay, beta = torch.exp(-torch.nn.functional.softplus(d("z", dk), threshold=50)), torch.sigmoid(t["b"].double())
    want, at = torch.empty(sum(LENS), H, DV, dtype=torch.float64, device=DEV), 0
    for i, n in enumerate(LENS):
        S = t["S"][i].double()
        for r in range(at, at + n):
            S = decay[r][:, :, None] * S
            u = beta[r][:, None] * (d("v", DV)[r] - torch.einsum("hkv,hk->hv", S, d("k", dk)[r]))
            S = S + d("k", dk)[r][:, :, None] * u[:, None]
            want[r] = torch.einsum("hkv,hk->hv", S, d("q", dk)[r])
        at += n
    rel = lambda x: float((x.double() - want).norm() / want.norm())
    chunks, walk = (rel(run(K, t, c, dk)[0]) for c in (True, False))
    assert chunks < 1.5 * walk + 2.0 ** -22, (chunks, walk)

"""The experts' products of steps of few tokens (csrc/moe_few.cu): every number of tokens, widths that fill no tile, k that fills no
turn of the warps or several, more units than CTAs, rows of no sequence, an expert nobody chose."""
import pytest
import torch

from braidinfer_b200.csrc.api import KernelError, MOE_TC_TILE, get_kernels, interleave_experts

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -23               # a float32 sum that the tensor cores cut off instead of rounding it: a whole step


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


@pytest.mark.parametrize("rows", [1, 2, 5, 8])
@pytest.mark.parametrize("experts, top, j, k", [(2, 1, 8, 8), (5, 2, 24, 40), (9, 3, 264, 200), (70, 8, 520, 1160), (4, 4, 1032, 2056)])
@pytest.mark.parametrize("mode", ["plain", "gated", "gated, weight on the input", "relu2"])
@pytest.mark.parametrize("of_slots", [False, True])
def test_products(K, rows, experts, top, j, k, mode, of_slots):
    g = torch.Generator(device=DEV).manual_seed(j + k + rows)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    idx = torch.stack([torch.randperm(experts, device=DEV, generator=g)[:top] for _ in range(rows)]).to(torch.int32)
    if rows > 1:
        idx[-1, -1] = -1                                             # fewer allowed experts than choices
    seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    if rows > 4:
        seq[1] = -1                                                  # a padding row
    plan = K.moe_plan(idx, seq, experts, MOE_TC_TILE)
    slot_pair = plan[0].long()
    live = slot_pair >= 0
    x = rnd(rows, k + 8).to(torch.bfloat16)[:, :k]                   # rows further apart than they are long
    w0, w1 = [(rnd(experts, j, k) * k ** -0.5).to(torch.bfloat16) for _ in range(2)]
    wgt = torch.rand(rows, top, device=DEV, generator=g)
    xs = torch.full((slot_pair.numel(), k), float("nan"), device=DEV, dtype=torch.bfloat16)      # padding slots are not read
    xs[live] = x[slot_pair[live] // top]
    gated = mode.startswith("gated")
    in_wgt = wgt if "weight" in mode else None
    out = torch.full((slot_pair.numel(), j + 8), 3.0, device=DEV, dtype=torch.bfloat16)
    K.moe_few(xs if of_slots else x, interleave_experts(w0, w1) if gated else w0, out[:, :j], plan, rows, 0 if of_slots else top,
              gated=gated, relu2=mode == "relu2", in_wgt=in_wgt)
    K.check_device_errors()
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
    assert ((out[live, :j].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -14) * want.abs() + 1.01 * slack + 1e-30).all()
    assert (out[~live] == 3.0).all() and (out[:, j:] == 3.0).all()


def test_more_tokens_are_refused(K):
    idx = torch.zeros((9, 1), dtype=torch.int32, device=DEV)
    plan = K.moe_plan(idx, torch.zeros(9, dtype=torch.int32, device=DEV), 2, MOE_TC_TILE)
    x, w = torch.zeros((9, 8), device=DEV, dtype=torch.bfloat16), torch.zeros((2, 8, 8), device=DEV, dtype=torch.bfloat16)
    with pytest.raises(KernelError):
        K.moe_few(x, w, torch.zeros((plan[4] * MOE_TC_TILE, 8), device=DEV, dtype=torch.bfloat16), plan, 9, 1)

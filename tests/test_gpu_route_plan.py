"""Routing and plan of few tokens in one kernel (csrc/moe.cu, moe_route_plan_kernel) against the two kernels of any number of tokens:
the same choices and the same bits of the weights, and a plan that says the same."""
import pytest
import torch

from braidinfer_b200.csrc.api import KernelError, MOE_TC_TILE, get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def both(K, z, seq, top, groups, keep, **how):
    rows, experts = z.shape
    out = []
    for one in (False, True):
        idx = torch.full((rows, top), -7, dtype=torch.int32, device=DEV)
        wgt = torch.full((rows, top), -7.0, device=DEV)
        if one:
            plan = K.moe_route_plan(z, seq, idx, wgt, groups, keep, **how)
        else:
            K.moe_route(z, idx, wgt, groups, keep, **how)
            plan = K.moe_plan(idx, seq, experts, MOE_TC_TILE)
        K.check_device_errors()
        out.append((idx, wgt, plan))
    (idx, wgt, plan), (idx1, wgt1, plan1) = out
    assert torch.equal(idx, idx1) and torch.equal(wgt.view(torch.int32), wgt1.view(torch.int32))
    n, runs = int(plan[3][0]), int(plan[3][1])
    assert plan[4] == plan1[4] and torch.equal(plan[3][:2], plan1[3][:2]) and torch.equal(plan[2][:n], plan1[2][:n])
    assert torch.equal(plan[5].view(-1, 4)[:runs], plan1[5].view(-1, 4)[:runs])
    assert torch.equal(plan[1] // MOE_TC_TILE, plan1[1] // MOE_TC_TILE)              # a pair's tile (the slot in it is anyone's)
    placed = (plan1[1] >= 0).nonzero().flatten()
    assert torch.equal(plan1[0][plan1[1][placed].long()].long(), placed) and int((plan1[0] >= 0).sum()) == placed.numel()
    for t in range(n):                                                              # a tile's pairs lie at its front
        used = (plan1[0][t * MOE_TC_TILE:(t + 1) * MOE_TC_TILE] >= 0)
        assert used[:int(used.sum())].all()
    return idx


SHAPES = [(1, 1, 1, 1), (4, 1, 1, 1), (6, 3, 2, 2), (8, 2, 1, 4), (33, 1, 1, 5), (64, 8, 4, 6), (64, 1, 1, 6), (65, 5, 5, 3), (96, 32, 7, 8),
          (256, 1, 1, 32), (256, 16, 3, 8)]


@pytest.mark.parametrize("rows", [1, 3, 8])
@pytest.mark.parametrize("experts, groups, keep, top", SHAPES)
@pytest.mark.parametrize("sigmoid", [False, True])
def test_the_same_as_two_kernels(K, rows, experts, groups, keep, top, sigmoid):
    g = torch.Generator(device=DEV).manual_seed(experts + rows)
    z = torch.randn(rows, experts, device=DEV, generator=g) * 2
    seq = torch.arange(rows, dtype=torch.int32, device=DEV)
    seq[rows // 2] = -1 if rows > 1 else 0                                          # a padding row
    both(K, z, seq, top, groups, keep, mult=0.7, sigmoid=sigmoid)
    both(K, z, seq, top, groups, keep, mult=0.7, sigmoid=sigmoid, renorm=sigmoid)
    if groups == 1:
        corr = torch.randn(experts, device=DEV, generator=g)
        both(K, z, seq, top, groups, keep, sigmoid=sigmoid, correction=corr)
        corr[::2] = float("-inf")                                                   # fewer experts that can be chosen
        both(K, z, seq, top, groups, keep, sigmoid=sigmoid, correction=corr)


@pytest.mark.parametrize("experts, groups, keep, top", SHAPES)
def test_equal_scores_and_numbers_that_are_none(K, experts, groups, keep, top):
    seq = torch.zeros(5, dtype=torch.int32, device=DEV)
    z = torch.zeros(5, experts, device=DEV)
    z[1, 0] = float("nan")
    z[2] = float("nan")
    z[3] = float("-inf")
    z[4, experts // 2] = float("inf")
    idx = both(K, z, seq, top, groups, keep)
    if keep == groups:
        assert idx[0].tolist() == list(range(top))                                  # all equal: the lowest indices
    both(K, z, seq, top, groups, keep, sigmoid=True)


def test_more_than_a_cta_takes_is_refused(K):
    for rows, experts, top in ((9, 8, 1), (8, 257, 1), (1, 64, 33)):
        assert not K.moe_route_plan_fits(rows, experts, top, 1, MOE_TC_TILE)
        with pytest.raises(KernelError):
            K.moe_route_plan(torch.zeros(rows, experts, device=DEV), torch.zeros(rows, dtype=torch.int32, device=DEV),
                             torch.zeros((rows, top), dtype=torch.int32, device=DEV), torch.zeros((rows, top), device=DEV), 1, 1)

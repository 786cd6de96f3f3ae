"""The cases of perf/cases.py at small sizes: what a pass returns beside its own 64-bit results, model by model, so that neither the
equations there nor the bounds that it states drift from the library unnoticed."""
import random

import pytest
import torch

from perf import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["dense", "bidinex", "loduzen", "zisesun", "megerax"])
@pytest.mark.parametrize("seqs, longest, steps", [(2, 37, 3), (1, 90, 0)])
def test_a_float32_pass(model, seqs, longest, steps):
    case = C._turn(model, "w1024", seqs, longest, steps, "float32")
    out, want, bound = C.run(C.prepare(case, 5)), C.exact(case, 5), C.tolerance(case)
    assert len(out) == len(want) == 1 + (steps > 0)
    for a, b in zip(out, want):
        assert a.shape == b.shape and a.dtype == torch.float32
        # what is stated of two correct float32 runs holds beside 64 bits all the more
        assert float((a.double() - b).norm() / b.norm()) < bound["rel"]


@pytest.mark.parametrize("model", ["dense", "bidinex", "loduzen", "zisesun", "megerax"])
def test_a_bfloat16_pass(model):
    """Most rows lie within what bfloat16 between the kernels of four layers gives (0.002 to 0.015 of a row's norm); a router's near-tie
    that falls the other way moves single rows further."""
    case = C._turn(model, "w1024", 3, 60, 4)
    out, want = C.run(C.prepare(case, 6)), C.exact(case, 6)
    err = torch.cat([(a.double() - b).norm(dim=1) / b.norm(dim=1) for a, b in zip(out, want)])
    assert float(err.median()) < C.tolerance(case)["rel"]


def test_drawn_cases_stay_within_the_largest_listed_one():
    rng, most = random.Random(3), max(C.work(c)["bytes"] for c in C.listed())
    for _ in range(40):
        case = C.draw(rng)
        w = C.work(case)
        assert 0 < w["bytes"] <= 1.5 * most and w["flops"] >= 0

"""Dynamic Tanh at the edges of its CTAs and on rows that do not start on 16 bytes (csrc/pointwise.cu)."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("width", [1, 3, 4, 127, 508, 512, 516, 2049, 4096])
@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_every_number_of_a_row(width, skip, dtype):
    K = get_kernels(verbose=False)
    g = torch.Generator(device=DEV).manual_seed(width)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(5 * width + skip)[skip:].view(5, width) * 2               # one number on: rows off 16 bytes
    w, b, a = rnd(width).to(dtype), rnd(width).to(dtype), torch.tensor([0.7], device=DEV).to(dtype)
    idx = torch.tensor([4, -1, 0, 0, 2, 3], dtype=torch.int32, device=DEV)
    out = torch.full((6 * width + 8,), 7.0, device=DEV, dtype=dtype)
    K.dyt(x, w, b, a, out[:6 * width].view(6, width), row_index=idx, in_scale=1.5)
    got = out[:6 * width].view(6, width).double()
    xs = x[idx.clamp_min(0).long()].double() * 1.5
    want = torch.tanh(a.double() * xs) * w.double() + b.double()
    want[1] = 0
    # tanhf is off by 2 steps at most, its argument by two roundings (tanh falls behind x: no more than their relative error)
    slack = 8 * 2.0 ** -24 * (w.double().abs() + b.double().abs()) + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24) * want.abs()
    assert ((got - want).abs() <= slack).all() and (out[6 * width:] == 7.0).all()

"""The per-head product of up to 16 tokens (gemm_heads_few_kernel, csrc/latent.cu): token blocks, outputs that fill no tile, k of less
than one turn of the warps up to several."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("heads, k, j", [(1, 8, 1), (3, 24, 37), (2, 128, 512), (5, 136, 16), (16, 512, 128), (2, 1032, 33)])
@pytest.mark.parametrize("gated", [False, True])
def test_against_64_bits(rows, heads, k, j, gated):
    K = get_kernels(verbose=False)
    g = torch.Generator(device=DEV).manual_seed(rows + k)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16)
    x = rnd(rows, heads * (k + 8)).view(rows, heads, k + 8)[:, :, :k]
    w, gate = rnd(heads, j, k), rnd(rows, heads)
    out = torch.full((rows, heads, j + 2), 7.0, device=DEV, dtype=torch.bfloat16)
    K.gemm_heads(x, w, out[:, :, :j], gate=gate if gated else None, mult=0.7)
    K.check_device_errors()
    f = 0.7 * torch.sigmoid(gate.double())[:, :, None] if gated else 1.0
    want = torch.einsum("nhk,hjk->nhj", x.double(), w.double()) * f
    size = torch.einsum("nhk,hjk->nhj", x.double().abs(), w.double().abs()) * f
    # float32 sums in any order whose adds may cut off (a step of 2^-23 each), the gate's few steps, one rounding to bfloat16
    assert ((out[:, :, :j].double() - want).abs() <= (k + 8) * 2.0 ** -23 * size + 2.0 ** -8 * want.abs()).all()
    assert (out[:, :, j:] == 7.0).all()

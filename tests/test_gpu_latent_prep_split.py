"""The rows' preparation of latent attention with the rotation in CTAs of its own (up to 64 rows, csrc/latent.cu): a step of 65 rows, one CTA a
row, gives the numbers of its rows by themselves, for pairs that fill one CTA, several, more than there are, and none."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads, dim, rot, rank, rot_dims", [(1, 8, 8, 8, 8), (16, 128, 64, 512, 64), (3, 20, 12, 36, 8), (128, 16, 64, 64, 48), (2, 16, 0, 32, 0)])
@pytest.mark.parametrize("adjacent", [False, True])
def test_rows_by_themselves(dtype, heads, dim, rot, rank, rot_dims, adjacent):
    K = get_kernels(verbose=False)
    g = torch.Generator(device=DEV).manual_seed(heads + rank)
    rows, ps = 65, 64
    cols = heads * (dim + rot)
    proj = torch.randn(rows, cols + rank + rot, device=DEV, generator=g).to(dtype)
    norm_w = torch.rand(rank, device=DEV, generator=g).to(dtype)
    inv_freq = torch.rand(max(rot_dims // 2, 1), device=DEV, generator=g)
    positions = torch.arange(rows, dtype=torch.int32, device=DEV) * 2 + 1
    token_seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
    token_seq[7] = -1
    table = torch.tensor([[2, 0, 1]], dtype=torch.int32, device=DEV)
    out = []
    for n in (rows, 13):
        cache = torch.zeros(3, 1, 1, ps, rank + rot, device=DEV, dtype=dtype)
        q_lat = torch.zeros(rows, heads, rank + rot, device=DEV, dtype=dtype)
        for r in range(0, rows, n):
            s = slice(r, min(r + n, rows))
            K.latent_prep(proj[s], cols, norm_w, inv_freq, positions[s], token_seq[s], table, cache, q_lat[s], heads, dim, rot, rank,
                          rot_dims, ps, 1e-6, adjacent=adjacent)
        K.check_device_errors()
        out.append((cache, q_lat))
    # the squares are added in another order (2^-24 of the sum each) and a turn's two products may be contracted either way; then one
    # rounding, which may fall to either side
    step = 2.0 ** -7 if dtype == torch.bfloat16 else (rank + 8) * 2.0 ** -23
    for a, b in zip(*out):
        assert ((a.double() - b.double()).abs() <= step * a.double().abs() + 2.0 ** -20).all()
    assert out[0][0].abs().max() > 0

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


@pytest.mark.parametrize("rows", [13, 65, 300])
@pytest.mark.parametrize("adjacent", [False, True])
def test_a_turn_is_rounded_the_same_in_every_form(rows, adjacent):
    """x0 cos - x1 sin and x1 cos + x0 sin, the product with the cosine unrounded."""
    K = get_kernels(verbose=False)
    g = torch.Generator(device=DEV).manual_seed(rows)
    heads, dim, rot, rank, ps = 4, 16, 64, 64, 64
    cols, pages = heads * (dim + rot), -(-rows // ps)
    proj = torch.randn(rows, cols + rank + rot, device=DEV, generator=g)
    inv_freq, positions = torch.rand(rot // 2, device=DEV, generator=g), torch.arange(rows, dtype=torch.int32, device=DEV)
    cache = torch.zeros(pages, 1, 1, ps, rank + rot, device=DEV)
    q_lat = torch.zeros(rows, heads, rank + rot, device=DEV)
    K.latent_prep(proj, cols, torch.ones(rank, device=DEV), inv_freq, positions, torch.zeros_like(positions),
                  torch.arange(pages, dtype=torch.int32, device=DEV)[None], cache, q_lat, heads, dim, rot, rank, rot, ps, 1e-6, adjacent=adjacent)
    angle = positions.float()[:, None] * inv_freq
    sn, cs = angle.sin()[:, None], angle.cos()[:, None]
    part = lambda x: (x[..., ::2], x[..., 1::2]) if adjacent else (x[..., :rot // 2], x[..., rot // 2:])
    keys = cache.view(-1, rank + rot)[:rows, None, rank:]
    for x, y in ((proj[:, :cols].view(rows, heads, -1)[:, :, dim:], q_lat[:, :, rank:]), (proj[:, None, cols + rank:], keys)):
        (x0, x1), (y0, y1) = part(x), part(y)
        # (float64 holds the product and, all but never rounded twice, the sum)
        assert torch.equal(y0, (x0.double() * cs.double() - (x1 * sn).double()).float())
        assert torch.equal(y1, (x1.double() * cs.double() + (x0 * sn).double()).float())

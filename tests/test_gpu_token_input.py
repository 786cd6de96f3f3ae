"""A layer's own token input in fewer kernels: the gate's product with its activation and the token's table row (`gemm_few_table`), and the
norm of its result added to the stream together with the norm that reads the stream next (`rmsnorm_add_norm`); beside float64."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def rnd(*s, seed=0):
    return torch.randn(*s, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("dim, hidden", [(8, 72), (24, 1024), (128, 2056)])
@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_product_times_table_row(K, rows, dim, hidden, activation):
    x, w, table = rnd(rows, hidden + 4)[:, :hidden], (rnd(dim, hidden, seed=1) * hidden ** -0.5).to(BF), rnd(50, 3 * dim, seed=2).to(BF)
    ids = torch.randint(0, 50, (rows,), device=DEV, dtype=torch.int32)
    ids[0] = 49
    out = torch.full((rows + 1, dim), 7.0, device=DEV, dtype=BF)
    K.gemm_few_table(x, w, table, ids, dim, out[:rows], activation)
    z = x.to(BF).double() @ w.double().T
    act = torch.nn.functional.silu(z) if activation == "silu" else torch.nn.functional.gelu(z, approximate="tanh")
    want = act * table.double()[ids.long(), dim:2 * dim]
    # one rounding to bfloat16, and sums of `hidden` products in float32
    assert ((out[:rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all() and (out[rows] == 7.0).all()


@pytest.mark.parametrize("rows, width", [(1, 4), (3, 132), (8, 1024), (5, 2052), (300, 8192)])
@pytest.mark.parametrize("wt, w2t, out_t", [(BF, BF, BF), (torch.float32, BF, BF), (BF, torch.float32, torch.float32)])
@pytest.mark.parametrize("picked", [False, True])
def test_norm_added_and_normed(K, rows, width, wt, w2t, out_t, picked):
    h, y, w, w2 = rnd(rows, width), rnd(rows, width, seed=1) * 3, (1 + rnd(width, seed=2)).to(wt), (1 + rnd(width, seed=3)).to(w2t)
    y64 = y.double()
    want_h = h.double() + y64 / torch.sqrt((y64 * y64).mean(-1, keepdim=True) + 1e-5) * w.double()
    want = want_h / torch.sqrt((want_h * want_h).mean(-1, keepdim=True) + 1e-6) * w2.double()
    index = torch.tensor([rows - 1, -1, 0, 0], dtype=torch.int32, device=DEV) if picked else None
    if picked:
        want = want[index.long().clamp(min=0)] * (index >= 0)[:, None]
    n, before = want.shape[0], h.clone()
    out = torch.full((n + 1, width), 7.0, device=DEV, dtype=out_t)
    assert K.add_norm_fits(h, y, w, w2, out)
    K.rmsnorm_add_norm(h, y, w, 1e-5, w2, out[:n], 1e-6, row_index=index)
    assert ((out[:n].double() - want).abs() <= (2.0 ** -8 if out_t == BF else 2.0 ** -18) * want.abs() + 1e-5).all() and (out[n] == 7.0).all()
    if picked:
        assert torch.equal(h, before)
    else:
        assert ((h.double() - want_h).abs() <= 2.0 ** -20 * (before.double().abs() + (want_h - before.double()).abs())).all()

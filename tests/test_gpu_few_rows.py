"""The product of a few tokens in one kernel (csrc/gemm_few.cu) at the edges of its tiles, against float64."""
import pytest
import torch

from braidinfer_b200.csrc.api import KernelError, RowScale, get_kernels, interleave_gate_up

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
U = 2.0 ** -23         # of a float32 sum's terms (cut off or rounded); a bfloat16 result is rounded by at most 2^-8 of itself


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


# outputs: below, at and past a tile of 16 (8 where gated); tiles for 4, 8 and 16 warps a CTA, one CTA an SM and more; k: one load,
# a tail of a turn of 64, fewer turns than warps, many
@pytest.mark.parametrize("rows", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("m, k", [(1, 8), (16, 64), (40, 72), (1000, 1024), (2048, 2056), (3000, 2048), (4096, 4096), (7200, 136), (8000, 520)])
def test_product(K, rows, m, k):
    g = torch.Generator(device=DEV).manual_seed(rows + m + k)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(rows, k + 8).to(BF)[:, :k]
    w = (rnd(m, k + 16) * k ** -0.5).to(BF)[:, :k]
    shares = rnd(3, 16).abs() + 0.5
    scale = RowScale(shares, 7, 1e-5)
    rs = scale.values()[:rows, None].double()
    exact = x.double() @ w.double().T
    most = k * U * (x.double().abs() @ w.double().abs().T)
    for dtype, step in ((BF, 2.0 ** -8), (torch.float32, 0.0)):
        out = torch.full((rows + 1, m), 5.0, device=DEV, dtype=dtype)
        K.gemm_few(x, w, out[:rows])
        assert ((out[:rows].double() - exact).abs() <= (1 + step) * most + step * exact.abs()).all()
        K.gemm_few(x, w, out[:rows], in_scale=scale)
        assert ((out[:rows].double() - exact * rs).abs() <= ((1 + step) * most + (step + 1e-6) * exact.abs()) * rs).all()
        assert (out[rows] == 5.0).all()
    h = rnd(rows + 1, m)
    want = h[:rows].double() + exact
    keep = h[rows].clone()
    K.gemm_few(x, w, h[:rows], residual=h[:rows])
    assert ((h[:rows].double() - want).abs() <= most + U * want.abs()).all() and torch.equal(h[rows], keep)
    again = [torch.empty(rows, m, device=DEV) for _ in range(2)]
    for o in again:
        K.gemm_few(x, w, o)
    assert torch.equal(*again)


@pytest.mark.parametrize("rows", [1, 8, 16])
@pytest.mark.parametrize("m, k", [(1, 8), (8, 64), (24, 72), (1408, 1024), (2816, 2048), (700, 4096)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated(K, rows, m, k, act):
    g = torch.Generator(device=DEV).manual_seed(rows + m + k)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(rows, k).to(BF)
    w0, w1 = [(rnd(m, k) * k ** -0.5).to(BF) for _ in range(2)]
    scale = RowScale(torch.rand(2, 16, device=DEV, generator=g) + 0.5, 3, 1e-5)
    s = scale.values()[:rows, None].double()
    a, b = x.double() @ w0.double().T * s, x.double() @ w1.double().T * s
    e0, e1 = [k * U * (x.double().abs() @ w.double().abs().T) * s for w in (w0, w1)]
    f = a * torch.sigmoid(a) if act == "silu" else torch.nn.functional.gelu(a, approximate="tanh")
    out = torch.full((rows, m), 5.0, device=DEV, dtype=BF)
    K.gemm_few(x, interleave_gate_up(w0, w1), out, swiglu=True, in_scale=scale, activation=act)
    # both activations' slopes stay below 1.2; their float32 forms are good to a part in 2^14 of their argument's size
    slack = 1.2 * e0 * b.abs() + f.abs() * e1 + 1.2 * e0 * e1 + 2.0 ** -14 * (a * b).abs()
    assert ((out.double() - f * b).abs() <= 1.01 * slack + 2.0 ** -8 * (f * b).abs() + 1e-30).all()


def test_refusals(K):
    x, w, out = (torch.zeros(*s, device=DEV, dtype=BF) for s in ((17, 16), (4, 16), (17, 4)))
    with pytest.raises(KernelError):
        K.gemm_few(x, w, out)                                         # too many rows
    with pytest.raises(KernelError):
        K.gemm_few(x[:2], w.float(), out[:2])
    with pytest.raises(KernelError):
        K.gemm_few(x[:2], w[:, :8], out[:2])

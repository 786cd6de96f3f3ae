"""The float32 product of prompts on the tensor cores (csrc/gemm_f32_tc.cu) beside float64 and beside the FFMA kernel: edges of its tiles in
every direction, residual sums in place, numbers that are not finite; and the plain attention of few items with all its loads in flight."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


def rnd(*s, seed=0):
    return torch.randn(*s, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


@pytest.mark.parametrize("rows", [17, 32, 33, 97, 129, 480])
@pytest.mark.parametrize("m, k", [(64, 128), (127, 132), (129, 1000), (1536, 1024), (6000, 260)])
def test_product(K, rows, m, k):
    assert K.f32_tc_pays(rows, m, k)
    x, w, r = rnd(rows, k + 4)[:, :k], rnd(m, k + 8, seed=1)[:, :k], rnd(rows, m + 1, seed=2)[:, :m]
    exact = x.double() @ w.double().T
    res = torch.full((rows + 1, m + 1), 7.0, device=DEV)
    K.gemm_simt(x, w, res[:rows, :m])
    # what the parts leave out is below 2^-25 of a product, sums of 64 are cut off at 2^-23 of their size: no more than a tenth of k's roundings
    most = (0.1 * k + 4) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((res[:rows, :m].double() - exact).abs() <= most).all()
    assert (res[rows] == 7.0).all() and (res[:, m] == 7.0).all()
    res[:rows, :m] = r
    K.gemm_simt(x, w, res[:rows, :m], residual=res[:rows, :m])
    assert ((res[:rows, :m].double() - exact - r.double()).abs() <= most + 2.0 ** -23 * (exact + r.double()).abs()).all()
    assert (res[rows] == 7.0).all() and (res[:, m] == 7.0).all()
    K.check_device_errors()


def test_error_is_no_larger_than_that_of_float32_sums(K, monkeypatch):
    for rows, m, k in ((33, 200, 1024), (480, 1024, 2816)):
        x, w = rnd(rows, k), rnd(m, k, seed=1)
        exact, out = x.double() @ w.double().T, torch.empty(rows, m, device=DEV)
        errors = []
        for tensor_cores in (True, False):
            monkeypatch.setattr(K, "f32_tc_pays", lambda *a: tensor_cores)
            K.gemm_simt(x, w, out)
            errors.append(float((out.double() - exact).norm()))
        assert errors[0] <= errors[1]


@pytest.mark.parametrize("ex, ew", [(-100, 0), (-112, 0), (0, -118), (-124, 3), (-124, 100), (-140, 0), (-60, -60), (60, 30), (100, -20), (60, 60)])
def test_numbers_of_any_size(K, ex, ew):
    """All of float32's bits count down to its smallest number, which the parts of an operand reach before the operand does."""
    k = 512
    x, w = rnd(40, k) * 2.0 ** (ex // 2) * 2.0 ** (ex - ex // 2), rnd(128, k, seed=1) * 2.0 ** ew
    exact, out = x.double() @ w.double().T, torch.empty(40, 128, device=DEV)
    K.gemm_simt(x, w, out)
    # as in test_product, and one rounding where the result is smaller than 2^-126
    most = (0.1 * k + 4) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -149
    assert ((out.double() - exact).abs() <= most).all()
    K.check_device_errors()


def test_numbers_that_are_not_finite(K, monkeypatch):
    x, w = rnd(100, 256), rnd(128, 256, seed=1)
    x[3, 5], x[7, 9], w[5, 9], x[60, 1] = float("inf"), float("nan"), float("-inf"), 3.4e38
    w[6] = 0.0
    w[:, 1] *= 1e-3
    got, want = torch.empty(100, 128, device=DEV), torch.empty(100, 128, device=DEV)
    K.gemm_simt(x, w, got)
    monkeypatch.setattr(K, "f32_tc_pays", lambda *a: False)
    K.gemm_simt(x, w, want)
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(got), same(want))
    ok = torch.isfinite(want)
    assert float((got[ok].double() - want[ok].double()).norm() / want[ok].double().norm()) < 2.0 ** -20

"""The 32-bit path's products and attention at the edges of their tiles: every size at which a kernel hands over to the next,
against float64."""
import pytest
import torch

from braidinfer_b200.csrc.api import get_kernels
from test_gpu_kernels import attention_case, rnd

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    return get_kernels(verbose=False)


# rows: one token, a token tile and one more, the last few-rows size and the next, a tile edge; outputs: below, at and past a
# group of four rows and a tile of 64; k: one 16-byte load, a tail of a lane pass, several slices, no multiple of 4
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8, 9, 16, 17, 64, 65, 130])
@pytest.mark.parametrize("m, k", [(1, 4), (3, 132), (64, 20), (65, 516), (200, 2816), (1030, 64), (40, 66), (5000, 36)])
def test_float32_product(K, rows, m, k):
    x, w, r = rnd(rows, k + 4)[:, :k], rnd(m, k, seed=1), rnd(rows, m + 1, seed=2)[:, :m]
    exact = x.double() @ w.double().T
    # any order of k fused multiply-adds is off by at most k u sum |x w| (u = 2^-24), the residual sum by one more rounding
    most = (k + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -24 * exact.abs()
    out = torch.full((rows + 1, m), 7.0, device=DEV)
    K.gemm_simt(x, w, out[:rows])
    assert ((out[:rows].double() - exact).abs() <= most).all()
    assert (out[rows] == 7.0).all()
    want = r.double() + exact
    res = torch.full((rows + 1, m + 1), 7.0, device=DEV)
    res[:rows, :m] = r
    K.gemm_simt(x, w, res[:rows, :m], residual=res[:rows, :m])
    assert ((res[:rows, :m].double() - want).abs() <= most + 2.0 ** -23 * want.abs()).all()
    assert (res[rows] == 7.0).all() and (res[:, m] == 7.0).all()


# one item to a few thousand: 8 warps, 2 warps and one warp a (token, head); contexts below, at and past a block of 32 keys
@pytest.mark.parametrize("hd", [16, 20, 64, 96, 250])
@pytest.mark.parametrize("seqs, window", [([(0, 1)], None), ([(31, 1), (32, 1)], None), ([(700, 1)], None), ([(700, 1)], 40),
                                          ([(90, 150), (3, 2)], None), ([(0, 700)], 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_plain_attention_with_several_warps_an_item(K, hd, seqs, window, dtype):
    worst, out, _ = attention_case(K, "simple", dtype, hd, 4, 2, seqs, window)
    assert worst < (2e-5 if dtype == torch.float32 else 2e-2)       # as test_gpu_kernels.py asks of this kernel
    assert (out[-1] == 0).all()                                     # the row of padding


def attend_one(K, dtype, spoil):
    """One query of four heads over 700 keys, eight warps a (token, head): 22 blocks of 32 keys, every eighth a warp's."""
    heads, kv_heads, hd, keys = 4, 2, 64, 700
    k, v = rnd(keys, kv_heads, hd, dtype=dtype, seed=1), rnd(keys, kv_heads, hd, dtype=dtype, seed=2)
    qkv = rnd(1, (heads + 2 * kv_heads) * hd, dtype=dtype, seed=3)
    qkv[0, 0:heads * hd:hd] = 1.0
    spoil(k)
    cache = torch.zeros(11, 2, kv_heads, 64, hd, device=DEV, dtype=dtype)
    for p in range(keys):
        cache[p // 64, 0, :, p % 64], cache[p // 64, 1, :, p % 64] = k[p], v[p]
    i = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out = torch.empty(1, heads * hd, device=DEV, dtype=dtype)
    K.attn_simple(qkv, out, cache, i(*range(11))[None], i(keys - 1), i(0), heads, kv_heads, hd, 64, None, 0.125)
    q = qkv[0, :heads * hd].view(heads, hd).double()
    s = torch.einsum("hd,khd->hk", q, k.double().repeat_interleave(2, 1)) * 0.125
    return out.view(heads, hd), torch.einsum("hk,khd->hd", torch.softmax(s, -1), v.double().repeat_interleave(2, 1))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("blocks", [[0], [1], [5, 13, 21], [0, 1, 2, 3, 4, 5, 6, 7]])
def test_blocks_of_keys_without_a_finite_score(K, dtype, blocks):
    """A warp whose blocks, the first or all, hold no finite score: scores of -inf weigh nothing, a NaN is not lost."""
    def spoil(value):
        def f(k):
            for b in blocks:
                k[32 * b:32 * b + 32, :, 0] = value
        return f

    out, want = attend_one(K, dtype, spoil(float("-inf")))
    assert (out.double() - want).abs().max() < (2e-5 if dtype == torch.float32 else 2e-2)
    out, _ = attend_one(K, dtype, spoil(float("nan")))
    assert torch.isnan(out).all()

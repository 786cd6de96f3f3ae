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


def products(monkeypatch, cfg, seqs):
    """(weights whose products of one decode step go through `gemm_few`, through deferred partial sums), [rows, k] each."""
    from braidinfer_b200.csrc.api import Kernels
    from braidinfer_b200.engine import Engine
    eng = Engine.from_random(cfg, 1, max_tokens=64 * seqs, max_slots=seqs, use_graphs=False, verbose=False)
    slots = [eng.open() for _ in range(seqs)]
    eng.step([(s, [1, 2, 3]) for s in slots])
    few, deferred = [], []
    run_few, run_partial = Kernels.gemm_few, Kernels.gemm_tc_partial
    monkeypatch.setattr(Kernels, "gemm_few", lambda self, x, w, *a, **kw: (few.append(tuple(w.shape)), run_few(self, x, w, *a, **kw))[1])
    monkeypatch.setattr(Kernels, "gemm_tc_partial", lambda self, x, w, *a, **kw: (deferred.append(tuple(w.shape)), run_partial(self, x, w, *a, **kw))[1])
    logits = eng.step([(s, [4]) for s in slots])
    eng.check()
    monkeypatch.undo()
    assert torch.isfinite(logits).all()
    return few, deferred


@pytest.mark.parametrize("seqs", [1, 8])
def test_sums_that_ride_in_the_next_kernel_stay_deferred(monkeypatch, seqs):
    """Products of 8.4 and 12.6 MB: with a norm and a rotary encoding that add the sums up they gain nothing from the other kernel;
    where what follows needs finished rows (dynamic tanh), they do."""
    dense = {"architectures": ["MistralForCausalLM"], "model_type": "mistral", "torch_dtype": "bfloat16", "num_hidden_layers": 1, "hidden_size": 2048,
             "num_attention_heads": 16, "num_key_value_heads": 4, "head_dim": 128, "intermediate_size": 1024, "vocab_size": 512, "rope_theta": 1e6,
             "rms_norm_eps": 1e-5, "sliding_window": None, "tie_word_embeddings": False, "max_position_embeddings": 4096}
    few, deferred = products(monkeypatch, dense, seqs)
    assert (2048, 2048) in deferred and (3072, 2048) in deferred
    assert (2048, 1024) in few and (2048, 1024) not in deferred       # 4.2 MB: the lone kernel pays all the same
    mixer = {"heads": 16, "dim": 128, "rot_dim": 64, "rot": {"base": 10000.0, "dims": 64}, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5}
    mlp = {"kind": "moe", "expert": {"ff": 64}, "router": {"experts": 4, "top": 2, "groups": {"count": 1, "keep": 1}}}
    bidinex = {"architecture": "Bidinex", "vocab": 256, "width": 2048, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "residual_mult": 1.0,
               "logit_softcap": 30.0, "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp}], "loop": None}
    few, deferred = products(monkeypatch, bidinex, seqs)
    assert (2048, 2048) in few and (2048, 2048) not in deferred

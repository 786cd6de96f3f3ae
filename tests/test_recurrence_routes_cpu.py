"""Which kernels a call of the recurrences reaches (csrc/api.py), on the CPU: a library that notes the entry points it is asked for and
launches nothing."""
import types

import pytest
import torch

from braidinfer_b200.csrc.api import KernelError, Kernels
from braidinfer_b200.parts.linear_attention import GatedLinearAttention

BF = torch.bfloat16


class Entries:
    """Every entry point, returning 0 and noting its name and arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0

    def names(self):
        return [n for n, _ in self.calls]


@pytest.fixture
def K(monkeypatch):
    k = object.__new__(Kernels)
    k.launches, k.entries = 0, Entries()
    monkeypatch.setattr(k, "part_library", lambda name: k.entries, raising=False)
    monkeypatch.setattr(k, "_stream", lambda: 0, raising=False)
    return k


def step(lens):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32)
    return types.SimpleNamespace(n_seqs=len(lens), max_q_len=max(lens), q_start=i32([sum(lens[:i]) for i in range(len(lens))]),
                                 q_len=i32(lens), slot_ids=i32(list(range(len(lens)))))


def scan(K, mode, lens, heads=2, dk=128, dv=64, dtype=BF, v_cols=None, settled=False, **how):
    rows = sum(lens)
    vc = dv if v_cols is None else v_cols
    q, k, v = (torch.zeros(rows, n, dtype=dtype) for n in (heads * dk, heads * dk, heads * vc))
    gate = {"channel": torch.zeros(rows, heads * dk), "head": torch.zeros(rows, heads, dtype=dtype), "constant": torch.zeros(heads)}[mode]
    bias = torch.zeros(heads * dk if mode == "channel" else heads, dtype=dtype)
    state = torch.zeros(len(lens), heads * dk * dv * 4, dtype=torch.uint8)
    ctx = step(lens)
    ctx.settled = settled
    K.linear_scan(q, k, v, gate, None if mode == "constant" else bias, torch.zeros(rows, heads * dv), state, 0, ctx, heads, heads, dk, dv, mode,
                  a_log=torch.zeros(heads, dtype=dtype) if mode == "head" else None, v_cols=v_cols, **how)
    return [n for n in K.entries.names() if not n.endswith("_floats")]


# one token a sequence, a short prompt, a prompt over chunks
@pytest.mark.parametrize("lens", [[1, 1], [20], [300]])
@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("mode", ["channel", "head", "constant"])
def test_options_of_another_mode_are_refused_on_every_route(K, mode, dtype, lens):
    scan(K, mode, lens, dtype=dtype)
    if mode != "constant":
        with pytest.raises(KernelError):
            scan(K, mode, lens, dtype=dtype, act_silu=True)
    with pytest.raises(KernelError):
        scan(K, mode, lens, dtype=dtype, v_cols=48)
    assert len([n for n in K.entries.names() if not n.endswith("_floats")]) == 1            # the refused calls reached no kernel


# a view into a packed buffer may start anywhere: the kernel that also does the norm moves four of its weights at a time
@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("off", [0, 1, 2, 4])
def test_norm_weights_that_start_anywhere(K, dtype, off):
    H, dk, dv, rank = 2, 64, 128, 8
    part = object.__new__(GatedLinearAttention)
    rows = lambda n, dt=dtype: types.SimpleNamespace(forward=lambda x, **how: torch.zeros(x.shape[0], n, dtype=how.get("out_dtype", dt)))
    part.rt = types.SimpleNamespace(kernels=K, empty=lambda *s: torch.empty(*s, dtype=dtype))
    part.heads, part.dk, part.dv, part.rank, part.tau, part.eps, part.out_mult = H, dk, dv, rank, 16.0, 1e-6, 1.0
    part.cols = [H * dk, H * dk, H * dv, H * dv, rank]
    part.proj, part.a2, part.o = rows(sum(part.cols)), rows(H * dk), rows(64)
    part.a2_bias, part.norm_w = torch.zeros(H * dk, dtype=dtype), torch.zeros(dv + off, dtype=dtype)[off:]
    ctx = step([1, 1, 1])
    ctx.rows, ctx.n_tokens, ctx.token_seq = 3, 3, torch.arange(3, dtype=torch.int32)
    part.forward(torch.zeros(3, 64, dtype=dtype), torch.zeros(3, 64), ctx, None, torch.zeros(3, part.state_bytes(), dtype=torch.uint8))
    assert K.entries.names() == (["braid_scan_step"] if off % 4 == 0 else ["braid_scan_step", "braid_gated_norm"])


# A kernel may read a state before the kernels ahead of it have ended only where the step says that nobody ahead writes it: two calls on one
# state with nothing between them are anyone's right.
@pytest.mark.parametrize("settled", [None, False, True])
def test_states_are_read_early_only_in_steps_that_say_so(K, settled):
    scan(K, "channel", [1, 1], settled=bool(settled))
    scan(K, "head", [20], settled=bool(settled))
    ctx = step([1, 1])
    if settled is not None:
        ctx.settled = settled
    ctx.token_seq = torch.arange(2, dtype=torch.int32)
    state = torch.zeros(2, 2 * 64 * 64 * 4, dtype=torch.uint8)
    x = torch.zeros(2, 128)
    K.causal_conv(x, torch.zeros(2, 128), torch.zeros(128, 4), None, state, 0, ctx)
    for dk, dv in ((64, 64), (32, 64)):                              # the kernel of one token, the walk
        K.delta_rule(torch.zeros(2, 2 * dk), torch.zeros(2, 2 * dk), torch.zeros(2, 2 * dv), torch.zeros(2, 2 * dk), torch.zeros(2 * dk), torch.ones(2),
                     torch.zeros(2, 2), torch.zeros(2, 2 * dv), state, 0, ctx, 2, 2, dk, dv, False)
    assert K.entries.names() == ["braid_scan_step", "braid_ssd_scan", "braid_causal_conv", "braid_delta_step", "braid_delta_rule"]
    assert [args[-2] for _, args in K.entries.calls] == [int(bool(settled))] * 5          # (the stream comes last)


# The forms over chunks keep numbers of every chunk: without room for them the step is walked, as far as the device is concerned by the
# same kernels as steps they do not take.
def test_without_room_for_the_chunks_the_step_is_walked(K, monkeypatch):
    empty = torch.empty

    def full(*size, **how):
        if size == (1 << 40,):
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **how)

    monkeypatch.setattr(torch, "empty", full)
    K.entries.braid_scan_chunk_work_floats = lambda *a: 1 << 40
    K.entries.braid_delta_work_floats = lambda *a: 1 << 40
    before = K.launches
    assert scan(K, "channel", [300]) == ["braid_linear_scan"] and scan(K, "constant", [300], act_silu=True) == ["braid_linear_scan"] * 2
    ctx, state = step([300]), torch.zeros(1, 2 * 64 * 64 * 4, dtype=torch.uint8)
    K.delta_rule(torch.zeros(300, 128), torch.zeros(300, 128), torch.zeros(300, 128), torch.zeros(300, 128), torch.zeros(128), torch.ones(2),
                 torch.zeros(300, 2), torch.zeros(300, 128), state, 0, ctx, 2, 2, 64, 64, True)
    name, args = K.entries.calls[-1]
    assert name == "braid_delta_rule" and args[-4:] == (None, 0, 0, 0)                # no scratch: token by token
    assert K.launches - before == 3


# steps whose chunks are more than a launch takes (keys of 64: where the walk, in chunks of 128, still runs)
@pytest.mark.parametrize("longest, dv, fits", [(65535 * 64, 64, True), (65535 * 64 + 1, 64, False), (16383 * 64, 256, True), (16383 * 64 + 1, 256, False)])
def test_steps_beyond_a_launch_go_on_to_the_walk(K, longest, dv, fits):
    x, out, state = torch.zeros(1, 2 * dv, dtype=BF), torch.zeros(1, 2 * dv), torch.zeros(1, 64, dtype=torch.uint8)
    ctx = types.SimpleNamespace(n_seqs=1, max_q_len=longest)
    assert K.scan_chunk_fits(x, x, x, out, state, 0, ctx, 64, dv) is fits
    assert K.f32_tc_pays(65535 * 32, 64, 128) and not K.f32_tc_pays(65535 * 32 + 1, 64, 128)


@pytest.mark.parametrize("settled", [None, False, True])
def test_cached_keys_are_read_early_only_where_the_caller_says_so(K, monkeypatch, settled):
    monkeypatch.setattr(K, "latent_attention_library", lambda rank, rot: K.entries, raising=False)
    K._error_flag = torch.zeros(8, dtype=torch.int32)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32)
    K.attn_latent_mma(torch.zeros(1, 2, 80, dtype=BF), torch.zeros(1, 2, 64, dtype=BF), torch.zeros(3, 1, 1, 64, 80, dtype=BF), i32(0, 1)[None],
                      i32(0), i32(1), i32(70), i32(0), 1, 1, 64, None, 0.1, **({} if settled is None else {"settled": settled}))
    name, args = K.entries.calls[-1]
    assert name == "braid_latent_attn_mma" and args[-3] == int(bool(settled))        # (then the error flag and the stream)

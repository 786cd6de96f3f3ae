"""What a part that adds deferred sums up itself is handed (StepContext.deferred), on the CPU: a norm of one's own that knows the partial
sums of a product, and nothing else, is given streams that wait for nothing else."""
import types

import pytest
import torch

from braidinfer_b200.engine.step import StepContext
from braidinfer_b200.parts.base import Norm
from braidinfer_b200.parts.block import PreNormResidualBlock
from braidinfer_b200.parts.norm import RMSNorm


class OwnNorm(Norm):
    accepts_deferred = True

    def __init__(self):
        self.taken = []

    def forward(self, x, ctx, row_index=None, rows=None, reader_takes_row_scale=False):
        d = ctx.take_deferred(x)
        assert d is None or d[1] == "residual"
        self.taken.append(d)
        return x


def context(calls):
    none = torch.zeros(0, dtype=torch.int32)
    kernels = types.SimpleNamespace(rmsnorm_add=lambda h, y, w, eps: calls.append(("rmsnorm_add", h, y, w, eps)),
                                    streamk_reduce=lambda *a, **kw: calls.append(("streamk_reduce",)))
    return StepContext(rows=1, n_tokens=1, n_seqs=1, token_ids=none, positions=none, token_seq=none, q_start=none, q_len=none, kv_before=none,
                       slot_ids=none, page_tables=[], want_rows=None, n_want=0, max_q_len=1, max_kv_len=1, all_decode=True, kernels=kernels)


@pytest.mark.parametrize("kind", ["normed", "residual"])
def test_a_norm_is_handed_what_it_knows(kind):
    calls, norm, h = [], OwnNorm(), torch.zeros(1, 4)
    ctx = context(calls)
    handle = ("y", "w", 1e-5) if kind == "normed" else "partial sums"
    ctx.defer(h, handle, kind)
    reader = types.SimpleNamespace(takes_row_scale=lambda: False)
    assert PreNormResidualBlock._norm(norm, h, ctx, reader) is h
    if kind == "normed":
        assert [c[0] for c in calls] == ["rmsnorm_add"] and calls[0][1] is h and norm.taken == [None]
    else:
        assert calls == [] and norm.taken == [(handle, kind)]
    assert not ctx.deferred
    assert RMSNorm.accepts_normed and not Norm.accepts_normed

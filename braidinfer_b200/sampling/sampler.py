"""Chooses the next token of every sequence of a batch on the device.

Rows that are plainly greedy go through the argmax kernel; everything else through
the sampling kernel, which applies the reference's chain in its order
(crates/braidinfer-runtime/src/sampling.rs:49-171).  The uniform number of each draw
comes from `rng.uniform(seed, sequence, step)`.
"""
from __future__ import annotations

from collections import Counter
from typing import List, Optional, Sequence

import numpy as np
import torch

from .params import SamplingParams
from .rng import entropy_seed, uniforms


class Sampler:
    # The device's error flags are sticky; they are read every this many draws (and by
    # `Engine.check()` whenever the caller wants), not after every draw.
    CHECK_EVERY = 32

    def __init__(self, kernels, device) -> None:
        self.K = kernels
        self.device = device
        self._draws = 0
        self._stages = []            # (pinned int32, device int32, event of the last copy), used in turn
        self._turn = 0
        self._work_buf: Optional[torch.Tensor] = None

    def _stage(self, words: np.ndarray) -> torch.Tensor:
        """Copy a step's option words to the device through pinned memory without blocking the
        host; three buffers in turn, each waiting for its own last copy only."""
        n = int(words.size)
        if len(self._stages) < 3:
            self._stages.append([None, None, None])
        st = self._stages[self._turn % len(self._stages)]
        self._turn += 1
        if st[0] is None or st[0].numel() < n:
            cap = max(1024, 1 << (n - 1).bit_length())
            st[0] = torch.empty(cap, dtype=torch.int32, pin_memory=True)
            st[1] = torch.empty(cap, dtype=torch.int32, device=self.device)
            st[2] = None
        if st[2] is not None:
            st[2].synchronize()
        st[0].numpy()[:n] = words
        st[1][:n].copy_(st[0][:n], non_blocking=True)
        st[2] = torch.cuda.Event()
        st[2].record()
        return st[1]

    def _work(self, rows: int, vocab: int) -> torch.Tensor:
        if self._work_buf is None or self._work_buf.numel() < rows * vocab:
            self._work_buf = torch.empty(rows * vocab, dtype=torch.float32, device=self.device)
        return self._work_buf[:rows * vocab].view(rows, vocab)

    def choose(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               sequence_ids: Sequence[int], steps: Sequence[int], histories=None) -> List[int]:
        """logits [rows, vocab] float32 on the device -> one token id per row (host ints).
        `histories` is a list, or a function returning the list, of what the repetition
        penalty looks at for each row (prompt + generated); it is only asked for when some
        row has a penalty."""
        return self._read(self._launch(logits, params, seeds, sequence_ids, steps, histories))

    def _launch(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int], sequence_ids: Sequence[int],
                steps: Sequence[int], histories=None, staged: bool = False) -> torch.Tensor:
        """The choice on the device: every option of the step in one copy, the chain's kernel behind it.  `staged`: through the
        sampler's pinned buffers and its work area, without waiting; else through memory of the call's own.  Returns the
        tokens (int32, on the device)."""
        rows, vocab = logits.shape
        out = torch.empty(rows, dtype=torch.int32, device=self.device)
        one = params[0] if rows and params and all(p is params[0] for p in params) else None       # one set of options for all rows
        if one.is_plain_greedy if one is not None else all(p.is_plain_greedy for p in params):
            self.K.argmax(logits, out)
            return out
        if len(params) != rows or min(len(seeds), len(sequence_ids), len(steps)) < rows:
            raise ValueError(f"{rows} rows of logits want as many options, seeds, sequences and steps, got {len(params)}, {len(seeds)}, "
                             f"{len(sequence_ids)} and {len(steps)}")
        distinct = params if one is None else (one,)
        penalty = [p.repetition_penalty for p in distinct] * (rows if one is not None else 1)
        penalised = any(p.repetition_penalty != 1.0 for p in distinct)
        if callable(histories):
            histories = histories() if penalised else None
        f = np.empty((5, rows), dtype=np.float32)      # temperature, top_p, min_p, rep_penalty, uniform
        f[0] = [p.temperature for p in distinct]               # (one number fills the row)
        f[1] = [p.top_p for p in distinct]
        f[2] = [p.min_p for p in distinct]
        f[3] = penalty
        f[4] = uniforms(seeds[:rows], sequence_ids[:rows], steps[:rows])
        k = np.empty(rows, dtype=np.int32)
        k[:] = [p.top_k for p in distinct]
        # what the penalty and the biases of each row name: offsets, tokens, numbers
        hist_off, bias_off = np.zeros(rows + 1, np.int32), np.zeros(rows + 1, np.int32)
        hist_tok, hist_cnt, bias_tok, bias_val = [], [], [], []
        if penalised and histories is not None:
            for i, v in enumerate(penalty):
                if v != 1.0:
                    for tok, cnt in Counter(histories[i]).items():
                        hist_tok.append(tok)
                        hist_cnt.append(cnt)
                hist_off[i + 1] = len(hist_tok)
        if any(p.logit_bias for p in distinct):
            for i, p in enumerate(params):
                for tok, delta in (p.logit_bias or ()):
                    bias_tok.append(tok)
                    bias_val.append(delta)
                bias_off[i + 1] = len(bias_tok)
        parts = [f.reshape(-1).view(np.int32), k, hist_off, bias_off, np.asarray(hist_tok, np.int32), np.asarray(hist_cnt, np.int32),
                 np.asarray(bias_tok, np.int32), np.asarray(bias_val, np.float32).view(np.int32)]
        sizes = [part.size for part in parts]
        words = np.concatenate(parts)
        if staged:
            words, work = self._stage(words), self._work(rows, vocab)
        else:
            words = torch.from_numpy(words).to(self.device)
            work = torch.empty((rows, vocab), dtype=torch.float32, device=self.device)
        opts, kd, ho, bo, ht, hc, bt, bv = words[:sum(sizes)].split(sizes)
        fd = opts.view(torch.float32).view(5, rows)
        self.K.sample(logits, work, out, fd[0], fd[4], top_k=kd, top_p=fd[1], min_p=fd[2],
                      rep_penalty=fd[3] if penalised else None, hist_off=ho if penalised else None,
                      hist_tok=ht if hist_tok else None, hist_cnt=hc if hist_cnt else None,
                      bias_off=bo, bias_tok=bt if bias_tok else None, bias_val=bv.view(torch.float32) if bias_tok else None)
        return out

    def choose_async(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
                     sequence_ids: Sequence[int], steps: Sequence[int]) -> "PendingTokens":
        """Like `choose` for rows that need no history (no repetition penalty): launches the
        choice and the copy of the tokens to pinned host memory and returns at once.  The
        tokens stay on the device too (`PendingTokens.device`), where the next step can read them."""
        if any(p.repetition_penalty != 1.0 for p in params):
            raise ValueError("choose_async cannot apply a repetition penalty: it needs the tokens on the host")
        out = self._launch(logits, params, seeds, sequence_ids, steps, staged=True)
        host = torch.empty(out.numel(), dtype=torch.int32, pin_memory=True)
        host.copy_(out, non_blocking=True)
        done = torch.cuda.Event()
        done.record()
        return PendingTokens(self, out, host, done)

    def _read(self, out: torch.Tensor) -> List[int]:
        toks = out.tolist()                    # synchronises: the step's results are complete here
        self._draws += 1
        if self._draws % self.CHECK_EVERY == 0:
            self.K.check_device_errors()
        return toks


class PendingTokens:
    """Tokens chosen on the device whose copy to the host is under way."""

    def __init__(self, sampler: Sampler, device: torch.Tensor, host: torch.Tensor, done) -> None:
        self.sampler, self.device, self.host, self.done = sampler, device, host, done

    def read(self) -> List[int]:
        self.done.synchronize()
        s = self.sampler
        s._draws += 1
        if s._draws % s.CHECK_EVERY == 0:
            s.K.check_device_errors()
        return self.host.tolist()

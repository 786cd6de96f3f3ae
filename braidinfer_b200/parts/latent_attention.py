"""Latent attention: one low-rank vector per token stands for the keys and values of all heads.

For the mixer's input x (a row per token):
    q            = Wq x                      per head [dim unrotated | rot_dim rotated] numbers
    [c' ; kr']   = Wdkv x                    kv_rank + rot_dim numbers
    c            = c' / sqrt(mean(c'^2) + eps) * w_norm           (the latent)
    kr           = rotate(kr', position)     (one rotated key part, shared by all heads)
    head h:  key = [Wuk_h c ; kr],  value = Wuv_h c
    score(i, j)  = (q_u(i) . Wuk_h c(j) + rotate(q_r(i)) . kr(j)) * scale,   j <= i, softmax over j
    out          = Wo concat_h( sigmoid(Wg x)_h * sum_j p(i, j) Wuv_h c(j) )
(Multi-head latent attention as in DeepSeek-AI, "DeepSeek-V2", 2024; the output gate per head is this
part's own option.)  Only c and kr are cached: kv_rank + rot_dim numbers a token, whatever the head count.

The cache is never expanded into keys and values.  q_u . (Wuk_h c) = (Wuk_h^T q_u) . c, so each query
head is carried into the latent space (`gemm_heads` with Wuk_h^T), attention runs as multi-query
attention over the cached rows (key: the whole row; value: its first kv_rank numbers), and the head's
output is Wuv_h applied to the attended latent (`gemm_heads` again, with the gate in its epilogue).  Wuk
and Wuv are used as stored; per-head transposes are made once at load, no product of weights is formed.

A constant factor on the mixer's output (`out_mult`, a model's residual multiplier) rides on the gate.

Options for other designs: the rotation may pair neighbours (2i, 2i + 1) instead of halves (the position encoding's
`pairing`); `window` limits a query to the last `window` positions, itself included; `shared_kv` makes a layer
without a down-projection of its own: it reads the latent and the rotated key part that an earlier layer cached
(the schedule's `cache_of`), with its own queries, Wuk, Wuv, window and output; `cache_window` widens what the
cache keeps beyond the layer's own window, for readers with a longer one.  `q_rank`: the queries are low-rank too,
q = Wuq (RMS norm of Wdq x, a weight a number); Wdq rides in the stacked product, and one kernel norms both low-rank
vectors, rotates the shared key part and writes the cache.  `sink_name`: a learned score a head that joins the softmax's
denominator once, unscaled, and has no value.
"""
from __future__ import annotations

from typing import Dict, Optional

import torch

from .base import MIXERS, POSITION_ENCODINGS, Mixer
from .linear import Linear
from .spec import CacheRequest, PartSpec, TensorSpec


EXPAND_QUERIES = 16
EXPAND_BYTES = 1 << 30
EXPAND_BESIDE_FLOPS = 6 * 10 ** 10       # what expanding the contexts of sequences of fewer queries may cost (see _expanded_pages)
STEP_SEQUENCES = slice(None)             # all sequences of a step


@MIXERS.register("latent_attention")
class LatentAttention(Mixer):
    """params: hidden_size, num_heads, dim (unrotated query/key numbers a head), rot_dim (rotated ones),
    vdim (value size a head), kv_rank, scale (on the scores), eps (of the latent's RMS norm), window
    (int | None), out_mult (default 1), gated (default True), position_encoding (a PartSpec of kind "rope"
    with head_dim = rot_dim: its rope_dim leading numbers of the rotated part turn), shared_kv (default False),
    cache_window (default: window), q_rank (default None), sink_name (default None), and the tensor names q (or dq, dq_norm,
    uq), dkv, dkv_norm, uk, uv, g, o (under the prefix)."""

    def __init__(self, params, prefix, runtime) -> None:
        super().__init__(params, prefix, runtime)
        p = params
        self.hidden = int(p["hidden_size"])
        self.heads = int(p["num_heads"])
        self.dim = int(p["dim"])
        self.rot = int(p["rot_dim"])
        self.vdim = int(p["vdim"])
        self.rank = int(p["kv_rank"])
        self.scale = float(p["scale"])
        self.eps = float(p["eps"])
        self.window = p.get("window")
        self.out_mult = float(p.get("out_mult", 1.0))
        self.gated = bool(p.get("gated", True))
        pe: PartSpec = p["position_encoding"]
        self.pe = POSITION_ENCODINGS.get(pe.kind)(pe.params, prefix, runtime)
        if self.pe.head_dim != self.rot or getattr(self.pe, "amplitude", 1.0) != 1.0:
            raise ValueError("latent_attention rotates the rot_dim part of queries and the shared key part, without a "
                             "factor on sine and cosine")
        self.adjacent = getattr(self.pe, "pairing", "half") == "adjacent"
        self.shared_kv = bool(p.get("shared_kv", False))
        self.cache_window = p.get("cache_window") or self.window
        if self.window and self.cache_window < self.window:
            raise ValueError("latent_attention: the cache must keep at least the layer's own window")
        self.q_cols = self.heads * (self.dim + self.rot)
        self.D = self.rank + self.rot
        self.q_rank = int(p["q_rank"]) if p.get("q_rank") else None
        if self.q_rank:
            # rows of zeros after the low-rank part, so that what follows and the second product's input start on 16 bytes
            self.q_rank_pad = -(-self.q_rank // 8) * 8
            self.dq_norm_name = prefix + p.get("dq_norm", "mix.dq.norm")
            self.uq = Linear(runtime, [prefix + p.get("uq", "mix.uq")], [self.q_cols], self.q_rank)
            names, outs = [prefix + p.get("dq", "mix.dq")], [self.q_rank]
        else:
            names, outs = [prefix + p.get("q", "mix.q")], [self.q_cols]
        self.sink_name = prefix + p["sink_name"] if p.get("sink_name") is not None else None
        self.sinks = self.dq_norm_w = None
        if not self.shared_kv:
            names.append(prefix + p.get("dkv", "mix.dkv"))
            outs.append(self.D)
        self.c_col = self.q_rank_pad if self.q_rank else self.q_cols       # where the latent's columns start
        self.gate_col = self.c_col + sum(outs[1:])
        if self.gated:
            names.append(prefix + p.get("g", "mix.g"))
            outs.append(self.heads)
        self.proj = Linear(runtime, names, outs, self.hidden)          # one stacked product: q, [c' ; kr'], gate
        self.norm_name = prefix + p.get("dkv_norm", "mix.dkv.norm")
        self.uk_name = prefix + p.get("uk", "mix.uk")
        self.uv_name = prefix + p.get("uv", "mix.uv")
        self.o = Linear(runtime, [prefix + p.get("o", "mix.o")], [self.hidden], self.heads * self.vdim)
        self.norm_w = self.uk_t = self.uv = self.ukv = None

    def tensor_specs(self) -> Dict[str, TensorSpec]:
        d = dict(self.proj.tensor_specs())
        if not self.shared_kv:
            d[self.norm_name] = TensorSpec((self.rank,), init="one_plus_normal")
        if self.q_rank:
            d[self.dq_norm_name] = TensorSpec((self.q_rank,), init="one_plus_normal")
            d.update(self.uq.tensor_specs())
        if self.sink_name:
            d[self.sink_name] = TensorSpec((self.heads,), std=1.0)
        d[self.uk_name] = TensorSpec((self.heads * self.dim, self.rank))
        d[self.uv_name] = TensorSpec((self.heads * self.vdim, self.rank))
        d.update(self.o.tensor_specs())
        d.update(self.pe.tensor_specs())
        return d

    def load(self, tensors) -> None:
        self.proj.load(tensors)
        w = self.proj.weight
        if self.q_rank:
            zeros = torch.zeros((self.q_rank_pad - self.q_rank, w.shape[1]), dtype=w.dtype, device=w.device)
            w = self.proj.weight = torch.cat([w[:self.q_rank], zeros, w[self.q_rank:]]).contiguous()
            self.uq.load(tensors)
            u = self.uq.weight
            if self.q_rank_pad != self.q_rank:
                u = torch.cat([u, torch.zeros((u.shape[0], self.q_rank_pad - self.q_rank), dtype=u.dtype, device=u.device)], 1)
            pad = -u.shape[0] % 8
            if pad:
                u = torch.cat([u, torch.zeros((pad, u.shape[1]), dtype=u.dtype, device=u.device)])
            self.uq.share(u.contiguous())
            self.dq_norm_w = tensors[self.dq_norm_name]
        if self.sink_name:
            self.sinks = tensors[self.sink_name].float().contiguous()     # scores are float32 in every run
        pad = -w.shape[0] % 8            # rows of zeros, so that a row of the stacked result starts on 16 bytes
        if pad:
            self.proj.weight = torch.cat([w, torch.zeros((pad, w.shape[1]), dtype=w.dtype, device=w.device)]).contiguous()
        self.o.load(tensors)
        self.pe.load(tensors)
        self.norm_w = tensors[self.norm_name] if not self.shared_kv else None
        # [heads, kv_rank, dim]: head h's matrix that carries q_u into the latent space, [out, in]
        self.uk_t = tensors[self.uk_name].view(self.heads, self.dim, self.rank).transpose(1, 2).contiguous()
        uk, uv = tensors[self.uk_name], tensors[self.uv_name]
        if (self.rt.gemm_backend == "auto" and self.rt.attention_backend == "auto" and self.rt.kernels is not None
                and self.rt.act_dtype == uk.dtype == uv.dtype == torch.bfloat16
                and self.rt.kernels.attn_latent_tc_supports(self.dim, self.rot, self.vdim, self.rank)):
            self.ukv = torch.cat([uk, uv])                  # both as one weight: prompts expand keys and values with it
            uv = self.ukv[uk.shape[0]:]
        self.uv = uv.view(self.heads, self.vdim, self.rank).contiguous()

    def cache_request(self) -> Optional[CacheRequest]:
        return CacheRequest("window" if self.window else "full", 1, self.D, self.cache_window if self.window else None, planes=1)

    def takes_row_scale(self) -> bool:
        return self.proj.takes_row_scale()

    def forward(self, x, residual, ctx, cache, state):
        if cache is None:
            raise RuntimeError("latent_attention needs a cache view")
        K = self.rt.kernels
        rows = x.shape[0]
        # [rows, q (or its low-rank part, padding) | c' kr' | gate | padding]
        proj = self.proj.forward(x, in_scale=ctx.take_row_scale(x))
        q_lat = self.rt.empty(rows, self.heads, self.D)
        writable = not cache.read_only
        if self.shared_kv and writable:
            raise RuntimeError("latent_attention: a layer without a down-projection reads another layer's cache (cache_of)")
        table, storage = (cache.page_table, cache.storage) if writable else (None, None)
        queries = proj
        if self.q_rank:
            c_q = self.rt.empty(rows, self.q_rank_pad)
            K.latent_down(proj, self.c_col, c_q, self.dq_norm_w, self.norm_w, self.pe.inv_freq, ctx.positions, ctx.token_seq,
                          table, storage, self.rot, self.rank, self.pe.rope_dim, cache.page_size, self.eps, adjacent=self.adjacent)
            table = storage = None                                    # the key part is done
            queries = self.uq.forward(c_q)
        K.latent_prep(queries, self.c_col, self.norm_w, self.pe.inv_freq, ctx.positions, ctx.token_seq, table, storage, q_lat,
                      self.heads, self.dim, self.rot, self.rank, self.pe.rope_dim, cache.page_size, self.eps,
                      adjacent=self.adjacent)
        q_u = queries[:, :self.q_cols].view(rows, self.heads, self.dim + self.rot)[:, :, :self.dim]
        gate = proj[:, self.gate_col:self.gate_col + self.heads] if self.gated else None
        if gate is None and self.out_mult != 1.0:
            raise RuntimeError("latent_attention: an output factor needs the gate's epilogue")
        out = self.rt.empty(rows, self.heads * self.vdim)
        pages, min_q = self._expanded_pages(ctx)
        if pages is None:
            self._attend_latents(q_u, q_lat, gate, out, ctx, cache)
        else:
            if ctx.rows > ctx.n_tokens:
                out.zero_()                                   # rows of padding are not written by the kernels
            for seqs in self._runs(pages):
                self._attend_latents(q_u, q_lat, gate, out, ctx, cache, seqs)
            self._attend_expanded(q_u, q_lat, gate, pages, min_q, out, ctx, cache)
        return self.o.forward(out, residual=residual, defer_to=ctx)

    @staticmethod
    def _runs(pages):
        """The neighbouring sequences without expanded pages, a slice a run."""
        none = [i for i, p in enumerate(pages) if p == 0]
        starts = [i for i in none if i == 0 or pages[i - 1]]
        ends = [i + 1 for i in none if i + 1 == len(pages) or pages[i + 1]]
        return [slice(a, b) for a, b in zip(starts, ends)]

    def _expanded_pages(self, ctx):
        """(the pages of every sequence's context that this step expands keys and values from (csrc/latent_attn_tc.cu), 0 for
        sequences that keep the latent form, and the fewest tokens of a sequence that has pages), or (None, 0) if all keep it.
        Steps that a graph may hold keep it: the context's extent is read on the host.

        Expanding costs a product of 2 kv_rank (dim + vdim) a row and head, attention saves 2 (2 kv_rank - dim - vdim) a query, row
        and head and a kernel that runs at a tenth of this one's rate: a sequence's rows pay for it where EXPAND_QUERIES of its
        queries meet them.  Sequences that bring fewer (ones that decode beside a prompt) keep the latent form, in launches of
        their own, unless all their rows cost no more than EXPAND_BESIDE_FLOPS, which is less than those launches do.  A step of
        four layers, ms, all expanded / each by itself: 16 heads of 128, rank 512, a prompt of 2,048 tokens beside 12 contexts of
        8,192 4.43 / 2.60, of 1,024 2.22 / 2.34, one of 512 beside 4 of 4,096 1.75 / 1.69; 8 heads of 64, rank 256, one of 300
        beside 16 of 2,048 1.20 / 1.72.  EXPAND_BYTES bounds the expanded rows a step holds."""
        if self.ukv is None or ctx.may_be_captured or ctx.max_q_len <= 8 or not ctx.host_q_len:
            return None, 0
        if self.gated is False and self.out_mult != 1.0:
            return None, 0
        if not self.scale > 0:                                # that kernel masks before the factor
            return None, 0
        if max(ctx.host_q_len) < EXPAND_QUERIES or (self.window and self.window < EXPAND_QUERIES):
            return None, 0
        numbers = 64 * self.heads * (self.dim + self.vdim)    # of a page, expanded
        pages = {n: self.rt.kernels.latent_pages(ctx.host_q_len, ctx.host_kv_before, self.window, n) for n in (1, EXPAND_QUERIES)}
        beside = sum(pages[1]) - sum(pages[EXPAND_QUERIES])
        min_q = EXPAND_QUERIES
        if beside * numbers * 2 * self.rank <= EXPAND_BESIDE_FLOPS and sum(pages[1]) * numbers * 2 <= EXPAND_BYTES:
            min_q = 1
        if sum(pages[min_q]) * numbers * 2 > EXPAND_BYTES:
            return None, 0
        return pages[min_q], min_q

    def _attend_expanded(self, q_u, q_lat, gate, pages, min_q, out, ctx, cache) -> None:
        K = self.rt.kernels
        rows = K.latent_expand_rows(cache.storage, cache.page_table, ctx.q_len, ctx.kv_before, self.rank, self.window, pages,
                                    min_q)
        kv = self.rt.empty(rows.shape[0], self.heads * (self.dim + self.vdim))
        K.gemm_tc(rows, self.ukv, kv)
        K.attn_latent_tc(q_u, q_lat, kv, cache.storage, out, cache.page_table, ctx.q_start, ctx.q_len, ctx.kv_before, ctx.n_seqs,
                         ctx.max_q_len, self.vdim, self.rank, self.window, self.scale, out_scale=self.out_mult, sinks=self.sinks, gate=gate,
                         min_q=min_q)

    def _attend_latents(self, q_u, q_lat, gate, out, ctx, cache, seqs=STEP_SEQUENCES) -> None:
        """Queries into the latent space, attention over the cached rows, values out of it, for the sequences `seqs` of the
        step (with all of them: its rows of padding too)."""
        K, tc = self.rt.kernels, self.rt.gemm_backend == "auto"
        row0, rows = 0, ctx.rows
        if seqs is not STEP_SEQUENCES:
            row0, rows = sum(ctx.host_q_len[:seqs.start]), sum(ctx.host_q_len[seqs])
        at = slice(row0, row0 + rows)
        K.gemm_heads(q_u[at], self.uk_t, q_lat[at, :, :self.rank], tensor_cores=tc)
        o_lat = self.rt.empty(rows, self.heads, self.rank)
        self._attend(q_lat[at], o_lat, ctx, cache, seqs, row0)
        K.gemm_heads(o_lat, self.uv, out[at].view(rows, self.heads, self.vdim), gate=gate[at] if gate is not None else None,
                     mult=self.out_mult, tensor_cores=tc)

    def _attend(self, q_lat, o_lat, ctx, cache, seqs, row0) -> None:
        """bfloat16 runs use the tensor-core kernel where it is built for the latent's size (prompts and decoding
        alike; steps of few tokens slice the context so that a handful of sequences still fills the machine);
        float32 runs, runs that ask for the plain kernels, and other sizes use one warp per (token, head)."""
        K = self.rt.kernels
        rows = slice(row0, row0 + q_lat.shape[0])
        if self.rt.is_f32 or self.rt.attention_backend == "plain" or not K.attn_latent_mma_supports(self.rank, self.rot):
            K.attn_latent_simple(q_lat, o_lat, cache.storage, cache.page_table, ctx.positions[rows], ctx.token_seq[rows],
                                 self.rank, self.window, self.scale, sinks=self.sinks)
            return
        n_seqs, max_q_len, max_kv_len = ctx.n_seqs, ctx.max_q_len, ctx.max_kv_len
        if seqs is not STEP_SEQUENCES:
            n_seqs, max_q_len = seqs.stop - seqs.start, max(ctx.host_q_len[seqs])
            max_kv_len = max(n + b for n, b in zip(ctx.host_q_len[seqs], ctx.host_kv_before[seqs]))
        elif ctx.rows > ctx.n_tokens:
            o_lat.zero_()                                     # rows of padding are not written by the kernel
        n_splits = 1
        if max_q_len <= 8:
            ctas = K.attn_latent_ctas(self.rank, self.rot, n_seqs, max_q_len, self.heads)
            span = min(max_kv_len, self.window) if self.window else max_kv_len
            tiles = max(1, -(-span // 32))
            # two CTAs an SM, and at least two key tiles a slice, which is what a CTA asks for before it waits for the queries (8 sequences
            # of 270 keys, 16 heads, attention and merge: 11.7 us a step's layer, with four tiles a slice 14.4)
            n_splits = max(1, min(296 // ctas, tiles // 2, 32))
        K.attn_latent_mma(q_lat, o_lat, cache.storage, cache.page_table[seqs], ctx.q_start[seqs], ctx.q_len[seqs], ctx.kv_before[seqs],
                          ctx.token_seq[rows], n_seqs, max_q_len, self.rank, self.window, self.scale, n_splits=n_splits,
                          sinks=self.sinks, row0=row0, settled=getattr(ctx, "settled", False))

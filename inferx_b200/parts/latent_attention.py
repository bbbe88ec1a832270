"""Latent attention: keys and values of all heads are widened from one small cached
vector per token.

Per token the input is projected down to ``kv_rank + rot_dim`` numbers: the first
``kv_rank``, RMS-normed, are the latent ``c``; the rest is a rotated key part shared by
all heads.  Head h's key is ``(W_uk[h] c | k_rot)`` and its value ``W_uv[h] c``; only
``c`` and ``k_rot`` are cached, as one record per token.  The key matrix is folded into
the query instead of widening cached latents:

    q_plain . (W_uk[h] c) = (W_uk[h]^T q_plain) . c

so attention runs with one shared key head of ``kv_rank + rot_dim`` entries whose values
are the latents themselves, and the head's output ``sum_j p_j c_j`` is widened by
``W_uv[h]`` afterwards.  That is the form for a few queries per sequence: a pair costs the
latent's size instead of a head's.  Prompt portions of enough tokens (decided by the shape
of the step) widen the records they can see once and attend over keys and values of the head's
own size, keys in two bfloat16 terms.  Queries carry ``dim`` plain and ``rot_dim`` rotated
entries per head; an optional sigmoid gate computed from the mixer's input multiplies the heads'
outputs before the output projection.

The projections that read the input (query, down-projection, gate) are one product over
concatenated weights; the per-head products are library calls batched over heads.

Two options.  Queries may go through a latent of their own (``q_rank``): the first product
then makes c_q beside the down-projection, one pass normalises c_q and writes the record,
and a second product widens c_q to the queries.  A layer without records of its own
(``own_records`` off) has no down-projection: the schedule points it at another layer's
cache, which holds that layer's records of this step too by the time it runs.
"""
from __future__ import annotations

from types import SimpleNamespace

import torch

from ..weights.loader import TensorDecl
from .base import PagedKvNeed
from .registry import build_part, register_part

ENTRY = "latent"


class LatentAttentionMixer:
    def __init__(self, spec, ctx, prefix: str):
        self.spec, self.ctx, self.prefix = spec, ctx, prefix
        self.position = build_part("position", spec.position, ctx, prefix)
        self.names = dict(spec.names)
        self.in_w = self.uk_t = self.uv = self.o_w = self.latent_gain = None
        s = spec
        self.q_width = s.heads * (s.dim + s.rot_dim)
        self.q_rank = s.q_rank              # -1 until the checkpoint says it
        self.uq_w = self.q_gain = self.kv_w = None
        self._place()

    def _place(self):
        """Columns of the first product: query (or its latent), down-projection, gate."""
        s = self.spec
        self.kv_off = self.q_rank if self.q_rank else self.q_width
        self.gate_off = self.kv_off + (s.kv_rank + s.rot_dim if s.own_records else 0)

    def check_limits(self):
        check = getattr(self.ctx.ops, "check_latent_attention_limits", None)
        if check is not None:
            check(self.spec.kv_rank, self.spec.rot_dim, self.prefix)

    def _n(self, key):
        return f"{self.prefix}.{self.names[key]}"

    def tensors(self):
        s = self.spec
        hv = s.heads * s.vdim
        if s.q_rank:
            decls = [TensorDecl(self._n("dq"), (s.q_rank, s.hidden)),
                     TensorDecl(self._n("dq_norm"), (s.q_rank,), keep="float32", init="gain"),
                     TensorDecl(self._n("uq"), (self.q_width, s.q_rank))]
        else:
            decls = [TensorDecl(self._n("q"), (self.q_width, s.hidden))]
        if s.own_records:
            decls += [TensorDecl(self._n("dkv"), (s.kv_rank + s.rot_dim, s.hidden)),
                      TensorDecl(self._n("dkv_norm"), (s.kv_rank,), keep="float32",
                                 init="gain")]
        decls += [
            TensorDecl(self._n("uk"), (s.heads * s.dim, s.kv_rank)),
            TensorDecl(self._n("uv"), (hv, s.kv_rank)),
            TensorDecl(self._n("o"), (s.hidden, hv)),
        ]
        if s.output_gate:
            decls.append(TensorDecl(self._n("g"), (hv, s.hidden)))
        return decls

    def bind(self, w):
        s = self.spec
        parts = [w[self._n("dq" if s.q_rank else "q")]]
        if s.q_rank:
            self.uq_w, self.q_gain = w[self._n("uq")], w[self._n("dq_norm")]
            self.q_rank = self.uq_w.shape[1]
            if parts[0].shape[0] != self.q_rank or self.q_gain.numel() != self.q_rank:
                raise ValueError(f"{self.prefix}: {parts[0].shape[0]} rows make the query's "
                                 f"latent, {self.q_rank} columns read it")
        if s.own_records:
            parts.append(w[self._n("dkv")])
            self.latent_gain = w[self._n("dkv_norm")]
        if s.output_gate:
            parts.append(w[self._n("g")])
        self._place()
        self.in_w = torch.cat(parts, dim=0).contiguous()
        # [heads, kv_rank, dim]: q_lat[h] = q_plain[h] . uk[h] summed over dim
        self.uk_t = w[self._n("uk")].view(s.heads, s.dim, s.kv_rank).transpose(1, 2).contiguous()
        self.uv = w[self._n("uv")].view(s.heads, s.vdim, s.kv_rank).contiguous()
        self.o_w = w[self._n("o")]
        applies = getattr(self.ctx.ops, "widened_latent_applies", None)
        self.kv_w = None
        if applies is not None and self.in_w.is_cuda and s.scale > 0 and applies(
                self.in_w.dtype, s.dim, s.rot_dim, s.vdim, s.kv_rank,
                (self.kv_off, self.gate_off, self.in_w.shape[0])):
            self.kv_w = w[self._n("uk")], self.uv

    def cache_needs(self):
        s = self.spec
        if not s.own_records:
            return []
        return [PagedKvNeed(1, s.kv_rank + s.rot_dim, s.window, entries=(ENTRY,))]

    def step_scratch_bytes(self, tokens, seqs, max_len):
        """The most that a step's attention takes beside its activations."""
        s = self.spec
        if self.kv_w is None:
            return 0
        return self.ctx.ops.widened_scratch_bytes(tokens, seqs, max_len, s.window, s.heads,
                                                  s.kv_rank, s.rot_dim, s.dim, s.vdim)

    def _pair_table(self, x):
        if self.position is not None:
            return self.position.pair_table()
        return torch.empty(0, dtype=torch.float32, device=x.device), 1.0, 0

    def _queries(self, x, proj, step, cache, group, records):
        """(rotated query parts, plain ones heads outermost); the step's records are in the
        cache when this returns."""
        s, ops = self.spec, self.ctx.ops
        freq, mag, rot_dims = self._pair_table(x)
        writes = s.own_records and cache.writes
        if not s.q_rank and s.own_records:
            return ops.latent_prepare(
                proj, 0, self.kv_off, step.positions, freq, mag, self.latent_gain, s.latent_eps,
                s.heads, s.dim, s.rot_dim, rot_dims, s.kv_rank,
                records if writes else None, group.slots if writes else None)
        q = proj
        if s.q_rank:
            c_q = ops.latent_front(
                proj, self.q_rank, self.q_gain, s.latent_eps, self.kv_off, step.positions, freq,
                mag, self.latent_gain, s.kv_rank, s.rot_dim, rot_dims,
                records if writes else None, group.slots if writes else None)
            q = ops.linear(c_q, self.uq_w)
        return ops.latent_queries(q, step.positions, freq, mag, s.heads, s.dim, s.rot_dim,
                                  rot_dims)

    def forward(self, x, step, cache):
        s, ops = self.spec, self.ctx.ops
        T = x.shape[0]
        group = step.groups[cache.group]
        proj = ops.linear(x, self.in_w)
        # single tokens come first in a batch; what follows them may attend over widened keys
        alone, rows = T, 0
        if self.kv_w is not None and not step.all_decode:
            nd = step.num_decode_seqs
            kv_lens = getattr(step, "kv_lens", None)
            rows = ops.widened_latent_rows(
                step.q_lens[nd:], step.max_kv_len, s.window, s.heads, s.kv_rank, s.rot_dim,
                s.dim + s.rot_dim + s.vdim, mixed=nd > 0, vdim=s.vdim,
                fp32_weights=s.fp32_weights, kv_lens=kv_lens[nd:] if kv_lens else None,
                bound=getattr(step, "captured", False))
            if rows:
                alone = nd
        if alone == T:
            o = self._folded(x, proj, step, cache, group)
        else:
            o = torch.empty((T, s.heads * s.vdim), dtype=x.dtype, device=x.device)
            if alone:
                group_alone = SimpleNamespace(block_table=group.block_table[:alone],
                                              slots=group.slots[:alone])
                first = SimpleNamespace(
                    positions=step.positions[:alone], seq_of_token=step.seq_of_token[:alone],
                    cu_q=step.cu_q[:alone + 1], q_pos0=step.q_pos0[:alone],
                    q_lens=step.q_lens[:alone], max_kv_len=step.max_kv_len)
                self._folded(x[:alone], proj[:alone], first, cache, group_alone, o[:alone])
            self._widened(x, proj, step, cache, group, alone, rows, o[alone:])
        return ops.linear(o, self.o_w, out_dtype=torch.float32 if s.out_float32 else None)

    def _folded(self, x, proj, step, cache, group, out=None):
        """The heads' gated outputs [T, heads * vdim], keys folded into the queries."""
        s, ops = self.spec, self.ctx.ops
        T = x.shape[0]
        records = cache.pages[ENTRY]
        q_rot, q_plain = self._queries(x, proj, step, cache, group, records)
        q_lat = ops.batched_linear(q_plain, self.uk_t)                       # [heads, T, rank]
        mixed = ops.latent_attention(q_lat, q_rot, records, group.block_table, step, s.window,
                                     s.scale, **({"fp32_weights": True} if s.fp32_weights
                                                 else {}))                   # [heads, T, rank]
        if s.output_gate:
            o = ops.gate_heads(ops.batched_linear(mixed, self.uv), proj, self.gate_off)
            return o if out is None else out.copy_(o)
        # the heads' values land beside each other, ready for the output projection
        o = out if out is not None else torch.empty((T, s.heads * s.vdim), dtype=x.dtype,
                                                    device=x.device)
        ops.batched_linear(mixed, self.uv, out=o.view(T, s.heads, s.vdim).transpose(0, 1))
        return o

    def _widened(self, x, proj, step, cache, group, first, rows, out):
        """The same for the tokens from ``first`` on (the first ``first`` sequences bring one
        token each), over widened keys and values, into ``out``."""
        s, ops = self.spec, self.ctx.ops
        records = cache.pages[ENTRY]
        ld = proj.shape[1]
        flat = proj[first:].view(-1)
        positions = step.positions[first:]
        freq, mag, rot_dims = self._pair_table(x)
        writes = s.own_records and cache.writes
        kept = records if writes else None
        slots = group.slots[first:] if writes else None
        q, q_ld = flat, ld
        if s.q_rank:
            c_q = ops.latent_front(
                proj[first:], self.q_rank, self.q_gain, s.latent_eps, self.kv_off, positions,
                freq, mag, self.latent_gain, s.kv_rank, s.rot_dim, rot_dims, kept, slots)
            q, q_ld = ops.linear(c_q, self.uq_w).view(-1), self.q_width
            kept = slots = None
        ops.latent_front_inplace(q, q_ld, flat[self.kv_off:] if kept is not None else None, ld,
                                 positions, freq, mag, self.latent_gain, s.latent_eps, s.heads,
                                 s.dim, s.rot_dim, rot_dims, s.kv_rank, kept, slots)
        rec = ops.latent_collect(records, group.block_table[first:], step.q_pos0[first:],
                                 step.kv_len[first:], rows, s.window)
        kv = ops.latent_widen(rec, s.kv_rank, *self.kv_w, s.heads, s.dim)
        ops.widened_attention(
            q, q_ld, kv, step.cu_q_prompt if first else step.cu_q, step.q_pos0[first:],
            x.shape[0] - first, s.heads, s.dim + s.rot_dim, s.vdim, rows, s.window, s.scale,
            gate=flat[self.gate_off:] if s.output_gate else None, gate_ld=ld, out=out,
            second=s.dim, fp32_weights=s.fp32_weights)


register_part("mixer", "latent_attention", LatentAttentionMixer)

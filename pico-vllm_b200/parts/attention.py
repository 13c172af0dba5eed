"""Grouped-query attention over the paged cache: the mixer of this architecture.

qkv projection (bias added inside the rotary kernel) -> rotation of q and k and store of k, v
into pages (one kernel) -> paged causal attention (optionally over a window) -> output
projection.  Same order as pico_vllm/model.py:200-227 (projection, split, RoPE, cache store,
paged attention, o_proj); scale head_dim^-1/2 (pico_vllm/kernels/attention.py:92,231).  One
code path serves portions of prompts and single decoded tokens; the reference has three
(pico_vllm/model.py:186-302).
"""
from __future__ import annotations

from dataclasses import dataclass, replace
from typing import List, Optional

import torch

from .. import ops
from ..errors import KernelError
from .base import CacheView, MixerPlan, PagedKV, Param, Part, Piece, StepShape
from .registry import register


@dataclass(frozen=True)
class AttentionPlan(MixerPlan):
    splits: int = 1            # parts each single token's key range is cut into
    pair_min_keys: int = 0     # > 0: prompt attention gives every query tile two blocks, which share a tile
                               # that sees at least this many keys (two partial results per token and head in scratch)
    run_parts: int = 0         # > 0: instead of `splits`, parts of every run of rows, portions included (the general kernel)
    part_keys: int = 0         # > 0: but no more than have this many keys each


MAX_MIXED_SCRATCH = 32 << 20       # float32 numbers (128 MB) that splitting the single tokens of a mixed step may ask for


MIXED_MIN_KEYS = 1024              # longest context of the single tokens of a mixed step from which they are counted alone


RUN_MIN_KEYS, RUN_SHARED = 384, 228 << 10      # see GQAAttention._run_parts; bytes of shared memory of a multiprocessor


DECODE_RAGGED_KEYS = 4096          # longest context from which the parts of a ragged batch need not all run at once


def adds_in_cluster(shape: StepShape, n_heads: int, n_kv_heads: int, head_dim: int) -> bool:
    """Whether single tokens run in the kernel that adds the parts of a token's keys up in a cluster (see :func:`decode_splits`)."""
    engine = shape.engine
    dtype = getattr(torch, getattr(engine, "dtype", "") or "float32")
    return ops.mma_attention_takes(dtype, n_heads, n_kv_heads, head_dim) and ops.decode_tma_takes(head_dim, getattr(engine, "page_size", 0))


def decode_splits(shape: StepShape, n_kv_heads: int, window: Optional[int] = None, cluster: bool = True) -> int:
    """How many parts to cut each single token's key range into: a power of two (the parts of one
    token and kv head run as one thread-block cluster): up to 16 while that is at most one block
    per SM, else up to 8 while the blocks make no more than one wave of two per SM; each part at
    least two tiles of 64 keys of the context, or of the ``window`` a token sees of it.

    bfloat16, in the kernel that adds a token's parts up in a ``cluster`` (in the others a second launch does, and a part costs more: 16
    tokens of 2 kv heads with 512 keys in 1 / 2 / 4 parts 29 / 19 / 14 us, here 8.9 / 8.0 / 6.6): eight or four parts of one tile and more,
    eight while that is at most one block per SM, four up to seven blocks per four (us of the kernel, heads of 128, in 1 / 2 / 4 / 8
    parts: 16 blocks unsplit, 512 and 800 keys 8.8 / 8.0 / 6.4 / 6.1 and 12.3 / 10.0 / 7.6 / 6.8; 32 blocks 8.9 / 8.0 / 6.7 / 7.4 and 12.3 / 10.1 / 8.0 /
    8.1; 64 blocks, 300 and 504 keys 7.2 / 8.0 / 7.4 / 13 and 9.3 / 9.0 / 8.0 / 14; 74 blocks 6.9 / 7.2 / 12 / 18 and 8.9 / 8.3 / 13 / 18: clusters of
    four no longer run all at once); no two parts under 512 keys (64 tokens, 2 kv heads, in 1 / 2 parts: 400 keys 8.5 / 9.3, 504 9.5 / 9.3,
    616 10.8 / 10.0, 1,000 15.4 / 12.5).  Contexts of all ages, the longest DECODE_RAGGED_KEYS and more: four parts also where that
    makes more than a wave, since unsplit the longest sets the time (up to 8,000 keys, 4 kv heads: batch 40 / 64 / 48 in 139 / 158 /
    145 us, now 108 / 133 / 119; up to 4,096, batch 40 / 64: 88 / 100, now 80 / 96; at 3,000 some gain and some lose), but in no more
    than seven blocks a multiprocessor: the kernel alone, one of 8,000 / 4,096 keys beside 63 of 300 / 1,000, 4 kv heads 95 / 56 us, 29 / 41
    in four parts; beside 127 97 / 63, 58 / 77; beside 255 105 / 88, 112 / 144; beside 511 of 8 kv heads 117 / 301, 367 / 498.  Of
    one length they stay whole (8,000 keys, batch 40: 150 us, 156 in four parts)."""
    groups = max(1, shape.num_tokens * n_kv_heads)
    keys = shape.max_kv if window is None else min(shape.max_kv, window)
    want = 16 if groups * 16 <= shape.num_sms else min(2 * shape.num_sms // groups, 8)
    short = cluster and getattr(shape.engine, "dtype", "") == "bfloat16"
    if short and want < 4 and keys >= DECODE_RAGGED_KEYS and 4 * groups <= 7 * shape.num_sms:
        seen = [min(st + 1, keys) for n, st in zip(shape.q_lens, shape.starts) if n == 1]
        portions = sum(n for n in shape.q_lens if n > 1)
        counted = portions == 0 or shape.num_tokens < len(seen) + portions      # (scratch is for all tokens: not beside portions
        if counted and seen and 4 * sum(seen) <= 3 * keys * len(seen):          # that the mixer has not taken off)
            want = 4
    want = min(want, keys // 128)
    splits = 1
    while splits * 2 <= want:
        splits *= 2
    if short:
        for parts, blocks in ((8, shape.num_sms), (4, 7 * shape.num_sms // 4)):
            if splits < parts <= keys // 64 and parts * groups <= blocks:
                return parts
        if splits == 2 and keys < 512:
            return 1
    return splits


@register("mixer", "gqa_attention")
class GQAAttention(Part):
    fuses_residual = True   # forward(..., residual=x) may add its output to x and return None

    def __init__(self, width: int, n_heads: int, n_kv_heads: int, head_dim: int, position: Part,
                 qkv_bias: bool = True, window: Optional[int] = None, scale: Optional[float] = None):
        self.width, self.n_heads, self.n_kv_heads, self.head_dim = width, n_heads, n_kv_heads, head_dim
        self.position, self.has_bias, self.window = position, qkv_bias, window
        self.scale = head_dim ** -0.5 if scale is None else scale
        self.qkv_weight = self.qkv_bias = self.o_weight = None

    def params(self) -> List[Param]:
        q, kv = self.n_heads * self.head_dim, self.n_kv_heads * self.head_dim
        ps = [Param("qkv_weight", (Piece("q.weight", (q, self.width)), Piece("k.weight", (kv, self.width)),
                                   Piece("v.weight", (kv, self.width)))),
              Param("o_weight", (Piece("o.weight", (self.width, q)),))]
        if self.has_bias:
            ps.append(Param("qkv_bias", (Piece("q.bias", (q,)), Piece("k.bias", (kv,)), Piece("v.bias", (kv,))),
                            kind="vector"))
        return ps

    def cache_spec(self):
        return PagedKV(self.n_kv_heads, self.head_dim, self.window)

    def materialize(self, device, dtype):
        self.position.materialize(device, dtype)

    # ------------------------------------------------------------------ launch policy of the attention kernels
    def plan_key(self):
        return ("gqa_attention", self.n_heads, self.n_kv_heads, self.head_dim, self.window)

    def plan(self, shape: StepShape) -> AttentionPlan:
        splits = self._splits(shape)
        run_parts, part_keys = self._run_parts(shape, splits)
        pair = self._pair_min_keys(shape)
        parts = max(splits, 2) if pair > 0 else max(splits, run_parts)
        scratch = ops.attention_scratch_floats(shape.num_tokens, self.n_heads, self.head_dim, parts)
        return AttentionPlan(key=(splits, pair, run_parts, part_keys), scratch_floats=scratch, splits=splits, pair_min_keys=pair, run_parts=run_parts,
                             part_keys=part_keys)

    def _run_parts(self, shape: StepShape, splits: int):
        """(parts, least keys of a part) of a float32 step with portions whose time its longest run of rows sets, a portion's rows or a single
        one; (0, 0): as in other steps.  What the runs are held against is the load: the keys that all blocks of 8 rows see over the
        blocks that the device holds at once, as many steps of keys as every place of it would take if all were dealt evenly.
        In up to four parts of 128 keys and more: where the longest run has 256 keys more than 1.3 loads (in two or three parts already, half or a
        third of them and 192), while blocks of 32 rows would not fill the device.  All in four, which makes blocks of 32 rows: portions
        that take more than one round of blocks of 8, of four query heads a key head or more and not beside many single tokens (poor rows of 32),
        as long as blocks of 32 are no more than four a multiprocessor; of both, the former from two loads on, more where a head's queries leave rows of the 8
        empty (12 / 2 heads of 128, a layer, all in four / in parts of 128 keys: 150 and 137 tokens beside 8 single ones, 2.1 loads, 121 / 129; 260 beside 8,
        3 loads, 122 / 109).
        2,700 random steps of seven head sizes, up to 1,400 tokens and 200 single ones, 50 to 2,500 keys, us of the kernel whole / in parts: 683 are cut, 1.6
        times as fast in the geometric mean, five of them slower, by 8 % at most (12 / 2 heads of 128, 145 tokens beside 16 of up to 1,242 keys 127 / 46, 70
        after 530 in two parts 45 / 50 in four, left; 16 / 2, 184 beside 16 of 1,350 116 / 46; 4 / 1 of 256, 884 after 1,100 beside 8 528 / 269; 16 / 2, 2 beside 200
        of 694 84 / 109, left; 32 / 8, 63 beside 64 of 1,832 232 / 344, left)."""
        if getattr(shape.engine, "dtype", "") != "float32" or shape.max_kv < RUN_MIN_KEYS or self.window is not None:
            return 0, 0
        portions = sum(n for n in shape.q_lens if n > 1)
        if not portions:
            return 0, 0
        if 4 * shape.num_tokens * self.n_heads * (self.head_dim + 2) > MAX_MIXED_SCRATCH or splits >= 4 or not shape.spare:
            return 0, 0
        g = self.n_heads // self.n_kv_heads
        rows, tall = max(1, 8 // g), max(1, 32 // g)                   # tokens a block of 8 or 32 rows
        held = shape.num_sms * max(1, min(4, RUN_SHARED // (544 * (self.head_dim + 4) + 3264)))
        blocks = keys = 0
        for n, start in zip(shape.q_lens, shape.starts):
            b = -(-n // rows) * -(-rows * g // 8) * self.n_kv_heads
            blocks += b
            keys += b * (start + (n + 1) / 2)
        talls, singles = shape.num_tokens // tall * self.n_kv_heads, sum(1 for n in shape.q_lens if n == 1)
        many = (splits == 1 and g >= 4 and shape.max_kv * min(self.head_dim, 128) >= 640 * 128 and shape.num_sms <= 2 * talls
                and talls < 4 * shape.num_sms and 10 * blocks >= 11 * held and portions >= 2 * singles * tall)
        if talls < 2 * shape.num_sms and (splits == 1 or shape.max_kv >= 512):
            over = shape.max_kv / splits - (256 if splits == 1 else 192)
            if over * held >= (2 * (8 / (min(rows * g, 8))) ** 0.5 if many else 1.3) * keys:
                return 4, 128
        return (4, 0) if many else (0, 0)

    def _splits(self, shape: StepShape) -> int:
        """As :func:`decode_splits`, but where single tokens run in a kernel of their own beside the portions and the longest sees
        MIXED_MIN_KEYS and more, only they are
        counted: 37 of them with 3,001 tokens at most beside two portions (2,013 tokens, 28 / 4 heads) make 148 blocks unsplit,
        and the longest sets the time (68 us; 58 in two parts).  A layer with its projections, a portion of 500
        beside 20 tokens of up to 2,500 keys, 1.5B / 7B shape: 68 / 94 us, now 51 / 82; beside one of 3,000 66 / 86, now 45 / 68.  With
        short ones the kernel gains no more than what the parts cost the host (27 tokens of 504 keys, 16 / 2 heads: 8.8 us whole,
        7.5 in four parts, but the layer 57 and 60).  Scratch is laid out for every token of the step: no more parts than
        MAX_MIXED_SCRATCH holds."""
        portions = sum(n for n in shape.q_lens if n > 1)
        dtype = getattr(torch, getattr(shape.engine, "dtype", "") or "float32")
        cluster = adds_in_cluster(shape, self.n_heads, self.n_kv_heads, self.head_dim)
        if not portions or not ops.mma_attention_takes(dtype, self.n_heads, self.n_kv_heads, self.head_dim):
            return decode_splits(shape, self.n_kv_heads, cluster=cluster)
        if portions == shape.num_tokens:
            return 1
        longest = max([st + n for n, st in zip(shape.q_lens, shape.starts) if n == 1], default=1)
        if longest < MIXED_MIN_KEYS:
            return decode_splits(shape, self.n_kv_heads, cluster=cluster)
        splits = decode_splits(replace(shape, num_tokens=shape.num_tokens - portions, max_kv=longest), self.n_kv_heads, cluster=cluster)
        while splits > 1 and ops.attention_scratch_floats(shape.num_tokens, self.n_heads, self.head_dim, splits) > MAX_MIXED_SCRATCH:
            splits //= 2
        return splits

    def _pair_min_keys(self, shape: StepShape) -> int:
        """Whether prompt attention should give every query tile two blocks (the threshold in keys, or 0):
        only when every portion of the step comes after a long context (``pair_min_context`` of the engine
        configuration), where a tile takes long enough to pay for the pair, and when the tiles are too few
        to keep the SMs busy by themselves (under two per SM)."""
        m = getattr(shape.engine, "pair_min_context", 0)
        portions = [(n, st) for n, st in zip(shape.q_lens, shape.starts) if n > 1]
        if not (m > 0 and portions and shape.num_sms > 1 and getattr(shape.engine, "dtype", "") == "bfloat16"
                and min(st for _, st in portions) >= m):
            return 0
        tiles = len(portions) * self.n_heads * -(-max(n for n, _ in portions) // 128)
        return m if tiles <= 2 * shape.num_sms else 0

    def can_fuse_norm(self, x: torch.Tensor, norm) -> bool:
        """True when forward can take the residual stream itself and apply ``norm`` inside its
        first kernel (small batches)."""
        return getattr(norm, "plain_rms", False) and getattr(norm, "weight", None) is not None \
            and ops.skinny_norm_takes(x, self.qkv_weight)

    def forward(self, h: Optional[torch.Tensor], batch, cache: CacheView, residual: Optional[torch.Tensor] = None,
                norm=None):
        """Returns what is to be added to the residual stream - or, when ``residual`` is given
        and the fused small-batch kernels take the sizes, adds it there itself and returns None.
        With ``norm`` (after ``can_fuse_norm``), ``h`` is None and the normed input is computed from
        ``residual`` inside the first kernel."""
        gb = batch.groups[cache.group]
        slots = gb.slots if cache.store else None
        plan = batch.plan(self)
        pairing = getattr(self.position, "pairing", "half")
        splits, pair_min_keys = (plan.splits, plan.pair_min_keys) if plan is not None else (1, 0)
        if norm is not None:
            qkv = ops.skinny_qkv_rope_store(residual, self.qkv_weight, self.qkv_bias, batch.positions,
                                            self.position.inv_freq, slots, cache.k, cache.v, self.n_heads,
                                            self.n_kv_heads, self.head_dim, cache.page_size, norm.weight, norm.eps,
                                            pairing=pairing)
            h = qkv             # only its dtype and device are used below
        elif ops.skinny_takes(h, self.qkv_weight):
            # a handful of tokens: projection, bias, rotation and cache store are one kernel
            qkv = ops.skinny_qkv_rope_store(h, self.qkv_weight, self.qkv_bias, batch.positions,
                                            self.position.inv_freq, slots, cache.k, cache.v, self.n_heads,
                                            self.n_kv_heads, self.head_dim, cache.page_size, pairing=pairing)
        else:
            qkv = ops.linear(h, self.qkv_weight)
            ops.rope_store(qkv, self.qkv_bias, batch.positions, self.position.inv_freq, slots, cache.k, cache.v,
                           self.n_heads, self.n_kv_heads, self.head_dim, cache.page_size, pairing=pairing)
        out = torch.empty((h.shape[0], self.n_heads * self.head_dim), dtype=h.dtype, device=h.device)
        if ops.mma_attention_takes(h.dtype, self.n_heads, self.n_kv_heads, self.head_dim):
            ops.paged_attention_mma(qkv, cache.k, cache.v, out, batch.tok_seg, batch.positions, gb.block_table,
                                    batch.cu_q, batch.prefill_segs, batch.num_prefill_segs, batch.max_prefill_q,
                                    batch.decode_tokens, batch.num_decode_tokens, self.n_heads, self.n_kv_heads,
                                    self.head_dim, cache.page_size, self.window, self.scale, splits,
                                    batch.scratch, cache.k_map, cache.v_map, cache.k_map2d, cache.v_map2d,
                                    pair_min_keys)
        else:       # float32, or sizes the tensor-core kernels do not take
            parts = {"part_keys": plan.part_keys} if plan is not None and plan.run_parts else {}
            ops.paged_attention(qkv, cache.k, cache.v, out, batch.tok_seg, batch.positions, gb.block_table,
                                self.n_heads, self.n_kv_heads, self.head_dim, cache.page_size, self.window,
                                self.scale, max(splits, plan.run_parts) if plan is not None else 1, batch.scratch, **parts)
        if residual is not None and ops.skinny_takes(out, self.o_weight):
            ops.skinny_linear_residual(out, self.o_weight, residual)
            return None
        return ops.linear(out, self.o_weight)


def _linear(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """A handful of tokens: the weight-streaming kernel; more: :func:`ops.linear`."""
    if ops.skinny_takes(x, weight):
        return ops.skinny_linear(x, weight)
    return ops.linear(x, weight)


@register("mixer", "qk_norm_attention")
class QKNormAttention(Part):
    """Grouped-query softmax attention with a per-head RMS norm on queries and keys before the rotation, an optional
    soft cap on the scores, an optional sigmoid output gate, and - ``values_from_keys`` - no value projection: the
    values are the keys as projected (bias added), before norm and rotation.

        q = W_q h + b_q, k = W_k h + b_k            v = k  (or W_v h + b_v)
        q' = rot(rms(q) * w_q), k' = rot(rms(k) * w_k)        (norm over head_dim, one weight shared by the heads)
        s = scale * q' . k'(j);  s <- cap * tanh(s / cap);  p = softmax over j <= i (the last ``window`` keys, if any)
        out = W_o ( concat_heads(sum_j p(j) v(j)) * sigmoid(W_g h) )

    Launches: one product for q, k, (v) and the gate logits -> norm, rotation and cache store (one kernel) -> paged
    attention -> gate -> output product.  Norms, angles, scores and the softmax are float32."""

    def __init__(self, width: int, n_heads: int, n_kv_heads: int, head_dim: int, position: Part, eps: float,
                 scale: Optional[float] = None, softcap: Optional[float] = None, qk_norm: bool = True,
                 qk_bias: bool = True, values_from_keys: bool = False, gate: bool = False, window: Optional[int] = None):
        self.width, self.n_heads, self.n_kv_heads, self.head_dim = width, n_heads, n_kv_heads, head_dim
        self.position, self.eps, self.window = position, float(eps), window
        self.row = -(-head_dim // 16) * 16           # a head in the kernels: padded with zeros to a multiple of 16
        self.scale = head_dim ** -0.5 if scale is None else float(scale)
        self.softcap = float(softcap) if softcap else None
        self.qk_norm, self.has_bias, self.values_from_keys, self.has_gate = qk_norm, qk_bias, values_from_keys, gate
        self.proj_weight = self.proj_bias = self.q_norm = self.k_norm = self.o_weight = None

    def params(self) -> List[Param]:
        q, kv = self.n_heads * self.head_dim, self.n_kv_heads * self.head_dim
        proj = [Piece("q.weight", (q, self.width)), Piece("k.weight", (kv, self.width))]
        bias = [Piece("q.bias", (q,)), Piece("k.bias", (kv,))]
        if not self.values_from_keys:
            proj.append(Piece("v.weight", (kv, self.width)))
            bias.append(Piece("v.bias", (kv,)))
        if self.has_gate:
            proj.append(Piece("g.weight", (q, self.width)))
        ps = [Param("proj_weight", tuple(proj)), Param("o_weight", (Piece("o.weight", (self.width, q)),))]
        if self.has_bias:
            ps.append(Param("proj_bias", tuple(bias), kind="vector"))
        if self.qk_norm:
            ps += [Param("q_norm", (Piece("q.norm", (self.head_dim,)),), kind="vector", init="one_plus_normal"),
                   Param("k_norm", (Piece("k.norm", (self.head_dim,)),), kind="vector", init="one_plus_normal")]
        return ps

    def assign(self, attr: str, tensor: torch.Tensor) -> None:
        """A head size that is no multiple of 16 is padded with zeros, head by head: rows of the projections, the biases
        and the norm weights, columns of the output matrix.  Padded dimensions are zero in q, k and v and change nothing."""
        d, r = self.head_dim, self.row
        if r != d:
            if attr in ("proj_weight", "proj_bias"):
                tail = tensor.shape[1:]
                t = tensor.view(-1, d, *tail)
                tensor = torch.cat([t, t.new_zeros((t.shape[0], r - d) + tuple(tail))], 1).reshape(-1, *tail)
            elif attr in ("q_norm", "k_norm"):
                tensor = torch.cat([tensor, tensor.new_zeros(r - d)])
            elif attr == "o_weight":
                t = tensor.view(self.width, self.n_heads, d)
                tensor = torch.cat([t, t.new_zeros(self.width, self.n_heads, r - d)], 2).reshape(self.width, -1)
        setattr(self, attr, tensor.contiguous())

    def cache_spec(self):
        return PagedKV(self.n_kv_heads, self.row, self.window)

    def materialize(self, device, dtype):
        self.position.materialize(device, dtype)

    def plan_key(self):
        return ("qk_norm_attention", self.n_heads, self.n_kv_heads, self.row, self.window)

    def plan(self, shape: StepShape) -> AttentionPlan:
        splits = decode_splits(shape, self.n_kv_heads, cluster=adds_in_cluster(shape, self.n_heads, self.n_kv_heads, self.row))
        scratch = ops.attention_scratch_floats(shape.num_tokens, self.n_heads, self.row, splits)
        return AttentionPlan(key=(splits, 0), scratch_floats=scratch, splits=splits, pair_min_keys=0)

    def forward(self, h: torch.Tensor, batch, cache: CacheView) -> torch.Tensor:
        gb = batch.groups[cache.group]
        slots = gb.slots if cache.store else None
        H, G, d = self.n_heads, self.n_kv_heads, self.row
        pairing = getattr(self.position, "pairing", "rot_half")
        rot = 2 * self.position.inv_freq.shape[0]
        if pairing not in ("rot_half",) and not (pairing == "half" and rot in (0, self.head_dim)):
            raise KernelError(f"qk_norm_attention: rotary pairing {pairing!r} is not built")
        proj = _linear(h, self.proj_weight)                      # [T, q | k | (v) | (gate logits)]
        ops.qk_norm_rope_store(proj, self.proj_bias, batch.positions, self.position.inv_freq,
                               getattr(self.position, "mult", 1.0), self.q_norm, self.k_norm, self.eps, slots, cache.k,
                               cache.v, H, G, d, cache.page_size, self.values_from_keys, norm_dim=self.head_dim)
        out = torch.empty((h.shape[0], H * d), dtype=h.dtype, device=h.device)
        plan = batch.plan(self)
        splits = plan.splits if plan is not None else 1
        if ops.mma_attention_takes(h.dtype, H, G, d):
            ops.paged_attention_mma(proj, cache.k, cache.v, out, batch.tok_seg, batch.positions, gb.block_table,
                                    batch.cu_q, batch.prefill_segs, batch.num_prefill_segs, batch.max_prefill_q,
                                    batch.decode_tokens, batch.num_decode_tokens, H, G, d, cache.page_size, self.window,
                                    self.scale, splits, batch.scratch, cache.k_map, cache.v_map, cache.k_map2d,
                                    cache.v_map2d, 0, softcap=self.softcap)
        else:       # float32, or sizes the tensor-core kernels do not take
            ops.paged_attention(proj, cache.k, cache.v, out, batch.tok_seg, batch.positions, gb.block_table, H, G, d,
                                cache.page_size, self.window, self.scale, splits, batch.scratch, softcap=self.softcap)
        if self.has_gate:
            g0 = (H + G * (1 if self.values_from_keys else 2)) * d
            ops.sigmoid_gate(out, proj[:, g0:g0 + H * d])
        return _linear(out, self.o_weight)

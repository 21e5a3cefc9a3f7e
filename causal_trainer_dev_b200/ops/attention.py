"""Segment-masked flash attention: visibility metadata, the sm_100a kernels and the oracle.

Visibility rule (shared by every backend):

    key j is visible to query i  <=>  seg[j] == seg[i] != 0  and  j <= max(i, attention_end[i])

``seg`` holds canonical run ids (0 = padding) and ``attention_end`` is the optional
inclusive end index that gives MaskGIT image blocks block-local bidirectional attention.
Rows that see no key produce a zero output and zero gradients.

Reference counterparts: ``vanilla_attention`` (src/causal_trainer/modeling/attention.py:100-148),
``efficient_attention`` and its block summaries
(src/causal_trainer/kernels/efficient_attention.py:313-412, 1890-1960).
"""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch

from . import lib as _lib

BLOCK = 128


@dataclass
class AttentionMeta:
    """Per-step visibility metadata, built once and reused by every layer."""

    seg: torch.Tensor            # [B,S] int32 canonical segment ids
    lim: torch.Tensor | None     # [B,S] int32 inclusive last visible key (None: plain causal)
    kv_lo: torch.Tensor          # [B,S/128] int32
    kv_hi: torch.Tensor          # [B,S/128] int32
    q_lo: torch.Tensor           # [B,S/128] int32 first query that sees the key block
    q_hi: torch.Tensor           # [B,S/128] int32 one past the last such query
    attention_end: torch.Tensor | None = None  # kept for the oracle backend
    start: torch.Tensor | None = None        # [B,S] int32 first token of the token's run
    end: torch.Tensor | None = None          # [B,S] int32 last token of the token's run
    first_q: torch.Tensor | None = None      # [B,S] int32 first query that sees the token as a key

    @property
    def batch(self) -> int:
        return self.seg.shape[0]

    @property
    def seq(self) -> int:
        return self.seg.shape[1]


def attention_metadata(attention_mask: torch.Tensor, segment_ids: torch.Tensor | None = None,
                       attention_end: torch.Tensor | None = None) -> tuple[torch.Tensor, torch.Tensor, AttentionMeta]:
    """Canonical segment ids, restart positions and the block summaries of one micro-batch.

    On a GPU this is one launch of ``ctb_attention_meta`` (``csrc/attention_meta.cu``); elsewhere
    the PyTorch formulation (also the kernel's test oracle).  Returns ``(seg, pos, meta)``.
    """
    if not attention_mask.is_cuda:
        from ..models.decoder import canonicalize_segment_ids, make_position_ids
        seg = canonicalize_segment_ids(attention_mask, segment_ids)
        return seg, make_position_ids(attention_mask, seg, canonical=True), build_attention_meta_reference(seg, attention_end)
    bsz, s = attention_mask.shape
    if s % BLOCK:
        raise ValueError(f"sequence length {s} must be a multiple of {BLOCK}")
    dev = attention_mask.device
    i32 = lambda t: None if t is None else t.to(torch.int32).contiguous()  # noqa: E731
    mask, label, end = i32(attention_mask), i32(segment_ids), i32(attention_end)
    seg = torch.empty((bsz, s), dtype=torch.int32, device=dev)
    pos = torch.empty_like(seg)
    lim = torch.empty_like(seg)
    rows = torch.empty((4, bsz, s), dtype=torch.int32, device=dev)
    s128 = torch.empty((4, bsz, s // BLOCK), dtype=torch.int32, device=dev)
    code = _lib.lib().ctb_attention_meta(_lib.ptr(mask), _lib.ptr(label), _lib.ptr(end), bsz, s, _lib.ptr(seg),
                                         _lib.ptr(pos), _lib.ptr(lim), _lib.ptr(rows), _lib.ptr(s128),
                                         _lib.stream_ptr())
    _lib.check(code, "ctb_attention_meta")
    meta = AttentionMeta(seg, lim if attention_end is not None else None, s128[0], s128[1], s128[2], s128[3],
                         attention_end, rows[0], rows[1], rows[2])
    return seg, pos, meta


def build_attention_meta(segment_ids: torch.Tensor, attention_end: torch.Tensor | None = None) -> AttentionMeta:
    """Block summaries from canonical segment ids (contiguous runs numbered 1.., 0 for padding) and
    MaskGIT ends; ``S`` must be a multiple of 128."""
    if segment_ids.is_cuda:
        return attention_metadata(segment_ids != 0, segment_ids, attention_end)[2]
    return build_attention_meta_reference(segment_ids, attention_end)


def build_attention_meta_reference(segment_ids: torch.Tensor, attention_end: torch.Tensor | None = None) -> AttentionMeta:
    """PyTorch formulation of :func:`build_attention_meta` (CPU path and test oracle)."""
    seg = segment_ids.to(torch.int32).contiguous()
    bsz, s = seg.shape
    if s % BLOCK:
        raise ValueError(f"sequence length {s} must be a multiple of {BLOCK}")
    dev = seg.device
    idx = torch.arange(s, device=dev, dtype=torch.int32).expand(bsz, s)
    valid = seg != 0
    big = torch.iinfo(torch.int32).max
    prev = torch.cat([torch.zeros_like(seg[:, :1]), seg[:, :-1]], dim=1)
    nxt = torch.cat([seg[:, 1:], torch.zeros_like(seg[:, :1])], dim=1)
    starts = valid & (seg != prev)
    ends = valid & (seg != nxt)
    seg_start = torch.cummax(torch.where(starts, idx, torch.zeros_like(idx)), dim=1).values
    rev_end = torch.where(ends, idx, torch.full_like(idx, big)).flip(1)
    seg_end = torch.cummin(rev_end, dim=1).values.flip(1)  # inclusive last index of the run
    if attention_end is None:
        lim = None
        lim_full = idx
    else:
        lim_full = torch.maximum(idx, attention_end.to(torch.int32))
        lim_full = torch.minimum(lim_full, torch.where(valid, seg_end, idx)).contiguous()
        lim = lim_full
    nb = s // BLOCK

    def blk(x):
        return x.reshape(bsz, nb, BLOCK)

    kv_lo = blk(torch.where(valid, seg_start, torch.full_like(idx, big))).amin(-1)
    kv_hi = blk(torch.where(valid, lim_full + 1, torch.zeros_like(idx))).amax(-1)
    kv_lo = torch.where(kv_hi > 0, kv_lo, torch.zeros_like(kv_lo))
    # first query that sees key j: suffix-min over p >= j of min{i : lim[i] == p}
    if attention_end is None:
        first_q = idx
    else:
        m = torch.full((bsz, s), big, device=dev, dtype=torch.int32)
        m = m.scatter_reduce(1, lim_full.long(), torch.where(valid, idx, torch.full_like(idx, big)), "amin")
        first_q = torch.cummin(m.flip(1), dim=1).values.flip(1)
        first_q = torch.minimum(first_q, idx)
    q_lo = blk(torch.where(valid, first_q, torch.full_like(idx, big))).amin(-1)
    q_hi = blk(torch.where(valid, seg_end + 1, torch.zeros_like(idx))).amax(-1)
    q_lo = torch.where(q_hi > 0, q_lo, torch.zeros_like(q_lo))
    i32 = lambda t: t.to(torch.int32).contiguous()  # noqa: E731
    return AttentionMeta(
        seg, lim, i32(kv_lo), i32(kv_hi), i32(q_lo), i32(q_hi), attention_end,
        i32(seg_start), i32(seg_end), i32(first_q),
    )


def visibility_mask(segment_ids: torch.Tensor, attention_end: torch.Tensor | None = None) -> torch.Tensor:
    """Dense [B,S,S] boolean mask of the visibility rule (oracle only)."""
    seg = segment_ids
    s = seg.shape[1]
    idx = torch.arange(s, device=seg.device)
    lim = idx.expand_as(seg) if attention_end is None else torch.maximum(idx.expand_as(seg), attention_end.long())
    same = (seg[:, :, None] == seg[:, None, :]) & (seg[:, :, None] != 0)
    return same & (idx[None, None, :] <= lim[:, :, None])


def vanilla_attention(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, segment_ids: torch.Tensor,
    attention_end: torch.Tensor | None = None, scale: float | None = None,
) -> torch.Tensor:
    """O(S^2) fp32-softmax oracle with GQA.  q [B,S,Hq,D]; k, v [B,S,Hkv,D]."""
    b, s, hq, d = q.shape
    hkv = k.shape[2]
    scale = 1.0 / math.sqrt(d) if scale is None else scale
    g = hq // hkv
    qf = q.float().view(b, s, hkv, g, d)
    scores = torch.einsum("bqhgd,bkhd->bhgqk", qf, k.float()) * scale
    mask = visibility_mask(segment_ids, attention_end)[:, None, None]
    scores = scores.masked_fill(~mask, torch.finfo(torch.float32).min)
    probs = torch.softmax(scores, dim=-1)
    probs = torch.where(mask.any(-1, keepdim=True), probs, torch.zeros_like(probs))
    probs = probs * mask
    out = torch.einsum("bhgqk,bkhd->bqhgd", probs, v.float())
    return out.reshape(b, s, hq, d).to(q.dtype)


def _row_stride(t: torch.Tensor) -> int:
    # [B,S,H,D] view: D contiguous, heads D apart, batches S rows apart.
    b, s, _, d = t.shape
    batch, row, head, channel = t.stride()
    if channel != 1 or head != d or (b > 1 and batch != row * s):
        raise ValueError("attention operands must be [B,S,H,D] views with contiguous heads")
    return row


def _at(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


def flash_attention_forward(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, meta: AttentionMeta, scale: float | None = None,
    out: torch.Tensor | None = None, spin_budget: int = 0, q_offset: int = 0,
    kv_flags: tuple[torch.Tensor, int, int, int] | None = None,
) -> tuple[torch.Tensor, torch.Tensor]:
    """Runs the tcgen05 forward kernel; returns (O [B,Sq,Hq,D] bf16, LSE [B,Hq,Sq] fp32).

    Under sequence parallelism ``q`` holds only the queries ``[q_offset, q_offset + Sq)`` of every
    row while ``k`` / ``v`` (and ``meta``) cover the whole sequence.  ``kv_flags = (flags, chunk
    elements, elements per gathered row, epoch)`` says that ``k`` / ``v`` are the two halves of a
    buffer an all-gather pull is still filling: the kernel's producer warp acquires the chunk flags
    of every key tile before loading it.
    """
    b, sq, hq, d = q.shape
    s = k.shape[1]
    hkv = k.shape[2]
    scale = 1.0 / math.sqrt(d) if scale is None else scale
    dev = q.device
    # (sizes as arguments of their own: 1.7 us of host time an allocation, 2.5 as a tuple; a small call is bound by that)
    if out is None:
        out = torch.empty(b, sq, hq, d, dtype=torch.bfloat16, device=dev)
    lse = torch.empty(b, hq, sq, dtype=torch.float32, device=dev)
    common = (q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), meta.seg.data_ptr(), _at(meta.lim),
              _at(meta.start), meta.kv_lo.data_ptr(), meta.kv_hi.data_ptr(), b, s, sq, q_offset, hq, hkv, d,
              _row_stride(q), _row_stride(k), _row_stride(v), _row_stride(out), float(scale))
    if kv_flags is None:
        code = _lib.lib().ctb_attn_fwd_range(*common, int(spin_budget), _lib.raw_stream())
        _lib.check(code, "ctb_attn_fwd_range")
    else:
        flags, chunk, row_elems, epoch = kv_flags
        code = _lib.lib().ctb_attn_fwd_gathered(*common, flags.data_ptr(), int(chunk), int(row_elems), int(epoch),
                                                int(spin_budget), _lib.raw_stream())
        _lib.check(code, "ctb_attn_fwd_gathered")
    return out, lse


def flash_attention_backward(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, dout: torch.Tensor, lse: torch.Tensor,
    meta: AttentionMeta, scale: float | None = None, spin_budget: int = 0,
    dq: torch.Tensor | None = None, dk: torch.Tensor | None = None, dv: torch.Tensor | None = None,
    q_offset: int = 0, stats: tuple[torch.Tensor, torch.Tensor] | None = None,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """dQ (query-tile-owned work items) and dK/dV (key-tile-owned ones, group reduced in TMEM), in one launch.

    With a query range (``q_offset``, ``Sq < S``) dK / dV are this rank's partial sums over its
    queries, for all ``S`` keys.  ``stats`` are used in the place of ``lse``.  ``dq`` may take the place of ``q`` or ``dout``
    (then dK / dV are a launch of their own, before it); no other output may share memory with an input but ``out``.
    """
    b, sq, hq, d = q.shape
    s = k.shape[1]
    hkv = k.shape[2]
    scale = 1.0 / math.sqrt(d) if scale is None else scale
    out_stride, dout_stride = _row_stride(out), _row_stride(dout)
    # [B,Hq,Sq] fp32 each; a caller that splits one softmax over several passes hands in the shared ones
    dev = q.device
    if stats is None:
        both = torch.empty(2 * b * hq * sq, dtype=torch.float32, device=dev)
        neg_lse2 = both.data_ptr()
        neg_delta = neg_lse2 + 4 * b * hq * sq
    else:
        neg_lse2, neg_delta = stats[0].data_ptr(), stats[1].data_ptr()
    dq = torch.empty(b, sq, hq, d, dtype=torch.bfloat16, device=dev) if dq is None else dq
    dk = torch.empty(b, s, hkv, d, dtype=torch.bfloat16, device=dev) if dk is None else dk
    dv = torch.empty(b, s, hkv, d, dtype=torch.bfloat16, device=dev) if dv is None else dv
    # partial sums of dK / dV where the key tiles are too few for the GPU; without memory for them they are computed in one piece,
    # fp32 sums in another order: where memory runs out, the last bits of dK / dV are those of the uncut call
    # (an item of up to four iterations of 128 queries costs less than the sum of its parts: the smallest calls need not ask)
    wanted = _lib.lib().ctb_attn_bwd_workspace(b, s, sq, hq, hkv, d) if hq // hkv * sq > 512 else 0
    work = None
    if wanted:
        try:
            work = torch.empty(wanted, dtype=torch.uint8, device=dev)
        except torch.cuda.OutOfMemoryError:
            wanted = 0
    code = _lib.lib().ctb_attn_bwd_range(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr() if stats is None else None, dout.data_ptr(),
        lse.data_ptr() if stats is None else None,
        dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), neg_lse2, neg_delta, meta.seg.data_ptr(),
        _at(meta.lim), meta.kv_lo.data_ptr(), meta.kv_hi.data_ptr(), meta.q_lo.data_ptr(), meta.q_hi.data_ptr(),
        _at(meta.start), _at(meta.end), _at(meta.first_q), b, s, sq, q_offset, hq, hkv, d, _row_stride(q), _row_stride(k),
        _row_stride(v), out_stride, dout_stride, _row_stride(dq), _row_stride(dk), _row_stride(dv), float(scale),
        int(spin_budget), _at(work), wanted, _lib.raw_stream())
    _lib.check(code, "ctb_attn_bwd_range", (1 if stats is not None else 2) + (work is not None))
    return dq, dk, dv


class _FlashAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, meta, scale):
        out, lse = flash_attention_forward(q, k, v, meta, scale)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.meta = meta
        ctx.scale = scale
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out, lse = ctx.saved_tensors
        dout = dout if dout.stride(3) == 1 and dout.stride(2) == dout.shape[3] else dout.contiguous()
        dq, dk, dv = flash_attention_backward(q, k, v, out, dout, lse, ctx.meta, ctx.scale)
        return dq, dk, dv, None, None


def flash_attention(q, k, v, meta: AttentionMeta, scale: float | None = None) -> torch.Tensor:
    """Differentiable segment-masked flash attention on the sm_100a kernels."""
    return _FlashAttention.apply(q, k, v, meta, scale)

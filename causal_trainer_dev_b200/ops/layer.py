"""Python face of ``csrc/layer.cu``: a decoder layer of a small batch as one library call per direction.

The launches, their order and their arguments are those of ``training.engine.LayerwiseEngine``, so the results are the
same bits; what goes is the host time of issuing them one by one from Python (10 to 15 us each).
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import lib as _lib

_P = ctypes.c_void_p
FORWARD_LAUNCHES, BACKWARD_LAUNCHES = 9, 22


class _Shape(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("batch", "seq", "hidden", "q_heads", "kv_heads", "head_dim", "inner",
                                            "rotary_dim", "rope_style", "grad_f32", "whole_tiles")]
    _fields_ += [("eps", ctypes.c_float), ("scale", ctypes.c_float)]


class _Context(ctypes.Structure):
    _fields_ = [(n, _P) for n in ("cosine", "sine", "seg", "lim", "start", "end", "first_q", "kv_lo", "kv_hi", "q_lo", "q_hi")]


class _Weights(ctypes.Structure):
    _fields_ = [(n, _P) for n in ("ln1", "ln2", "qkv_w", "qkv_b", "o_w", "gu_w", "down_w")]


_SEGMENTS = {name for name, _ in _Weights._fields_}


def takes(layout) -> bool:
    """Whether the library's layer has all that a unit of this layout has, and trains it: the schedule in ``csrc/layer.cu`` is
    written for these segments (``qkv_b`` may be missing)."""
    names = {seg.name for seg in layout.segments}
    return names <= _SEGMENTS and names | {"qkv_b"} == _SEGMENTS


def _plan(batch: int, seq: int, hidden: int, q_heads: int, kv_heads: int, head_dim: int, inner: int, rotary_dim: int,
          rope_style: int, grad_f32: int, eps: float) -> tuple[_Shape, int, int, int]:
    """The shape as the library takes it, and the bytes of its three blocks.  (They follow the GEMM switches and the device of
    the moment, and take 10 us a pass to ask for: not kept.)"""
    shape = _Shape(batch, seq, hidden, q_heads, kv_heads, head_dim, inner, rotary_dim, rope_style, grad_f32, 0, eps,
                   1.0 / math.sqrt(head_dim))
    sizes = [ctypes.c_long() for _ in range(3)]
    _lib.lib().ctb_layer_bytes(ctypes.byref(shape), *(ctypes.byref(x) for x in sizes))
    return shape, *(x.value for x in sizes)


def _pointers(layout, base: torch.Tensor | None, skip: tuple[str, ...] = ()) -> _Weights:
    out = _Weights()
    if base is not None:
        start, size = base.data_ptr(), base.element_size()
        for seg in layout.segments:
            if seg.name not in skip:
                setattr(out, seg.name, start + seg.offset * size)
    return out


class LayerCalls:
    """The layers of one engine pass over one micro-batch."""

    def __init__(self, cfg, ctx: dict, grad_dtype: torch.dtype, train_norm: bool):
        self._shape, self._kept, self._forward, self._backward = _plan(
            ctx["batch"], ctx["seq"], cfg.hidden_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim,
            cfg.intermediate_size, cfg.rotary_dim, 0 if cfg.rope_style == "gpt-j" else 1, int(grad_dtype == torch.float32),
            cfg.rms_norm_eps)
        meta = ctx["meta"]
        at = lambda t: None if t is None else t.data_ptr()  # noqa: E731
        self._held = (ctx["cos"], ctx["sin"], meta)          # the context holds addresses of these
        self._context = _Context(ctx["cos"].data_ptr(), ctx["sin"].data_ptr(), *(at(t) for t in (
            meta.seg, meta.lim, meta.start, meta.end, meta.first_q, meta.kv_lo, meta.kv_hi, meta.q_lo, meta.q_hi)))
        self._no_grad = () if train_norm else ("ln1", "ln2")
        s = self._shape
        # (pieces of the block are whole 256 bytes)
        self._sums = -(-_lib.lib().ctb_attn_bwd_workspace(s.batch, s.seq, s.seq, s.q_heads, s.kv_heads, s.head_dim) // 256) * 256

    @property
    def scratch_bytes(self) -> int:
        """Of the larger call, without the partial sums of dK / dV: they take their time from the device's, not from the host's."""
        return max(self._forward, self._backward - self._sums)

    @property
    def backward_launches(self) -> int:
        """Kernels of a backward call; the partial sums of dK / dV are added by one more."""
        return BACKWARD_LAUNCHES + (self._sums > 0)

    def forward(self, unit, resid: torch.Tensor, branch: torch.Tensor | None) -> tuple[torch.Tensor, torch.Tensor, tuple]:
        """Returns (h, mlp, what :meth:`backward` needs)."""
        dev = resid.device
        h, mlp = torch.empty_like(resid), torch.empty_like(resid)
        kept = torch.empty(self._kept, dtype=torch.uint8, device=dev)
        scratch = torch.empty(self._forward, dtype=torch.uint8, device=dev)
        code = _lib.lib().ctb_layer_forward(
            ctypes.byref(self._shape), ctypes.byref(self._context), ctypes.byref(_pointers(unit.layout, unit.data)),
            resid.data_ptr(), None if branch is None else branch.data_ptr(), kept.data_ptr(), kept.numel(), scratch.data_ptr(),
            scratch.numel(), h.data_ptr(), mlp.data_ptr(), _lib.raw_stream())
        _lib.check(code, "ctb_layer_forward", FORWARD_LAUNCHES)
        return h, mlp, (resid if branch is None else None, h, kept)

    def backward(self, unit, grads: torch.Tensor, saved: tuple, dout: torch.Tensor, accumulate: bool) -> torch.Tensor:
        """Gradient of the layer's input; the weight gradients go into ``grads``, which is laid out as the unit."""
        x, h, kept = saved
        dx = torch.empty_like(dout)
        try:
            scratch = torch.empty(self._backward, dtype=torch.uint8, device=dout.device)
        except torch.cuda.OutOfMemoryError:
            if self._sums == 0:
                raise
            # without the partial sums: key tiles in one piece each, here and in the layers that follow (dK / dV are then sums in
            # another order, as in ops.attention)
            self._shape.whole_tiles, self._backward, self._sums = 1, self._backward - self._sums, 0
            scratch = torch.empty(self._backward, dtype=torch.uint8, device=dout.device)
        code = _lib.lib().ctb_layer_backward(
            ctypes.byref(self._shape), ctypes.byref(self._context), ctypes.byref(_pointers(unit.layout, unit.data)),
            ctypes.byref(_pointers(unit.layout, grads, self._no_grad)), accumulate, None if x is None else x.data_ptr(),
            h.data_ptr(), dout.data_ptr(), kept.data_ptr(), kept.numel(), scratch.data_ptr(), scratch.numel(), dx.data_ptr(),
            _lib.raw_stream())
        _lib.check(code, "ctb_layer_backward", self.backward_launches)
        return dx

"""Norms around a residual stream whose sublayers are normed on both sides (csrc/misc/stream_norms.cu).

``stream_norms(h, eps, post, outs, y=...)``: ``h' = h + norm(y) * post`` and ``norm(h') * w * scale`` for up to three
``(w, scale)`` of ``outs``, in one kernel.  ``branches=(routed, w_routed, dense, w_dense)`` instead of ``y``: the sum of two normed
branches, the first the weighted rows of the routed experts.  CUDA tensors of one 16-bit type; values are rounded where separate
kernels would store them.
"""
from __future__ import annotations

import torch

from . import _lib
from . import _count, _p, _stream, _DT
from .moe import RoutedRows


def takes(h: torch.Tensor, *weights: torch.Tensor) -> bool:
    return (h.is_cuda and h.dtype in (torch.bfloat16, torch.float16) and h.is_contiguous() and h.shape[1] % 8 == 0
            and h.shape[1] <= 16384 and h.data_ptr() % 16 == 0
            and all(w.dtype == h.dtype and w.is_contiguous() and w.data_ptr() % 16 == 0 for w in weights))


def stream_norms(h: torch.Tensor, eps: float, post: torch.Tensor, outs: list[tuple[torch.Tensor, float]],
                 y: torch.Tensor | None = None,
                 branches: tuple[RoutedRows, torch.Tensor, torch.Tensor, torch.Tensor] | None = None):
    """Returns ``(h', [normed outputs])``."""
    T, H = h.shape
    new = torch.empty_like(h)
    normed = [torch.empty_like(h) for _ in outs]
    if T == 0:
        return new, normed
    routed, w_s, d, w_d = branches if branches is not None else (None, None, None, None)
    assert len(outs) <= 3 and all(w.dtype == h.dtype for w, _ in outs) and post.dtype == h.dtype
    assert all(t is None or (t.dtype == h.dtype and t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0) for t in (y, d))
    assert routed is None or (routed.rows.is_contiguous() and routed.rows.shape[1] == H and routed.slot_of.is_contiguous()
                              and routed.weights.is_contiguous())
    o = [(_p(n), _p(w), float(s)) for n, (w, s) in zip(normed, outs)] + [(None, None, 1.0)] * (3 - len(outs))
    rc = _lib.kernels().fi_stream_norms(
        _p(y), 0 if y is None else y.stride(0), _p(d), 0 if d is None else d.stride(0),
        None if routed is None else _p(routed.rows), None if routed is None else _p(routed.slot_of),
        None if routed is None else _p(routed.weights), 0 if routed is None else routed.slot_of.shape[1], _p(w_s), _p(w_d), _p(post),
        _p(h), _p(new), *o[0], *o[1], *o[2], T, H, float(eps), _DT[h.dtype], _stream())
    _lib.check(rc, "fi_stream_norms")
    _count()
    return new, normed

"""``rotary_pair``: the callers' rotary embedding of q and k in one launch.

The reference's layer rotates its queries and keys with ``self.rotary(q, k, seqlen_offset=...)``
(``nha_fla/layers/nha.py:145,235``; non-interleaved halves, tables of ``K/2`` columns, positions that
restart at every packed sequence) before it calls ``chunk_nha``; the hybrid models use rotate-half with
duplicated-halves tables of ``K`` columns (``nha_fla/models/qwen3_nha/qwennha.py:240-244``).  Both are
the same arithmetic on the first ``K/2`` table columns, so one kernel serves both: ``q_swa, k_swa =
rotary_pair(q, k, cos, sin, seqlen_offset, cu_seqlens)``.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from ._lib import host as _host


def rotary_pair(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, seqlen_offset: int = 0,
                cu_seqlens: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """Rotate ``q [B,T,HQ,K]`` and ``k [B,T,H,K]`` (``B == 1`` with ``cu_seqlens``); returns bf16 ``(q_rot, k_rot)``.

    ``cos, sin``: tables ``[P, K/2]`` (or ``[P, K]`` with duplicated halves), row ``p`` for position ``p``;
    token ``t`` of a sequence uses row ``seqlen_offset + t``.  Differentiable with respect to ``q`` and ``k``.
    """
    return _host.rotary_pair(q, k, cos, sin, seqlen_offset, cu_seqlens)

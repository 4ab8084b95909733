"""``fused_chunk_nha_prefill``: inference prefill on the chunked sm_100a forward.

Same signature and return convention as ``nha_fla/ops/nha/chunk_fused.py:291-380``
(window ``[t-W+1, t]``, slot memory holds tokens ``<= t-W``, inputs in the kv-head
layout).  The reference restricts ``W <= 64`` and power-of-two ``K, V, M <= 128``;
this op takes any ``W >= 1`` (the window loop walks 64-key tiles) and
``K, V in {32,64,96,128}``, ``M`` a multiple of 16 that fits shared memory.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from ._lib import host as _host


def fused_chunk_nha_prefill(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    rotary_q: torch.Tensor,
    rotary_k: torch.Tensor,
    s: torch.Tensor,
    g: torch.Tensor,
    window_size: int,
    initial_state: Optional[Tuple[torch.Tensor, torch.Tensor]] = None,
    output_final_state: bool = False,
    scale: Optional[float] = None,
) -> Tuple[torch.Tensor, Tuple[torch.Tensor, torch.Tensor]]:
    r"""Fused NHA prefill (inference only, no autograd).

    Args: ``q, rotary_q [B,T,HQ,K]``; ``k, rotary_k [B,T,H,K]``; ``v [B,T,H,V]``;
    ``s, g [B,T,H,M]`` (kv heads); ``window_size`` W >= 1; ``initial_state``
    ``(hk0 [B,H,K,M], hv0 [B,H,M,V])`` fp32 at the kv-head count.
    Returns ``(o [B,T,HQ,V], (hkt, hvt))`` with fp32 final states or ``(None, None)``.
    """
    return _host.prefill(q, k, v, rotary_q, rotary_k, s, g, window_size, initial_state, output_final_state, scale)

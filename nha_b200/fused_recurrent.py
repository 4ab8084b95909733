"""Single-token NHA ops on the fused sm_100a decode kernel.

Same names, arguments, return values and error behaviour as
``nha_fla/ops/nha/fused_recurrent.py`` (``fused_recurrent_nha_decode`` :431-584,
``fused_recurrent_nha`` :588-682); the arithmetic runs in one CUDA launch through
``nha_decode_step`` of the C ABI, which the host module calls (csrc/host/nha_host_decode.cpp).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from ._lib import host as _host


def _stream(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def fused_recurrent_nha_decode(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    g: torch.Tensor,
    sw_k: torch.Tensor,
    sw_v: torch.Tensor,
    sq: Optional[torch.Tensor] = None,
    s: Optional[torch.Tensor] = None,
    cos: Optional[torch.Tensor] = None,
    sin: Optional[torch.Tensor] = None,
    initial_state: Optional[Tuple[torch.Tensor, torch.Tensor]] = None,
    output_final_state: bool = False,
    scale: Optional[float] = None,
) -> Tuple[torch.Tensor, Tuple[torch.Tensor, torch.Tensor]]:
    r"""Single-token fused NHA decode step with GQA support (one kernel launch).

    Args (as nha_fla/ops/nha/fused_recurrent.py:446-486):
        q: raw queries ``[B, 1, HQ, K]``.
        k, v, g: the entry leaving the window, ``[B, 1, H, K|V|M]`` (kv heads).
        sw_k, sw_v: window keys/values ``[B, W, H, K|V]``, time ascending; keys
            un-rotated when ``cos``/``sin`` are given, pre-rotated otherwise.
        sq: pre-rotated queries ``[B, 1, HQ, K]`` (required without cos/sin).
        s: optional slot write weight ``[B, 1, H, M]``; ``1 - exp(g)`` in fp32 if omitted.
        cos, sin: rotate-half tables ``[B | 1, W2 >= W, K]``; the last W rows are the
            window positions and row ``W-1`` is the query position.
        initial_state: ``(hk0 [B,H,K,M], hv0 [B,H,M,V])`` fp32, or None / (None, None) for zeros.
        output_final_state: return the updated state.
        scale: defaults to ``K ** -0.5``.

    Returns ``(o [B,1,HQ,V], (hkt, hvt))``; the tuple is ``(None, None)`` when
    ``output_final_state=False``.

    State aliasing: with ``output_final_state=True`` and a contiguous fp32
    ``initial_state`` the returned states ARE the input buffers, updated in place
    (the reference does this for ``HQ == H`` and allocates new tensors otherwise;
    its callers always store the returned tuple back into the cache).
    """
    return _host.decode(q, k, v, g, sw_k, sw_v, sq, s, cos, sin, initial_state, output_final_state, scale, False)


@torch.compiler.disable
def fused_recurrent_nha_decode_bf16_state(*args, **kwargs):
    """``fused_recurrent_nha_decode`` with the slot memory kept in bf16: same arguments; ``initial_state`` tensors in
    bf16 are updated in place (others are converted once), and the returned states are bf16.  Half the state bytes per
    step.  An extension: the reference keeps fp32 states (nha_fla/ops/nha/fused_recurrent.py:536-545), so results follow
    it to bf16 accuracy of the state only.  ``K == V`` in {64, 128} with window keys (the streaming kernel)."""
    return _bf16_state(*args, **kwargs)


def _bf16_state(q, k, v, g, sw_k, sw_v, sq=None, s=None, cos=None, sin=None, initial_state=None, output_final_state=False, scale=None):
    return _host.decode(q, k, v, g, sw_k, sw_v, sq, s, cos, sin, initial_state, output_final_state, scale, True)


@torch.compiler.disable
def fused_recurrent_nha(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    sliding_window: torch.Tensor,
    s: torch.Tensor,
    g: torch.Tensor,
    scale: Optional[float] = None,
    initial_state: Optional[Tuple[torch.Tensor]] = None,
    output_final_state: Optional[bool] = False,
) -> Tuple[torch.Tensor, torch.Tensor, list]:
    r"""Single-token NHA inference step with caller-supplied window logits.

    Args (as nha_fla/ops/nha/fused_recurrent.py:599-623): ``q [B,1,HQ,K]``,
    ``k [B,1,H,K]``, ``v [B,1,H,V]``, ``sliding_window [B,1,HQ,W]`` logits of the
    current token, ``s, g [B,1,H,M]``.  Returns ``(o, swa_score, [hkt, hvt])``:
    the slot-only readout ``[B,1,HQ,V]``, the window part of the joint softmax
    ``[B,1,HQ,W]`` (fp32) and the updated states (``[None, None]`` unless
    ``output_final_state``).  Raises ``ValueError`` for ``T != 1`` and asserts that no
    gradient is requested, like the reference (:656-660).
    """
    T = q.shape[1]
    if T != 1:
        raise ValueError(
            f"fused_recurrent_nha is the single-token inference path and expects T == 1, got T = {T}."
        )
    return _host.decode_logits(q, k, v, sliding_window, s, g, scale, initial_state, output_final_state)

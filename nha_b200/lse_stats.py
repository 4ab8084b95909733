"""``gsa_aux_loss``: the training layer's consumers of the operator's two log-sum-exps, in one launch.

The reference's layer computes, from ``lse_swa`` and ``lse_gsa`` (``nha_fla/layers/nha.py:255-264, 288-323``)::

    gsa_ratio = (w_gsa / (w_swa + w_gsa)).mean()                       # monitoring, with an .item()
    delta     = lse_gsa.float() - lse_swa.detach().float()
    aux_loss  = F.binary_cross_entropy_with_logits(delta, full_like(delta, target), reduction='mean')

``gsa_aux_loss(lse_swa, lse_gsa, target)`` returns ``(aux_loss, gsa_ratio)`` as 0-dim device tensors (no host
synchronisation); ``aux_loss`` is differentiable with respect to ``lse_gsa`` only, as in the reference.
"""
from __future__ import annotations

from typing import Tuple

import torch

from ._lib import host as _host


def gsa_aux_loss(lse_swa: torch.Tensor, lse_gsa: torch.Tensor, target_ratio: float) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(aux_loss, gsa_ratio)``: mean BCE-with-logits of ``lse_gsa - lse_swa`` against ``target_ratio`` and the mean
    share of the slot branch ``sigmoid(lse_gsa - lse_swa)``; both 0-dim fp32 tensors on the device."""
    return _host.gsa_aux_loss(lse_swa, lse_gsa, target_ratio)

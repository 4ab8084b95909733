"""``slot_gates``: the callers' gate chain in one launch.

The reference's layers compute the operator's two gate inputs from the gate projection with a chain of
element-wise torch kernels (``nha_fla/layers/nha.py:229-231``)::

    f = F.logsigmoid(f) / self.gate_logit_normalizer
    s = (1 - f.exp()).to(f.dtype)
    g = f

and the hybrid models do the same around their own ``g`` (``nha_fla/models/qwen3_nha/qwennha.py:116``).
``slot_gates(f, gate_logit_normalizer)`` returns ``(g, s)`` from one pass over ``f`` (and one pass for the
backward), so a layer replaces those three lines with ``g, s = slot_gates(f, self.gate_logit_normalizer)``.
"""
from __future__ import annotations

from typing import Tuple

import torch

from ._lib import host as _host


def slot_gates(f: torch.Tensor, gate_logit_normalizer: float = 8.0) -> Tuple[torch.Tensor, torch.Tensor]:
    """``g = logsigmoid(f) / gate_logit_normalizer`` and ``s = 1 - exp(g)``, both bf16, same shape as ``f``.

    ``f`` is the gate projection on a CUDA device (any shape; cast to bf16 like the other inputs of the
    operator).  Differentiable with respect to ``f``.
    """
    return _host.slot_gates(f, gate_logit_normalizer)

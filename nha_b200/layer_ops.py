"""Element-wise work of the calling layer around the operator, one launch each.

``feature_maps(q, k, v, feature_map='swish')`` replaces the layer's three element-wise kernels in front of the
operator (``nha_fla/layers/nha.py:219-223``)::

    q_gsa, k_gsa = map(lambda x: self.feature_map(x), (q, k))
    v = F.silu(v)

and ``silu_rms_norm_linear(o, norm_weight, norm_bias, linear_weight, linear_bias)`` the output side
(``nha_fla/layers/nha.py:277-278``)::

    o = rms_norm_linear(F.silu(o), self.g_norm.weight, self.g_norm.bias, self.o_proj.weight, self.o_proj.bias)

with silu, the RMS normalisation and its affine part in one pass over ``o`` (and one for the backward); the
projection stays a library GEMM (``F.linear``).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
import torch.nn.functional as F

from ._lib import host as _host


def feature_maps(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, feature_map: Optional[str] = 'swish'
                 ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """``(feature_map(q), feature_map(k), silu(v))`` in bf16, one launch forward and one backward.

    ``feature_map``: ``'swish'`` (``x * sigmoid(x)``), ``'relu'`` or ``None`` (q and k pass through and only ``silu(v)``
    is computed).  CUDA tensors of any shape."""
    if feature_map not in ('swish', 'relu', None):
        raise NotImplementedError(f'Feature map `{feature_map}` is not supported now.')
    return _host.feature_maps(q, k, v, 0 if feature_map == 'swish' else 1 if feature_map == 'relu' else 2)


def silu_rms_norm(o: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, eps: float = 1e-5
                  ) -> torch.Tensor:
    """``rms_norm(silu(o)) * weight + bias`` over the last dimension (a multiple of 256, at most 2048), bf16."""
    return _host.silu_rms_norm(o, weight, bias, eps)


def silu_rms_norm_linear(o: torch.Tensor, norm_weight: torch.Tensor, norm_bias: Optional[torch.Tensor],
                         linear_weight: torch.Tensor, linear_bias: Optional[torch.Tensor] = None, eps: float = 1e-5
                         ) -> torch.Tensor:
    """The layer's ``rms_norm_linear(F.silu(o), norm_weight, norm_bias, linear_weight, linear_bias)``
    (nha_fla/layers/nha.py:277-278; eps is that function's default, which the layer does not override)."""
    y = silu_rms_norm(o, norm_weight, norm_bias, eps)
    return F.linear(y.to(linear_weight.dtype), linear_weight, linear_bias)

"""The mixer and block glue (conv4 + SiLU, decay gate, sigmoid-gated RMSNorm,
residual add + RMSNorm, gated MLP).  BF16 CUDA activations, FP32 parameters;
the arithmetic is in the CUDA library (include/solvedelta_b200.h), checks and
autograd nodes are in the host extension (csrc/sd_host_glue.cpp); there is no
fallback.

Upstream counterparts: causallsso/model.py:110-164 (_packed_conv),
model.py:375-390 (decay gate), causallsso/ops/norm_gate.py:19-43,162-217.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib


def conv4_silu(x: torch.Tensor, weight: torch.Tensor, initial_state: Optional[torch.Tensor] = None,
               return_final_state: bool = False, valid_mask: Optional[torch.Tensor] = None,
               reset_mask: Optional[torch.Tensor] = None, _inplace_state: bool = False
               ) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """Depthwise causal conv (4 taps, tap 3 = current token) + SiLU over [B,T,D] BF16 rows
    (any batch/token strides, unit channel stride) with a carried [B,D,3] state.

    With masks (bool [B,T]) it is the masked token loop of causallsso/model.py:146-164, run inside
    the kernel on the padded batch: an invalid token gives zero output and leaves the state
    untouched, a reset on a valid token starts from the zero state, and the returned state of a
    row holds its last three valid inputs since the last reset (older slots show the carried state
    or zeros through).  No repacking and no host synchronisation (upstream's CUDA branch gathers
    segments around causal_conv1d instead, model.py:166-273)."""
    return _lib.host().conv4_silu(x, weight, initial_state, return_final_state, valid_mask, reset_mask, _inplace_state)


def conv4_silu_segmented(x: torch.Tensor, weight: torch.Tensor, plan, initial_state: Optional[torch.Tensor] = None,
                         return_final_state: bool = False) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """``conv4_silu`` with the masks of a segment plan from ``build_packed_segments`` (the plan is only
    checked against the input; the kernel works on the padded batch in place)."""
    if (plan.batch, plan.length) != tuple(x.shape[:2]):
        raise ValueError("packed segment plan does not match the conv input")
    return conv4_silu(x, weight, initial_state, return_final_state, plan.valid_mask, plan.reset_mask)


def add_rmsnorm_reverse_supported(width: int) -> bool:
    """Row widths the reverse pass of :func:`add_rmsnorm` is built for (whole groups of 256 channels, up to 2048)."""
    return width % 256 == 0 and 0 < width <= 2048


def add_rmsnorm(x: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float):
    """``s = x + delta`` and ``RMSNorm(s) * weight`` in one pass: returns ``(s, normed)``, both BF16 with the shape
    of ``x`` (``delta=None``: the norm alone, ``s`` is ``x``).  ``weight`` ``[D]``, FP32 without autograd; with
    autograd any floating dtype, and ``D`` must satisfy :func:`add_rmsnorm_reverse_supported`."""
    return _lib.host().add_rmsnorm(x, delta, weight, eps)


def swiglu(gate_value: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * value`` for rows ``[gate | value]``: ``[..., 2 I]`` -> ``[..., I]`` BF16, with a reverse pass
    that writes the gradient row ``[d gate | d value]`` in one kernel."""
    return _lib.host().swiglu(gate_value)


def small_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, *,
                 swiglu: bool = False) -> Optional[torch.Tensor]:
    """``F.linear(x, weight, bias)`` for the one to four rows of a cached single-token step (inference only) in the
    tensor-core kernel of the cached step (csrc/sd_token.cuh); with ``swiglu`` the result is ``silu(y[..., :N/2]) * y[..., N/2:]``.  Returns ``None`` when the
    call is not one the kernel takes (gradients recorded, more rows, not BF16 CUDA, unaligned), and the caller runs
    its library projection."""
    return _lib.host().small_linear(x, weight, bias, swiglu)


def gated_mlp(x: torch.Tensor, up: torch.Tensor, up_bias: Optional[torch.Tensor], down: torch.Tensor,
              down_bias: Optional[torch.Tensor]) -> torch.Tensor:
    """``F.linear(swiglu(F.linear(x, up, up_bias)), down, down_bias)`` for BF16 CUDA rows: library products and the
    activation kernel, or two :func:`small_linear` launches for the few rows of a cached single-token step."""
    return _lib.host().gated_mlp(x, up, up_bias, down, down_bias)


def pack_rows(pieces, widths, row_shape, device) -> Optional[torch.Tensor]:
    """One BF16 row-shaped tensor ``[..., P]`` holding ``pieces`` side by side (``None``: zeros; columns past the
    last piece: zeros), written by one kernel; ``None`` when the layout is not one the kernel takes (widths in whole
    groups of eight channels, at most twelve pieces, BF16 CUDA) and the caller has to assemble the row itself."""
    return _lib.host().pack_rows(list(pieces), list(widths), list(row_shape), torch.device(device))


def kda_decay_gate(raw: torch.Tensor, log_rate: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """log_decay = -exp(log_rate[h]) * softplus(raw + bias[h,c]); raw BF16 [...,H,r] -> FP32."""
    return _lib.host().kda_decay_gate(raw, log_rate, bias)


class _NormGateLinear(torch.autograd.Function):
    """The norm and the projection without the normalised panel among the saved tensors (the mixer itself uses the host
    extension's node, which does the same)."""

    @staticmethod
    def forward(ctx, x, gate, norm_weight, linear_weight, linear_bias, eps):
        x, gate, weight = x.contiguous(), gate.contiguous(), norm_weight.detach().float().contiguous()
        packed = linear_weight.detach().to(torch.bfloat16)
        ctx.save_for_backward(x, gate, weight, packed)
        ctx.eps = float(eps)
        ctx.dtypes = (norm_weight.dtype, linear_weight.dtype, None if linear_bias is None else linear_bias.dtype)
        ctx.set_materialize_grads(False)
        return _lib.host().norm_linear_forward(x, gate, weight, packed, linear_bias, ctx.eps)

    @staticmethod
    def backward(ctx, dout):
        if dout is None:
            return (None,) * 6
        norm_dtype, weight_dtype, bias_dtype = ctx.dtypes
        dx, dg, dw, dlinear, dbias = _lib.host().norm_linear_backward(*ctx.saved_tensors, bias_dtype is not None, ctx.eps,
                                                                      dout)
        return (dx, dg, dw.to(norm_dtype), dlinear.to(weight_dtype), None if dbias is None else dbias.to(bias_dtype),
                None)


def rms_norm_gated_linear(x: torch.Tensor, gate: torch.Tensor, norm_weight: torch.Tensor, linear_weight: torch.Tensor,
                          linear_bias: Optional[torch.Tensor], eps: float) -> torch.Tensor:
    """``F.linear(rms_norm_gated(x, gate, norm_weight, eps).flatten(-2), linear_weight, linear_bias)`` in BF16,
    with the normalised panel recomputed in the reverse pass (upstream ``RMSNormGated.forward_linear``)."""
    return _NormGateLinear.apply(x, gate, norm_weight, linear_weight, linear_bias, eps)


def rms_norm_gated(x: torch.Tensor, gate: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """y = x * rsqrt(mean(x^2) + eps) * weight * sigmoid(gate) over the last axis (<= 128)."""
    return _lib.host().rms_norm_gated(x, gate, weight, eps)


__all__ = ["add_rmsnorm", "conv4_silu", "conv4_silu_segmented", "gated_mlp", "kda_decay_gate", "rms_norm_gated",
           "rms_norm_gated_linear", "swiglu"]

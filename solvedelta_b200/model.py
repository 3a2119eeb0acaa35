"""SolveDelta mixer: fused input projection, conv4 + SiLU, decay / geometry
gates, the chunked recurrence, sigmoid-gated RMSNorm and output projection.

Same parameter names, projection layout and call signature as upstream's
``SolveDelta`` (causallsso/model.py:27-474), so upstream state dicts load:
``in_proj`` packs (q, k, v, u, h, erase_raw, write_raw, geometry_raw,
decay_hidden, output_gate_hidden) and is padded to a multiple of 64 columns
(model.py:39-60); q/k/v go through the conv, the other slices are read in
place as strided views of the projection row; decay and geometry gates are
evaluated in FP32.  The module-level name ``solvedelta_native`` is the call
site upstream's tests patch (tests/model/test_modeling_solvedelta.py:343).

GEMMs run through torch (cuBLAS); everything else is this package's CUDA
library.  Inputs must be BF16 CUDA tensors: there is no CPU path here
(upstream's CPU branch is model.py:430-462).
"""
from __future__ import annotations

import math
from typing import NamedTuple, Optional

import torch
from torch import nn

from . import _lib
from .config import SolveDeltaConfig
from .mixer_ops import rms_norm_gated
from .ops import SolveDeltaState, solvedelta_masked_native, solvedelta_native


_OPERATOR = (solvedelta_native, solvedelta_masked_native)


class SolveDeltaLayerState(NamedTuple):
    operator: SolveDeltaState
    conv: Optional[torch.Tensor]


class RMSNormGated(nn.Module):
    """y = RMSNorm(x) * weight * sigmoid(gate) (causallsso/ops/norm_gate.py:162-217)."""

    def __init__(self, hidden_size: int, eps: float = 1e-6) -> None:
        super().__init__()
        self.hidden_size = hidden_size
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(hidden_size))

    def forward(self, x: torch.Tensor, gate: torch.Tensor) -> torch.Tensor:
        return rms_norm_gated(x, gate, self.weight, self.eps)

    def forward_linear(self, x: torch.Tensor, gate: torch.Tensor, linear: nn.Linear) -> torch.Tensor:
        """The following projection without saving the normalised panel (norm_gate.py:195-217)."""
        return _lib.host().rms_norm_gated_linear(x, gate, self.weight, linear.weight, linear.bias, self.eps)


class SolveDelta(nn.Module):
    def __init__(self, config: SolveDeltaConfig) -> None:
        super().__init__()
        self.config = config
        heads = config.num_heads
        width = config.resolved_head_k_dim
        value_width = config.resolved_head_v_dim
        gate_rank = value_width
        self.projection_sizes = (
            heads * width, heads * width, heads * value_width,   # q, k, v (through the conv)
            heads * width, heads * width,                         # u, h
            heads * width, heads * value_width,                   # erase_raw, write_raw
            heads, gate_rank, gate_rank)                          # geometry_raw, decay_hidden, gate_hidden
        self.projection_width = sum(self.projection_sizes)
        self.projection_padding = (-self.projection_width) % 64
        self.in_proj = nn.Linear(config.hidden_size, self.projection_width + self.projection_padding,
                                 bias=config.bias)
        self.output_proj = nn.Linear(heads * value_width, config.hidden_size, bias=config.bias)
        self.decay_proj = nn.Linear(gate_rank, heads * width, bias=False)
        self.output_gate_proj = nn.Linear(gate_rank, heads * value_width, bias=True)
        self.output_norm = RMSNormGated(value_width, eps=config.norm_eps)
        if config.use_short_conv:
            self.conv_weight = nn.Parameter(torch.empty(sum(self.projection_sizes[:3]), 4))
            nn.init.kaiming_uniform_(self.conv_weight, a=5 ** 0.5)
        self.geometry_write_bias = nn.Parameter(torch.full((heads,), math.log(9.0), dtype=torch.float32))
        rate = torch.empty(heads, dtype=torch.float32).uniform_(1, 16)
        self.associative_log_rate = nn.Parameter(rate.log())
        step = torch.exp(torch.rand(heads, width, dtype=torch.float32) * (math.log(0.1) - math.log(0.001))
                         + math.log(0.001)).clamp_min_(1e-4)
        self.associative_decay_bias = nn.Parameter(step + torch.log(-torch.expm1(-step)))
        for parameter in (self.geometry_write_bias, self.associative_log_rate, self.associative_decay_bias):
            parameter._no_weight_decay = True

    def _fp32_copies(self):
        """FP32 copies of parameters for the fused decode step, refreshed when a parameter changes."""
        copies = self.__dict__.get("_fp32_parameter_copies")
        if copies is None:
            copies = self.__dict__["_fp32_parameter_copies"] = _lib.host().Fp32Copies()
        return copies

    def _fused_decode_applies(self, inplace_state, masked, length, initial_state, geometry_enabled,
                              associative_decay_enabled, return_final_state) -> bool:
        if not (inplace_state and return_final_state and not masked and length == 1 and self.config.use_short_conv
                and geometry_enabled and associative_decay_enabled and not torch.is_grad_enabled()):
            return False
        if initial_state is None or initial_state.conv is None or initial_state.operator is None:
            return False
        conv, (C, S) = initial_state.conv, initial_state.operator
        return (conv.dtype == torch.bfloat16 and conv.is_contiguous() and C.dtype == torch.float32
                and S.dtype == torch.float32 and C.is_contiguous() and S.is_contiguous())

    def _one_node_applies(self, initial_state, return_final_state, geometry_enabled, associative_decay_enabled) -> bool:
        """Training from empty states: the layer is one autograd node of the host extension.  Not when the operator's
        call site below has been replaced, nor under autocast, which would cast the separate products."""
        return (initial_state is None and not return_final_state and self.config.use_short_conv and geometry_enabled
                and associative_decay_enabled and torch.is_grad_enabled() and not torch.is_autocast_enabled("cuda")
                and (solvedelta_native, solvedelta_masked_native) == _OPERATOR)

    def forward(self, hidden_states: torch.Tensor, *, initial_state: Optional[SolveDeltaLayerState] = None,
                valid_mask: Optional[torch.Tensor] = None, reset_mask: Optional[torch.Tensor] = None,
                geometry_enabled: bool = True, associative_decay_enabled: bool = True,
                return_final_state: bool = False, inplace_state: bool = False):
        if hidden_states.ndim != 3:
            raise ValueError("hidden_states must have shape [B,T,hidden_size]")
        batch, length, hidden_width = hidden_states.shape
        if hidden_width != self.config.hidden_size:
            raise ValueError("hidden state width does not match the configuration")
        if hidden_states.device.type != "cuda" or hidden_states.dtype != torch.bfloat16:
            raise TypeError("the B200 mixer requires BF16 CUDA hidden states (no CPU path)")
        masked = valid_mask is not None or reset_mask is not None
        if masked:
            # masks and resets are applied inside the conv and operator kernels on the padded batch: no segment
            # plan, no host synchronisation (upstream repacks into reset-free segments, causallsso/model.py:302-316)
            for name, mask in (("valid_mask", valid_mask), ("reset_mask", reset_mask)):
                if mask is None:
                    continue
                if mask.dtype != torch.bool or mask.shape != (batch, length):
                    raise ValueError(f"{name} must be bool [B,T]")
                if mask.device != hidden_states.device:
                    raise ValueError("masks must share the activation device")
        heads = self.config.num_heads
        width = self.config.resolved_head_k_dim
        value_width = self.config.resolved_head_v_dim
        host = _lib.host()
        in_proj, decay_proj, gate_proj = self.in_proj, self.decay_proj, self.output_gate_proj
        if self._fused_decode_applies(inplace_state, masked, length, initial_state, geometry_enabled,
                                      associative_decay_enabled, return_final_state):
            # cached single-token step: conv, decay gate, geometry rate and the recurrent step in one launch, the
            # cache's conv window and operator states updated in place
            operator, output_norm, output_proj = initial_state.operator, self.output_norm, self.output_proj
            result = host.mixer_decode(
                self._fp32_copies(), hidden_states, heads, width, value_width, in_proj.weight, in_proj.bias,
                self.conv_weight, initial_state.conv, decay_proj.weight, gate_proj.weight, gate_proj.bias,
                self.associative_log_rate, self.associative_decay_bias, self.geometry_write_bias,
                operator.predictor, operator.S, output_norm.weight, output_norm.eps, output_proj.weight,
                output_proj.bias)
            return result, SolveDeltaLayerState(SolveDeltaState(operator.predictor, operator.S), initial_state.conv)
        if self._one_node_applies(initial_state, return_final_state, geometry_enabled, associative_decay_enabled):
            output_norm, output_proj = self.output_norm, self.output_proj
            result = host.mixer_train(
                hidden_states, heads, width, value_width, in_proj.weight, in_proj.bias, self.conv_weight,
                decay_proj.weight, gate_proj.weight, gate_proj.bias, self.associative_log_rate,
                self.associative_decay_bias, self.geometry_write_bias, output_norm.weight, output_norm.eps,
                output_proj.weight, output_proj.bias, valid_mask, reset_mask)
            if result is not None:
                return result
        conv_state = initial_state.conv if initial_state is not None else None
        (u, h, q, keys, values, log_decay, erase_raw, write_raw, geometry_write, output_gate,
         final_conv) = host.mixer_front(
            hidden_states, heads, width, value_width, in_proj.weight, in_proj.bias,
            self.conv_weight if self.config.use_short_conv else None, conv_state, valid_mask, reset_mask,
            return_final_state, inplace_state, decay_proj.weight, gate_proj.weight, gate_proj.bias,
            self.associative_log_rate, self.associative_decay_bias, self.geometry_write_bias, geometry_enabled,
            associative_decay_enabled)
        operator_initial = initial_state.operator if initial_state is not None else None
        if not masked:
            extra = {"_inplace_state": True} if inplace_state else {}   # the public signature is upstream's
            output, operator_state = solvedelta_native(
                u, h, q, keys, values, log_decay, erase_raw, write_raw, geometry_write,
                initial_state=operator_initial, return_final_state=return_final_state, **extra)
        else:
            output, operator_state = solvedelta_masked_native(
                u, h, q, keys, values, log_decay, erase_raw, write_raw, geometry_write,
                valid_mask=valid_mask, reset_mask=reset_mask,
                initial_state=operator_initial, return_final_state=return_final_state)
        result = self.output_norm.forward_linear(output, output_gate, self.output_proj)
        if not return_final_state:
            return result
        if operator_state is None:
            raise RuntimeError("operator did not return the requested final state")
        return result, SolveDeltaLayerState(operator_state, final_conv)


__all__ = ["RMSNormGated", "SolveDelta", "SolveDeltaLayerState"]

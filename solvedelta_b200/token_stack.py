"""One cached token, or a prompt, through a model's blocks in one native call.

A single-token step of a generation loop is a chain of short launches, so per-layer module
calls cost more than the kernels behind them; so does a prompt of up to a few thousand tokens.
:func:`token_stack` gives the native stack of a ``SolveDeltaModel`` (csrc/sd_host_glue.cpp): it
holds the model's own parameter tensors and is rebuilt when a module, a parameter object or an
epsilon has been replaced; a hook or a replaced ``forward`` anywhere in the blocks turns it off,
and the module path runs.  That path calls the blocks, the mixers, the MLPs and an MLP's two
projections as modules; the norms and a mixer's own projections it uses through their weights.
"""
from __future__ import annotations

import weakref
from typing import Optional

from torch import nn
from torch.nn.modules import module as module_globals

from . import _lib, model as mixer_module
from .model import RMSNormGated, SolveDelta

_STACKS: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()
_FUSED_DECODE_APPLIES = SolveDelta._fused_decode_applies
_OPERATOR = mixer_module.solvedelta_native


def _eps(norm: nn.RMSNorm) -> float:
    return norm.eps if norm.eps is not None else 1e-6


def _build(model, block_type, adapter_type, mlp_type):
    """The native stack of ``model``, or None when its blocks are not the ones it knows."""
    if model.norm.weight is None:
        return None
    stack = _lib.host().TokenStack(model.norm.weight, _eps(model.norm))
    watched = [(model, type(model)), (model.layers, nn.ModuleList), (model.norm, nn.RMSNorm)]
    for block in model.layers:
        if type(block) is not block_type or type(block.mixer) is not adapter_type or type(block.mlp) is not mlp_type:
            return None
        mixer, mlp = block.mixer.mixer, block.mlp
        if type(mixer) is not SolveDelta or not mixer.config.use_short_conv or mlp.hidden_act != "swish":
            return None
        watched += [(block, block_type), (block.mixer, adapter_type), (mixer, SolveDelta), (mlp, mlp_type),
                    (block.mixer_norm, nn.RMSNorm), (block.mlp_norm, nn.RMSNorm), (mixer.output_norm, RMSNormGated)]
        watched += [(linear, nn.Linear) for linear in (mixer.in_proj, mixer.decay_proj, mixer.output_gate_proj,
                                                       mixer.output_proj, mlp.gate_up_proj, mlp.down_proj)]
        if (any(type(m) is not t for m, t in watched) or mlp.gate_up_proj.bias is not None
                or mlp.down_proj.bias is not None or block.mixer_norm.weight is None or block.mlp_norm.weight is None):
            return None
        config = mixer.config
        stack.add_layer(
            block.mixer_norm.weight, _eps(block.mixer_norm), block.mlp_norm.weight, _eps(block.mlp_norm),
            config.num_heads, config.resolved_head_k_dim, config.resolved_head_v_dim,
            mixer.in_proj.weight, mixer.in_proj.bias, mixer.conv_weight, mixer.decay_proj.weight,
            mixer.output_gate_proj.weight, mixer.output_gate_proj.bias, mixer.associative_log_rate,
            mixer.associative_decay_bias, mixer.geometry_write_bias, mixer.output_norm.weight, mixer.output_norm.eps,
            mixer.output_proj.weight, mixer.output_proj.bias, mlp.gate_up_proj.weight, mlp.down_proj.weight)
    for module, _ in watched:
        for children in (module._modules, module._parameters):
            for name, child in children.items():
                stack.watch_same(children, name, child)
        if "eps" in module.__dict__:
            stack.watch_same(module.__dict__, "eps", module.__dict__["eps"])
        if module is not model:   # the model's own forward and hooks belong to its caller
            stack.watch_absent(module.__dict__, "forward")
            stack.watch_empty(module._forward_hooks)
            stack.watch_empty(module._forward_pre_hooks)
    stack.watch_empty(module_globals._global_forward_hooks)
    stack.watch_empty(module_globals._global_forward_pre_hooks)
    return stack


def token_stack(model, block_type, adapter_type, mlp_type) -> Optional[object]:
    """The native stack of ``model`` in its present form, or None when the module path has to run."""
    if SolveDelta._fused_decode_applies is not _FUSED_DECODE_APPLIES or mixer_module.solvedelta_native is not _OPERATOR:
        return None
    entry = _STACKS.get(model)
    if entry is not None and entry[0] == len(model.layers) and (entry[1] is None or entry[1].unchanged()):
        return entry[1]
    stack = _build(model, block_type, adapter_type, mlp_type)
    if stack is not None and not stack.unchanged():
        return None   # hooks: tried again on the next call
    _STACKS[model] = (len(model.layers), stack)
    return stack

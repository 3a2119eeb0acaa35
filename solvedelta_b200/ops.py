"""Operator entry points with the upstream names, signatures and errors.

Mirrors causallsso/ops/operator.py:13-55 (``solvedelta_native``) and
causallsso/ops/residual_frame/operator.py:154-304
(``solvedelta_residual_frame_native``): BF16 CUDA activations with unit
innermost stride and arbitrary outer strides, FP32 ``associative_log_decay``
and ``geometry_write`` ([H], [1,H] or [B,T,H]), FP32 continuation states
``SolveDeltaState(predictor=C [B,H,r,r], S [B,H,r,V])``.  One
``torch.autograd.Function`` covers the whole operator; ``None`` incoming
gradients are legal (``set_materialize_grads(False)``), gradients are returned
for the nine tensor operands and for both initial states.

PyTorch is used for device memory and the current stream only; all arithmetic
is in the CUDA library behind ``include/solvedelta_b200.h``.  There is no CPU
or eager fallback.
"""
from __future__ import annotations

import ctypes
from typing import NamedTuple, Optional, Tuple

import torch

from . import _lib
from .packing import PackedSegments


class SolveDeltaState(NamedTuple):
    """Continuation state; same field names as causallsso/reference.py:14-16."""

    predictor: torch.Tensor
    S: torch.Tensor


def solvedelta_zero_state(batch: int, heads: int, rank: int, value_dim: int, *,
                          dtype: torch.dtype, device: torch.device) -> SolveDeltaState:
    return SolveDeltaState(
        predictor=torch.zeros(batch, heads, rank, rank, dtype=dtype, device=device),
        S=torch.zeros(batch, heads, rank, value_dim, dtype=dtype, device=device),
    )


def _operand(t: torch.Tensor) -> _lib.Operand:
    """[B,T,H,w] tensor (any outer strides, unit inner stride) -> C operand."""
    sb, st, sh = t.stride(0), t.stride(1), t.stride(2)
    return _lib.Operand(t.data_ptr(), sb, st, sh)


def _gamma_operand(t: torch.Tensor) -> _lib.Operand:
    return _lib.Operand(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


def _shape(u: torch.Tensor, value_dim: int) -> _lib.Shape:
    B, T, H, r = u.shape
    return _lib.Shape(B, T, H, r, value_dim)


def _stream_ptr(device) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def _buffer(nbytes: int, device) -> torch.Tensor:
    return torch.empty(max(int(nbytes), 16), dtype=torch.uint8, device=device)


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _fill_operands(args, tensors):
    names = ("u", "h", "q", "keys", "values", "erase_raw", "write_raw", "log_decay")
    u, h, q, k, v, ld, er, wr, gam = tensors
    for name, t in zip(names, (u, h, q, k, v, er, wr, ld)):
        setattr(args, name, _operand(t))
    args.gamma = _gamma_operand(gam)


class _OjaResidual(torch.autograd.Function):
    """forward(target, source, beta[B,T,H], log_decay, query, C0|None) -> (frame_action, update, C_T)."""

    @staticmethod
    def forward(ctx, target, source, beta, log_decay, query, C0):
        lib = _lib.load()
        device = target.device
        B, T, H, r = target.shape
        shape = _shape(target, r)
        with torch.cuda.device(device):
            action = torch.empty(B, T, H, r, dtype=torch.bfloat16, device=device)
            update = torch.empty(B, T, H, r, dtype=torch.bfloat16, device=device)
            C_T = torch.empty(B, H, r, r, dtype=torch.float32, device=device)
            saved = _buffer(lib.sd_saved_bytes(ctypes.byref(shape)), device)
            scratch = _buffer(lib.sd_forward_scratch_bytes(ctypes.byref(shape)), device)
            C0c = None if C0 is None else C0.contiguous()
            args = _lib.PredictorForwardArgs()
            args.shape = shape
            args.target, args.source, args.query = _operand(target), _operand(source), _operand(query)
            args.beta, args.log_decay = _gamma_operand(beta), _operand(log_decay)
            args.C0 = _ptr(C0c)
            args.frame_action, args.update, args.C_T = action.data_ptr(), update.data_ptr(), C_T.data_ptr()
            args.saved, args.saved_bytes = saved.data_ptr(), saved.numel()
            args.scratch, args.scratch_bytes = scratch.data_ptr(), scratch.numel()
            _lib.check(lib.sd_predictor_forward(ctypes.byref(args), _stream_ptr(device)))
        ctx.set_materialize_grads(False)
        ctx.has_state = C0 is not None
        ctx.save_for_backward(target, source, beta, log_decay, query, saved, action)
        return action, update, C_T

    @staticmethod
    def backward(ctx, d_action, d_update, dC_T):
        lib = _lib.load()
        target, source, beta, log_decay, query, saved, action = ctx.saved_tensors
        device = target.device
        B, T, H, r = target.shape
        shape = _shape(target, r)
        with torch.cuda.device(device):
            d_action = None if d_action is None else d_action.to(torch.bfloat16).contiguous()
            d_update = None if d_update is None else d_update.to(torch.bfloat16).contiguous()
            dC_T = None if dC_T is None else dC_T.float().contiguous()
            bf = dict(dtype=torch.bfloat16, device=device)
            dtarget, dsource, dquery = (torch.empty(B, T, H, r, **bf) for _ in range(3))
            dld = torch.empty(B, T, H, r, dtype=torch.float32, device=device)
            dbeta = torch.empty(B, T, H, dtype=torch.float32, device=device)
            dC0 = torch.empty(B, H, r, r, dtype=torch.float32, device=device)
            scratch = _buffer(lib.sd_backward_scratch_bytes(ctypes.byref(shape)), device)
            args = _lib.PredictorBackwardArgs()
            args.shape = shape
            args.target, args.source, args.query = _operand(target), _operand(source), _operand(query)
            args.beta, args.log_decay = _gamma_operand(beta), _operand(log_decay)
            args.frame_action = action.data_ptr()
            args.d_frame_action, args.d_update, args.dC_T = _ptr(d_action), _ptr(d_update), _ptr(dC_T)
            args.saved, args.saved_bytes = saved.data_ptr(), saved.numel()
            args.scratch, args.scratch_bytes = scratch.data_ptr(), scratch.numel()
            args.dtarget, args.dsource, args.dquery = dtarget.data_ptr(), dsource.data_ptr(), dquery.data_ptr()
            args.dbeta, args.dlog_decay, args.dC0 = dbeta.data_ptr(), dld.data_ptr(), dC0.data_ptr()
            _lib.check(lib.sd_predictor_backward(ctypes.byref(args), _stream_ptr(device)))
        return dtarget, dsource, dbeta, dld, dquery, dC0 if ctx.has_state else None


def oja_residual(target: torch.Tensor, source: torch.Tensor, beta: torch.Tensor, log_decay: torch.Tensor,
                 query: torch.Tensor, initial_state: Optional[torch.Tensor], *, chunk_size: int = 32,
                 output_final_state: bool = True):
    """The predictor sub-owner of causallsso/ops/residual_frame/predictor.py:285-305, same arguments and
    returns: ``(frame_action, update, final_state)`` with ``frame_action = C_t^T query`` accumulated through
    the sequence (what the operator adds to the normalised key to form the primal address), ``update``
    the residual step Delta of the NLMS solve, and ``final_state`` the predictor state ``C`` ``[B,H,r,r]`` (None
    unless requested).  ``source`` and ``query`` are used as given (upstream passes the L2-normalised panels)
    and receive the gradients of the rows themselves.  ``chunk_size`` is accepted for signature compatibility;
    the kernels work on 64-token chunks and the result does not depend on it."""
    for name, t in (("target", target), ("source", source), ("query", query)):
        if t.device.type != "cuda" or t.dtype != torch.bfloat16:
            raise TypeError(f"{name} must be a BF16 CUDA tensor")
        if t.ndim != 4 or t.shape != target.shape:
            raise ValueError(f"{name} must have shape [B,T,H,r]")
        if t.stride(-1) != 1:
            raise ValueError("native vector operands require unit innermost stride")
    batch, length, heads, rank = target.shape
    if rank > 128:
        raise ValueError("head width above 128 is not supported")
    if log_decay.dtype != torch.float32 or log_decay.shape != target.shape:
        raise TypeError("log_decay must be FP32 [B,T,H,r]")
    if beta.dtype != torch.float32 or beta.shape != (batch, length, heads):
        raise TypeError("beta must be FP32 [B,T,H]")
    if initial_state is not None and (initial_state.dtype != torch.float32
                                      or initial_state.shape != (batch, heads, rank, rank)):
        raise ValueError("initial_state must be FP32 [B,H,r,r]")
    if log_decay.stride(-1) != 1:
        log_decay = log_decay.contiguous()
    if length == 0:
        empty = target.new_zeros(target.shape)
        final = None
        if output_final_state:
            final = (initial_state.clone() if initial_state is not None
                     else torch.zeros(batch, heads, rank, rank, dtype=torch.float32, device=target.device))
        return empty, empty.clone(), final
    action, update, final = _OjaResidual.apply(target, source, beta, log_decay, query, initial_state)
    return action, update, (final if output_final_state else None)


def solvedelta_residual_frame_native(
    u: torch.Tensor,
    h: torch.Tensor,
    q: torch.Tensor,
    keys: torch.Tensor,
    values: torch.Tensor,
    associative_log_decay: torch.Tensor,
    erase_raw: torch.Tensor,
    write_raw: torch.Tensor,
    geometry_write: torch.Tensor,
    *,
    initial_state: Optional[SolveDeltaState] = None,
    return_final_state: bool = True,
    _valid_mask: Optional[torch.Tensor] = None,
    _reset_mask: Optional[torch.Tensor] = None,
    _inplace_state: bool = False,
) -> Tuple[torch.Tensor, Optional[SolveDeltaState]]:
    """Dense BF16 path from raw gate logits.

    Same checks, in the same order and with the same exception types, as
    causallsso/ops/residual_frame/operator.py:169-196 and :247-262.  Any
    sequence length is accepted: a ragged last chunk is completed inside the
    kernels with neutral tokens (the upstream path pads with zero tokens,
    residual_frame/operator.py:218-245, which is the same arithmetic).
    """
    C0, S0 = (None, None) if initial_state is None else initial_state
    y, C, S = _lib.host().residual_frame(
        u, h, q, keys, values, associative_log_decay, erase_raw, write_raw, geometry_write, C0, S0,
        return_final_state, _valid_mask, _reset_mask, _inplace_state)
    return y, (SolveDeltaState(C, S) if return_final_state else None)


def solvedelta_native(
    u: torch.Tensor,
    h: torch.Tensor,
    q: torch.Tensor,
    keys: torch.Tensor,
    values: torch.Tensor,
    associative_log_decay: torch.Tensor,
    erase_raw: torch.Tensor,
    write_raw: torch.Tensor,
    geometry_write: torch.Tensor,
    *,
    initial_state: Optional[SolveDeltaState] = None,
    return_final_state: bool = False,
    _inplace_state: bool = False,
) -> Tuple[torch.Tensor, Optional[SolveDeltaState]]:
    """Execute dense K=1 SolveDelta from raw fused-projection views.

    Same contract as causallsso/ops/operator.py:13-55.  ``_inplace_state`` (no upstream counterpart) lets a
    single-token no-grad step update the tensors of ``initial_state`` in place and return them, for a cache
    that owns its state; by default the step works on copies, as upstream returns new tensors.
    """
    C0, S0 = (None, None) if initial_state is None else initial_state
    y, C, S = _lib.host().dense(
        u, h, q, keys, values, associative_log_decay, erase_raw, write_raw, geometry_write, C0, S0,
        return_final_state, _inplace_state)
    return y, (SolveDeltaState(C, S) if return_final_state else None)


def solvedelta_segmented_native(
    u: torch.Tensor,
    h: torch.Tensor,
    q: torch.Tensor,
    keys: torch.Tensor,
    values: torch.Tensor,
    associative_log_decay: torch.Tensor,
    erase_raw: torch.Tensor,
    write_raw: torch.Tensor,
    geometry_write: torch.Tensor,
    plan: PackedSegments,
    *,
    initial_state: Optional[SolveDeltaState] = None,
    return_final_state: bool = False,
) -> Tuple[torch.Tensor, Optional[SolveDeltaState]]:
    """Masked / reset batches, same contract as causallsso/ops/operator.py:96-193.

    Invalid tokens produce zero output and leave the state untouched, a reset token
    starts from the zero state, the returned state of a batch row is the one after its
    last valid token (its initial state if it has none).  Upstream gathers the valid
    tokens into a padded batch of reset-free segments and scatters the result back;
    here the kernels read the two token masks of ``plan`` themselves (a masked token is
    a neutral token, a reset is extra forgetting that no decay-weighted term survives),
    so the operands stay where they are and the call does no host work.
    """
    batch, length, heads, rank = u.shape
    if (plan.batch, plan.length) != (batch, length):
        raise ValueError("packed segment plan does not match the operator input")
    if plan.valid_mask is None or plan.reset_mask is None:
        raise ValueError("the segment plan carries no token masks (build it with build_packed_segments)")
    return solvedelta_residual_frame_native(
        u, h, q, keys, values, associative_log_decay, erase_raw, write_raw, geometry_write,
        initial_state=initial_state, return_final_state=return_final_state,
        _valid_mask=plan.valid_mask, _reset_mask=plan.reset_mask)


def solvedelta_masked_native(
    u: torch.Tensor,
    h: torch.Tensor,
    q: torch.Tensor,
    keys: torch.Tensor,
    values: torch.Tensor,
    associative_log_decay: torch.Tensor,
    erase_raw: torch.Tensor,
    write_raw: torch.Tensor,
    geometry_write: torch.Tensor,
    *,
    valid_mask: Optional[torch.Tensor] = None,
    reset_mask: Optional[torch.Tensor] = None,
    initial_state: Optional[SolveDeltaState] = None,
    return_final_state: bool = False,
) -> Tuple[torch.Tensor, Optional[SolveDeltaState]]:
    """``solvedelta_segmented_native`` without the plan: the two bool ``[B,T]`` token masks of the
    token loop (causallsso/reference.py:157-164,216-226) go straight to the kernels.  No upstream
    counterpart (upstream needs the plan to gather segments); it exists so that a caller with
    device-side masks never synchronises with the host."""
    batch, length = u.shape[:2]
    for name, mask in (("valid_mask", valid_mask), ("reset_mask", reset_mask)):
        if mask is None:
            continue
        if mask.dtype != torch.bool or mask.shape != (batch, length):
            raise ValueError(f"{name} must be bool [B,T]")
        if mask.device != u.device:
            raise ValueError("masks must share the operand device")
    return solvedelta_residual_frame_native(
        u, h, q, keys, values, associative_log_decay, erase_raw, write_raw, geometry_write,
        initial_state=initial_state, return_final_state=return_final_state,
        _valid_mask=valid_mask, _reset_mask=reset_mask)


__all__ = [
    "SolveDeltaState",
    "oja_residual",
    "solvedelta_native",
    "solvedelta_masked_native",
    "solvedelta_segmented_native",
    "solvedelta_residual_frame_native",
    "solvedelta_zero_state",
]

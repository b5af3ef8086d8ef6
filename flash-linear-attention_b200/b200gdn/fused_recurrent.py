"""fused_recurrent_gated_delta_rule with the reference's signature
(fla/ops/gated_delta_rule/fused_recurrent.py:309-475): the decode / short-prefill step, forward only."""
from __future__ import annotations

import warnings
from typing import Optional

import torch

from . import _lib
from .recorded import seen_by_trace, untraced


class FusedRecurrentFunction(torch.autograd.Function):
    """The node of a call whose inputs ask for gradients, or that a trace records: the forward pass runs, the backward pass
    says that it does not exist (as in the reference, fla/ops/gated_delta_rule/fused_recurrent.py:299-306)."""

    @staticmethod
    def forward(ctx, q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state, flags, cu_seqlens,
                inplace_state, state_indices=None):
        with untraced():
            out = _lib.host().recurrent(q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state, flags,
                                        cu_seqlens, inplace_state, state_indices)
        if out is NotImplemented:
            raise _lib.B200GDNError('fused_recurrent_gated_delta_rule: tensors of unexpected shapes or devices')
        if out[1] is not None and out[1] is initial_state:
            ctx.mark_dirty(initial_state)   # updated in place and returned
            return out
        return seen_by_trace(out)

    @staticmethod
    def backward(ctx, do, dht):
        raise NotImplementedError(
            "Backward pass is not implemented for the fused recurrent path (as in the reference, "
            "fla/ops/gated_delta_rule/fused_recurrent.py:299-306); use chunk_gated_delta_rule for training.")


def fused_recurrent_gated_delta_rule(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    g: Optional[torch.Tensor] = None,
    gk: Optional[torch.Tensor] = None,
    gv: Optional[torch.Tensor] = None,
    beta: Optional[torch.Tensor] = None,
    scale: Optional[float] = None,
    initial_state: Optional[torch.Tensor] = None,
    output_final_state: bool = False,
    use_qk_l2norm_in_kernel: bool = False,
    use_gate_in_kernel: bool = False,
    A_log: Optional[torch.Tensor] = None,
    dt_bias: Optional[torch.Tensor] = None,
    use_beta_sigmoid_in_kernel: bool = False,
    allow_neg_eigval: bool = False,
    state_v_first: bool = False,
    cu_seqlens: Optional[torch.Tensor] = None,
    **kwargs,
):
    r"""Recurrent gated delta rule, same contract as the reference's ``fused_recurrent_gated_delta_rule``.

    q, k ``[B,T,H,K]``; v ``[B,T,HV,V]``; g, beta ``[B,T,HV]``; ``initial_state [N,HV,K,V]``
    (``[N,HV,V,K]`` with ``state_v_first``).  Per-dimension decays ``gk`` / ``gv`` and per-channel beta
    ``[B,T,HV,V]`` belong to other operators of the reference and are rejected.  The extra keyword
    ``inplace_state=True`` writes the final state over ``initial_state`` (fp32, contiguous) instead of
    allocating a new tensor.  The extra keyword ``state_indices [N]`` (no counterpart in the reference) makes
    ``initial_state`` a pool of state slots ``[n_slots,HV,K,V]``: sequence ``n`` reads and updates slot
    ``state_indices[n]`` in place (distinct slots per call), and the pool is returned as the final state.  An index
    outside ``[0, n_slots)`` (a serving engine's ``-1`` padding) marks a padding sequence: its slot is left untouched
    and its output row is meaningless.
    """
    inplace_state, state_indices = False, None
    if kwargs:
        if 'transpose_state_layout' in kwargs:
            if state_v_first:
                raise ValueError("Cannot pass both `state_v_first` and the deprecated `transpose_state_layout`.")
            warnings.warn("`transpose_state_layout` is deprecated and renamed to `state_v_first`.",
                          DeprecationWarning, stacklevel=2)
            state_v_first = kwargs.pop('transpose_state_layout')
        inplace_state = bool(kwargs.pop('inplace_state', False))
        state_indices = kwargs.pop('state_indices', None)
    if not use_gate_in_kernel:
        A_log = dt_bias = None
    flags = ((_lib.REC_L2NORM if use_qk_l2norm_in_kernel else 0) | (_lib.REC_GATE if use_gate_in_kernel else 0)
             | (_lib.REC_BETA_SIGMOID if use_beta_sigmoid_in_kernel else 0) | (_lib.REC_NEG_EIGVAL if allow_neg_eigval else 0)
             | (_lib.REC_STATE_V_FIRST if state_v_first else 0))
    if gk is None and gv is None:
        out = (_lib._host or _lib.host()).recurrent(q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state,
                                                    flags, cu_seqlens, inplace_state, state_indices)
        if out is not NotImplemented:
            return out
    # not served by the direct call: say what is wrong, or record the node that has no backward pass (as a trace does, which
    # sees nothing of a native call)
    if gk is not None or gv is not None:
        raise NotImplementedError('per-dimension decays gk / gv are not part of the gated delta rule path')
    if cu_seqlens is not None:
        if q.shape[0] != 1:
            raise ValueError(
                f"The batch size is expected to be 1 rather than {q.shape[0]} when using `cu_seqlens`."
                f"Please flatten variable-length inputs before processing.")
        if state_indices is None and initial_state is not None and initial_state.shape[0] != len(cu_seqlens) - 1:
            raise ValueError(
                f"The number of initial states is expected to be equal to the number of input sequences, "
                f"i.e., {len(cu_seqlens) - 1} rather than {initial_state.shape[0]}.")
    if scale is None:
        scale = k.shape[-1] ** -0.5
    if beta is None:
        beta = torch.ones_like(q[..., 0]).repeat_interleave(v.shape[2] // q.shape[2], dim=-1)
    if beta.ndim != 3:
        raise NotImplementedError('per-channel beta [B,T,HV,V] is not part of the gated delta rule path')
    if use_gate_in_kernel:
        if A_log is None:
            raise ValueError("`A_log` must be provided when `use_gate_in_kernel=True`.")
        if g is None:
            raise ValueError("`g` (raw pre-activation) must be provided when `use_gate_in_kernel=True`.")
    if allow_neg_eigval and not use_beta_sigmoid_in_kernel:
        raise ValueError("`allow_neg_eigval=True` requires `use_beta_sigmoid_in_kernel=True`.")
    if not q.is_cuda:
        raise _lib.B200GDNError('fused_recurrent_gated_delta_rule runs on a CUDA device only (no CPU path)')
    n_seq = q.shape[0] if cu_seqlens is None else cu_seqlens.numel() - 1
    if state_indices is not None:
        # a pool of state slots addressed per sequence; the update happens in the pool itself
        if initial_state is None or initial_state.dtype != torch.float32 or not initial_state.is_contiguous():
            raise ValueError("`state_indices` needs `initial_state` to be the fp32 contiguous pool of state slots.")
        if state_indices.numel() != n_seq:
            raise ValueError(f"`state_indices` must have one entry per sequence ({n_seq}), got {state_indices.numel()}.")
    return FusedRecurrentFunction.apply(q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state,
                                        flags, cu_seqlens, inplace_state, state_indices)


fused_recurrent_gdn = fused_recurrent_gated_delta_rule

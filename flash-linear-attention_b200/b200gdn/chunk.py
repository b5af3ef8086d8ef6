"""chunk_gated_delta_rule with the reference's signature (fla/ops/gated_delta_rule/chunk.py:395-593),
computed by the sm_100a kernels of libb200gdn.so through an autograd node of the native host path (csrc/host.cpp).

PyTorch is used for device memory, the current stream and autograd bookkeeping only; every stage of
the reference's pipeline (chunk.py:33-250) runs inside the library.
"""
from __future__ import annotations

import warnings
from typing import Optional

import torch

from . import _lib
from .index import native_plan
from .recorded import RecordedCall, recorded

_SUPPORTED_HEAD_DIMS = ((64, 64), (128, 128))


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


_DTYPE_CODE = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


class LayerOptionsFunction(torch.autograd.Function):
    """The three options fla.layers.GatedDeltaNet turns on (fla/layers/gated_deltanet.py:309-325), computed by
    b200gdn_prep_fwd / b200gdn_prep_bwd: q, k L2-normalised to bf16 (fla/modules/l2norm.py:84-144), the gate
    ``-exp(A_log) softplus(g + dt_bias)`` (fla/ops/gated_delta_rule/gate.py:63-158, with dA_log and ddt_bias) and
    ``beta = s sigmoid(beta)`` (fla/ops/common/gate.py:18-50).  Returns what the chunk kernels consume."""

    @staticmethod
    def forward(ctx, q, k, g, beta, A_log, dt_bias, flags):
        dev = q.device
        with torch.cuda.device(dev):
            a = _lib.PrepArgs()
            a.rows, a.H, a.K = q.shape[0] * q.shape[1], q.shape[2], q.shape[3]
            a.HV = g.shape[-1]
            a.flags = flags
            qn, kn, g_out, beta_out = q, k, g, beta
            rstd_q = rstd_k = None
            if flags & _lib.PREP_L2NORM:
                if q.dtype not in _DTYPE_CODE or k.dtype != q.dtype:
                    raise _lib.B200GDNError(f'q/k dtypes {q.dtype}/{k.dtype} are not supported by the L2-norm option')
                q, k = q.contiguous(), k.contiguous()
                a.qk_dtype = _DTYPE_CODE[q.dtype]
                qn, kn = (torch.empty(q.shape, dtype=torch.bfloat16, device=dev) for _ in range(2))
                rstd_q, rstd_k = (torch.empty(q.shape[:-1], dtype=torch.float32, device=dev) for _ in range(2))
                a.q, a.k, a.qn, a.kn = q.data_ptr(), k.data_ptr(), qn.data_ptr(), kn.data_ptr()
                a.rstd_q, a.rstd_k = rstd_q.data_ptr(), rstd_k.data_ptr()
            gb_in = (g.dtype if flags & _lib.PREP_GATE else beta.dtype)
            if (flags & _lib.PREP_GATE) and (flags & _lib.PREP_BETA_SIGMOID) and g.dtype != beta.dtype:
                gb_in = torch.float32
            if gb_in not in _DTYPE_CODE:
                gb_in = torch.float32
            a.gb_dtype = _DTYPE_CODE[gb_in]
            if flags & _lib.PREP_GATE:
                g = g.to(gb_in).contiguous()
                A_log_f = A_log.detach().float().contiguous()
                bias_f = None if dt_bias is None else dt_bias.detach().float().contiguous()
                g_out = torch.empty(g.shape, dtype=torch.float32, device=dev)
                a.g, a.A_log, a.dt_bias, a.g_out = g.data_ptr(), A_log_f.data_ptr(), _lib.ptr(bias_f), g_out.data_ptr()
            else:
                A_log_f = bias_f = None
            if flags & _lib.PREP_BETA_SIGMOID:
                beta = beta.to(gb_in).contiguous()
                beta_out = torch.empty(beta.shape, dtype=torch.float32, device=dev)
                a.beta, a.beta_out = beta.data_ptr(), beta_out.data_ptr()
            _lib.call('b200gdn_prep_fwd', a, _stream(q))
        ctx.flags, ctx.gb_in = flags, gb_in
        ctx.in_dtypes = (g.dtype, beta.dtype)
        ctx.has_bias = dt_bias is not None
        ctx.param_dtypes = (None if A_log is None else A_log.dtype, None if dt_bias is None else dt_bias.dtype)
        ctx.save_for_backward(q, k, rstd_q, rstd_k, g, beta, A_log_f, bias_f)
        return qn, kn, g_out, beta_out

    @staticmethod
    def backward(ctx, dqn, dkn, dg, dbeta):
        q, k, rstd_q, rstd_k, g, beta, A_log_f, bias_f = ctx.saved_tensors
        flags = ctx.flags
        dev = q.device
        dq, dk, dg_raw, dbeta_raw, dA_log, ddt_bias = dqn, dkn, dg, dbeta, None, None
        with torch.cuda.device(dev):
            a = _lib.PrepArgs()
            a.rows, a.H, a.K = q.shape[0] * q.shape[1], q.shape[2], q.shape[3]
            a.HV = g.shape[-1]
            a.flags = 0
            keep = []
            if (flags & _lib.PREP_L2NORM) and dqn is not None and dkn is not None:
                a.flags |= _lib.PREP_L2NORM
                a.qk_dtype = _DTYPE_CODE[q.dtype]
                dqn, dkn = dqn.to(torch.bfloat16).contiguous(), dkn.to(torch.bfloat16).contiguous()
                dq, dk = torch.empty_like(q), torch.empty_like(k)
                a.q, a.k, a.rstd_q, a.rstd_k = q.data_ptr(), k.data_ptr(), rstd_q.data_ptr(), rstd_k.data_ptr()
                a.dqn, a.dkn, a.dq, a.dk = dqn.data_ptr(), dkn.data_ptr(), dq.data_ptr(), dk.data_ptr()
            a.gb_dtype = _DTYPE_CODE[ctx.gb_in]
            if (flags & _lib.PREP_GATE) and dg is not None:
                a.flags |= _lib.PREP_GATE
                dg = dg.float().contiguous()
                dg_raw = torch.empty(g.shape, dtype=ctx.gb_in, device=dev)
                n_part = (a.rows + _lib.PREP_PART_ROWS - 1) // _lib.PREP_PART_ROWS
                partials = torch.empty(n_part, 2, a.HV, dtype=torch.float32, device=dev)
                dA_log = torch.empty(a.HV, dtype=torch.float32, device=dev)
                ddt_bias = torch.empty(a.HV, dtype=torch.float32, device=dev) if ctx.has_bias else None
                a.g, a.A_log, a.dt_bias = g.data_ptr(), A_log_f.data_ptr(), _lib.ptr(bias_f)
                a.dg, a.dg_raw, a.partials = dg.data_ptr(), dg_raw.data_ptr(), partials.data_ptr()
                a.dA_log, a.ddt_bias = dA_log.data_ptr(), _lib.ptr(ddt_bias)
                keep += [partials]
            if (flags & _lib.PREP_BETA_SIGMOID) and dbeta is not None:
                a.flags |= _lib.PREP_BETA_SIGMOID | (flags & _lib.PREP_NEG_EIGVAL)
                dbeta = dbeta.float().contiguous()
                dbeta_raw = torch.empty(beta.shape, dtype=ctx.gb_in, device=dev)
                a.beta, a.dbeta, a.dbeta_raw = beta.data_ptr(), dbeta.data_ptr(), dbeta_raw.data_ptr()
            if a.flags:
                _lib.call('b200gdn_prep_bwd', a, _stream(q))
        g_dtype, beta_dtype = ctx.in_dtypes
        if dg_raw is not None and dg_raw.dtype != g_dtype:
            dg_raw = dg_raw.to(g_dtype)
        if dbeta_raw is not None and dbeta_raw.dtype != beta_dtype:
            dbeta_raw = dbeta_raw.to(beta_dtype)
        if dA_log is not None:
            dA_log = dA_log.to(ctx.param_dtypes[0])
        if ddt_bias is not None:
            ddt_bias = ddt_bias.to(ctx.param_dtypes[1])
        return dq, dk, dg_raw, dbeta_raw, dA_log, ddt_bias, None


def new_chunk_args(q, k, v, scale, tables) -> _lib.ChunkArgs:
    chunk_meta, seq_meta, (n_chunks, n_seq) = tables
    a = _lib.ChunkArgs()
    a.rows = q.shape[0] * q.shape[1]
    a.H, a.HV, a.K, a.V = q.shape[2], v.shape[2], q.shape[3], v.shape[3]
    a.n_seq, a.n_chunks = n_seq, n_chunks
    a.scale = float(scale)
    a.stage_mask = 0
    a.chunk_meta, a.seq_meta = chunk_meta.data_ptr(), seq_meta.data_ptr()
    a.q, a.k, a.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    return a


def carve(dev, zero, *specs):
    """One device allocation cut into tensors: ``specs`` are (shape, dtype) pairs, every tensor starts on a 256-byte
    boundary.  A forward + backward pass needs about twenty intermediates; one allocation per pass instead of one per
    tensor keeps the host-side cost of a step small.  ``zero`` fills the allocation with zeros (needed when the packed
    buffer has rows that belong to no sequence: the kernels never write them)."""
    offs, total = [], 0
    for shape, dtype in specs:
        n = 1
        for x in shape:
            n *= int(x)
        offs.append(total)
        total += (n * dtype.itemsize + 255) // 256 * 256
    buf = (torch.zeros if zero else torch.empty)(max(total, 256), dtype=torch.uint8, device=dev)
    out = []
    for (shape, dtype), off in zip(specs, offs):
        n = 1
        for x in shape:
            n *= int(x)
        nbytes = n * dtype.itemsize
        out.append(buf[off:off + nbytes].view(dtype).view(*shape))
    return out


def prefix_chains(plan, M, h, x0, out, K, V, reverse: bool, stream: int, last=None, identity: bool = False) -> None:
    """b200gdn_cp_prefix over the chains of a split plan: the start state (reverse: the end gradient) of every piece."""
    a = _lib.PrefixArgs()
    a.HV, a.K, a.V = M.shape[1], K, V
    a.n_chains, a.reverse, a.identity = plan.n_chains, int(reverse), int(identity)
    a.table, a.M, a.h, a.x0 = plan.chains.data_ptr(), M.data_ptr(), _lib.ptr(h), _lib.ptr(x0)
    a.out, a.last = _lib.ptr(out), _lib.ptr(last)
    _lib.call('b200gdn_cp_prefix', a, stream)


def _native_chunk(q, k, v, g, beta, initial_state, A_log, dt_bias, scale, output_final_state, options, cu_seqlens, cu_seqlens_cpu):
    plan = native_plan(q.shape[0], q.shape[1], cu_seqlens, cu_seqlens_cpu, q.device, v.shape[2], v.shape[3] // 64)
    return _lib.host().chunk(q, k, v, g, beta, initial_state, A_log, dt_bias, scale, output_final_state, options, plan)


def chunk_gated_delta_rule(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    g: torch.Tensor,
    beta: torch.Tensor,
    scale: Optional[float] = None,
    initial_state: Optional[torch.Tensor] = None,
    output_final_state: bool = False,
    use_qk_l2norm_in_kernel: bool = False,
    use_beta_sigmoid_in_kernel: bool = False,
    allow_neg_eigval: bool = False,
    state_v_first: bool = False,
    cu_seqlens: Optional[torch.Tensor] = None,
    cu_seqlens_cpu: Optional[torch.Tensor] = None,
    chunk_indices: Optional[torch.Tensor] = None,
    cp_context=None,
    **kwargs,
):
    r"""Chunked gated delta rule, same contract as the reference's ``chunk_gated_delta_rule``
    (fla/ops/gated_delta_rule/chunk.py:395-593).

    q, k ``[B,T,H,K]``; v ``[B,T,HV,V]`` (``HV % H == 0``: each q/k head serves ``HV/H`` value heads);
    g, beta ``[B,T,HV]``; ``initial_state [N,HV,K,V]`` (``[N,HV,V,K]`` with ``state_v_first``);
    ``cu_seqlens [N+1]`` for packed sequences (then ``B == 1``).  Returns ``(o [B,T,HV,V] in q.dtype,
    final_state fp32 or None)``.  Keyword options ``use_gate_in_kernel``, ``A_log``, ``dt_bias``,
    ``chunk_size`` (16/32/64 accepted; the result does not depend on it and 64 is always used) and the
    deprecated ``transpose_state_layout`` are honoured; ``head_first`` raises as in the reference.
    ``chunk_indices`` is accepted and ignored (the chunk tables are rebuilt from ``cu_seqlens``).

    Precision: the tensor-core kernels compute on bf16 q, k, v (fp32 accumulation, fp32 gates and states).  fp16 /
    fp32 q, k, v are accepted, ROUNDED TO BF16 on entry, and ``o`` and the gradients are cast back to the caller's
    dtypes: the result has bf16 accuracy (the reference's own fp32 test uses the bf16-level tolerance 0.005,
    tests/ops/test_gdn.py:203-278).  Callers that need fp32 arithmetic use the reference's Triton path:
    ``B200GDNBackend``'s verifier declines non-bf16 inputs so that the dispatcher falls through to it.
    A packed buffer may have padding rows before ``cu_seqlens[0]`` or after ``cu_seqlens[-1]``; their outputs and
    gradients are zero, and their q / k / v / do values must be finite.
    """
    use_gate_in_kernel, A_log, dt_bias = False, None, None
    if kwargs:
        if 'transpose_state_layout' in kwargs:
            if state_v_first:
                raise ValueError("Cannot pass both `state_v_first` and the deprecated `transpose_state_layout`.")
            warnings.warn("`transpose_state_layout` is deprecated and renamed to `state_v_first`.",
                          DeprecationWarning, stacklevel=2)
            state_v_first = kwargs.pop('transpose_state_layout')
        use_gate_in_kernel = kwargs.get('use_gate_in_kernel', False)
        A_log = kwargs.get('A_log')
        dt_bias = kwargs.get('dt_bias')
    (B, T, H, K), (HV, V) = q.shape, v.shape[2:]
    if H != k.shape[2]:
        raise ValueError(
            f"q and k must have the same number of heads, "
            f"but got q.shape[2]={q.shape[2]} and k.shape[2]={k.shape[2]}")
    if HV % H != 0:
        raise ValueError(
            f"For GVA, num_v_heads (HV={HV}) must be evenly divisible by "
            f"num_heads (H={H}), but got HV % H = {HV % H}")
    if kwargs:
        if 'head_first' in kwargs:
            raise DeprecationWarning("head_first has been removed. Inputs must be in `[B, T, H, ...]` format.")
        chunk_size = kwargs.pop('chunk_size', 64)
        if chunk_size not in (16, 32, 64):
            raise ValueError(f"`chunk_size` must be 16, 32, or 64 for Gated Delta Rule, got {chunk_size}.")
    if cp_context is not None:
        assert initial_state is None, "Initial state is not supported for CP"
        assert output_final_state is False, "Output final state is not supported for CP"
        assert cp_context.cu_seqlens is not None, "cu_seqlens is required for CP"
        cu_seqlens = cp_context.cu_seqlens
        if cp_context.cu_seqlens_cpu is not None:
            cu_seqlens_cpu = cp_context.cu_seqlens_cpu
    if cu_seqlens is not None:
        if B != 1:
            raise ValueError(
                f"The batch size is expected to be 1 rather than {q.shape[0]} when using `cu_seqlens`."
                f"Please flatten variable-length inputs before processing.")
        if initial_state is not None and initial_state.shape[0] != len(cu_seqlens) - 1:
            raise ValueError(
                f"The number of initial states is expected to be equal to the number of input sequences, "
                f"i.e., {len(cu_seqlens) - 1} rather than {initial_state.shape[0]}.")
    if use_gate_in_kernel:
        assert A_log is not None, "A_log must be provided when use_gate_in_kernel=True."
    if allow_neg_eigval and not use_beta_sigmoid_in_kernel:
        raise ValueError("`allow_neg_eigval=True` requires `use_beta_sigmoid_in_kernel=True`.")
    if scale is None:
        scale = K ** -0.5
    if not q.is_cuda:
        raise _lib.B200GDNError('chunk_gated_delta_rule runs on a CUDA device only (no CPU path)')
    if (K, V) not in _SUPPORTED_HEAD_DIMS:
        raise _lib.B200GDNError(f'head dimensions K={q.shape[-1]}, V={v.shape[-1]} are not built; '
                                f'supported: {_SUPPORTED_HEAD_DIMS}')

    # The three options the layer turns on (fla/layers/gated_deltanet.py:309-325).
    flags = ((_lib.PREP_L2NORM if use_qk_l2norm_in_kernel else 0) | (_lib.PREP_GATE if use_gate_in_kernel else 0)
             | (_lib.PREP_BETA_SIGMOID if use_beta_sigmoid_in_kernel else 0) | (_lib.PREP_NEG_EIGVAL if allow_neg_eigval else 0))
    if use_gate_in_kernel and A_log.numel() != HV:
        raise ValueError(f"A_log must have HV={v.shape[2]} elements, got {A_log.numel()}.")
    if cp_context is not None and getattr(cp_context, 'group', None) is not None:
        # under context parallelism the options run as passes of their own before / after the chunk kernels
        out_dtype = q.dtype
        if flags & (_lib.PREP_L2NORM | _lib.PREP_GATE | _lib.PREP_BETA_SIGMOID):
            q, k, g, beta = LayerOptionsFunction.apply(q, k, g, beta, A_log if use_gate_in_kernel else None,
                                                       dt_bias if use_gate_in_kernel else None, flags)
        from .cp import chunk_gated_delta_rule_cp
        o = chunk_gated_delta_rule_cp(q, k, v, g, beta, scale, cp_context)   # no states cross this interface
        return o.to(out_dtype), None

    # The gate and beta activations are fused into the first forward and the last backward kernel; the L2 norm's backward
    # is fused into the kernels that complete dq and dk.  States stored [V,K] (state_v_first) are read and written in that
    # layout by the scans themselves.
    if not use_gate_in_kernel:
        A_log = dt_bias = None
    args = (q, k, v, g, beta, initial_state, A_log, dt_bias, scale, output_final_state,
            flags | (_lib.STATE_V_FIRST if state_v_first else 0), cu_seqlens, cu_seqlens_cpu)
    return RecordedCall.apply(_native_chunk, *args) if recorded(q) else _native_chunk(*args)


chunk_gdn = chunk_gated_delta_rule

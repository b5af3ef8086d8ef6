"""Calls of the operators while torch.jit.trace records.

A native call leaves nothing in a trace: its results would be recorded as constants.  While a trace is being recorded the
operators therefore run as an autograd function of Python's, which the trace keeps as one operation (and which computes its
chunk tables anew for the lengths it is replayed with).  That a trace is being recorded shows in a tensor's sizes, which are
then tensors and not numbers (a look at a size's type costs 0.01 us, torch's own query 0.14)."""
from __future__ import annotations

import contextlib

import torch


def recorded(x: torch.Tensor) -> bool:
    return type(x.shape[0]) is not int


@contextlib.contextmanager
def untraced():
    """What happens inside is not recorded, and lengths are plain numbers."""
    state = torch._C._get_tracing_state()
    torch._C._set_tracing_state(None)
    try:
        yield
    finally:
        torch._C._set_tracing_state(state)


def seen_by_trace(results):
    """Copies that the trace knows the making of, as it has to of a node's results; the tensors themselves without a trace."""
    if torch._C._get_tracing_state() is None:
        return results
    return tuple(None if r is None else torch.empty(r.shape, dtype=r.dtype, device=r.device).copy_(r) for r in results)


class RecordedCall(torch.autograd.Function):
    """``fn(*args)`` as one node; the graph that ``fn`` leaves inside serves the node's backward pass.  A state that ``fn``
    updates in place is not served (torch.jit replays no such operation)."""

    @staticmethod
    def forward(ctx, fn, *args):
        grad = any(ctx.needs_input_grad)
        with untraced():
            inner = [a.detach().requires_grad_(grad and a.requires_grad) if isinstance(a, torch.Tensor) else a for a in args]
            with torch.set_grad_enabled(grad):
                results = fn(*inner)
            single = isinstance(results, torch.Tensor)
            ctx.inner, ctx.results = inner, (results,) if single else results
            if any(r is not None and r is a for r in ctx.results for a in inner):
                raise RuntimeError('a state updated in place cannot be recorded by torch.jit.trace')
            out = tuple(None if r is None else r.detach() for r in ctx.results)
        out = seen_by_trace(out)
        ctx.mark_non_differentiable(*[o for o, r in zip(out, ctx.results) if r is not None and not r.requires_grad])
        ctx.set_materialize_grads(False)
        return out[0] if single else out

    @staticmethod
    def backward(ctx, *grads):
        pairs = [(r, g) for r, g in zip(ctx.results, grads) if r is not None and r.requires_grad and g is not None]
        leaves = [a for a in ctx.inner if isinstance(a, torch.Tensor) and a.requires_grad]
        got = iter(torch.autograd.grad([r for r, _ in pairs], leaves, [g for _, g in pairs], retain_graph=True, allow_unused=True))
        return (None, *[next(got) if isinstance(a, torch.Tensor) and a.requires_grad else None for a in ctx.inner])

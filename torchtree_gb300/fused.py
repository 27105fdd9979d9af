"""One-launch model set-up: category rates and rate matrices by the engine's
kernels (``csrc/tt_setup.cu``) in place of ten to thirty tensor operations.

The tensor compositions in ``site_models`` and ``substitution`` stay the
definition.  They take everything these kernels do not (other types, devices,
shapes, transforms, tracing) and every backward that has to be differentiated
again.
"""
from __future__ import annotations

import ctypes

import torch

from . import _native
from ._native import check

try:  # the transforms and modes under which an operation must stay a composition of tensor operations
    from torch._C import _has_storage, _len_torch_dispatch_stack, _len_torch_function_stack
    from torch._C._functorch import peek_interpreter_stack
    from torch.autograd import forward_ad
except ImportError:  # a torch without these names: never take the kernels
    peek_interpreter_stack = None

    def _has_storage(_):
        return False


def plain_cuda(*tensors) -> bool:
    """Whether every tensor is an ordinary non-empty FP64 CUDA tensor (no lazy negation) of the
    current device, used outside of transforms (vmap, forward mode), modes,
    tracing and compilation."""
    if peek_interpreter_stack is None:
        return False
    first = tensors[0].device
    for t in tensors:
        if (type(t) not in (torch.Tensor, torch.nn.Parameter) or t.dtype != torch.float64 or t.device != first
                or t.numel() == 0 or t.is_neg() or not _has_storage(t)):  # (a batch of tensors has none)
            return False
    return (first.type == "cuda" and first.index == torch.cuda.current_device() and peek_interpreter_stack() is None
            and forward_ad._current_level < 0 and _len_torch_dispatch_stack() == 0
            and _len_torch_function_stack() == 0 and not torch.jit.is_tracing()
            and not torch.compiler.is_compiling())


def plain_gradient(g) -> bool:
    """Whether a backward's incoming gradient (of a plain output's type and device) is an
    ordinary tensor: no batch of them, no lazy negation."""
    return type(g) is torch.Tensor and _has_storage(g) and not g.is_neg()


def _stream(t):
    return torch.cuda.current_stream(t.device).cuda_stream


def _again(compose, inputs, outputs_grad):
    """Gradients of ``compose(*inputs)``, with a graph of their own where one is wanted.  Each with respect to an
    alias: an input made from another one would pass its share on to that one here, and again
    in the graph that this backward is part of."""
    create = torch.is_grad_enabled()
    with torch.enable_grad():
        own = [t.view_as(t) if t.requires_grad else t for t in inputs]
        out = compose(*own)
        want = [t for t in own if t.requires_grad]
        got = iter(torch.autograd.grad(out, want, outputs_grad, create_graph=create, allow_unused=True))
    return tuple(next(got) if t.requires_grad else None for t in inputs)


class CategoryRates(torch.autograd.Function):
    """``(rates [..., K], weights [K])`` of ``shape [..., 1]``; ``kind`` names the
    C call, ``compose(shape)`` the tensor composition."""

    @staticmethod
    def forward(ctx, shape, k, kind, compose):
        lib = _native.load()
        s = shape.contiguous()
        rates = torch.empty(shape.shape[:-1] + (k,), dtype=torch.float64, device=shape.device)
        drates = torch.empty_like(rates)
        weights = torch.empty(k, dtype=torch.float64, device=shape.device)
        check(getattr(lib, kind)(s.numel(), k, s.data_ptr(), rates.data_ptr(), drates.data_ptr(),
                                 weights.data_ptr(), _stream(shape)))
        ctx.save_for_backward(shape, drates)
        ctx.compose = compose
        ctx.mark_non_differentiable(weights)
        return rates, weights

    @staticmethod
    def backward(ctx, grad, _):
        shape, drates = ctx.saved_tensors
        if torch.is_grad_enabled():
            return (*_again(ctx.compose, (shape,), grad), None, None, None)
        if not plain_gradient(grad):  # a batch of incoming gradients
            return (grad * drates).sum(-1, keepdim=True), None, None, None
        grad = grad.contiguous()
        out = torch.empty(shape.shape, dtype=torch.float64, device=shape.device)
        check(_native.load().tt_rates_backward(shape.numel(), drates.shape[-1], grad.data_ptr(), drates.data_ptr(),
                                               out.data_ptr(), _stream(shape)))
        return out, None, None, None


class ExchangeabilityQ(torch.autograd.Function):
    """``q [b,S,S]`` of one to three parameter tensors ``[b,n]`` and ``pi [b,S]``;
    ``index`` is the host map of mapped models (int8 ``[2, S(S-1)/2]``) or None."""

    @staticmethod
    def forward(ctx, pi, index, compose, *params):
        lib = _native.load()
        b, S = pi.shape
        rows = [t.contiguous() for t in params]
        freqs = pi.contiguous()
        q = torch.empty(b, S, S, dtype=torch.float64, device=pi.device)
        ctx.counts = (ctypes.c_int32 * 3)(*([t.shape[-1] for t in rows] + [0] * (3 - len(rows))))
        ptrs = [t.data_ptr() for t in rows] + [None] * (3 - len(rows))
        check(lib.tt_exchangeability_q(b, S, ctx.counts, *ptrs, _native.ptr(index),
                                       freqs.data_ptr(), q.data_ptr(), _stream(pi)))
        ctx.index, ctx.compose = index, compose
        ctx.save_for_backward(pi, *params)
        return q

    @staticmethod
    def backward(ctx, grad):
        pi, *params = ctx.saved_tensors
        if torch.is_grad_enabled() or not plain_gradient(grad):
            gpi, *rest = _again(lambda f, *p: ctx.compose(*p, f), (pi, *params), grad)
            return (gpi, None, None, *rest)
        b, S = pi.shape
        rows = [t.contiguous() for t in params]
        freqs, grad = pi.contiguous(), grad.contiguous()
        need = ctx.needs_input_grad
        new = lambda t, wanted: (torch.empty(t.shape, dtype=torch.float64, device=t.device)  # noqa: E731
                                 if wanted else None)
        outs = [new(t, n) for t, n in zip(params, need[3:])]
        dpi = new(pi, need[0])
        pad = [None] * (3 - len(rows))
        ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
        check(_native.load().tt_exchangeability_q_backward(
            b, S, ctx.counts, *[t.data_ptr() for t in rows], *pad, _native.ptr(ctx.index), freqs.data_ptr(), grad.data_ptr(),
            *map(ptr, outs), *pad, ptr(dpi), _stream(pi)))
        return (dpi, None, None, *outs)

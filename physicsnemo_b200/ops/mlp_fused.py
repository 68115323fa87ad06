"""Three linear layers, two activations, LayerNorm and residual of a 128-wide message-passing MLP as one kernel.

``mlp3_ln``: ``LayerNorm(act(act(x W1^T + b1) W2^T + b2) W3^T + b3) (+ post)`` where ``x`` is the concatenation of up to
three 128-wide tables, each read through an optional row index (``csrc/mlp_fused.cuh``): the edge update of a
MeshGraphNet step copies its node rows one by one, the node update reads tiles of (aggregate, node).  Layer by layer the same
chain (``ops.gather_rows``, ``ops.mlp_chain``, ``ops.layer_norm``) writes and re-reads every intermediate row.
"""
from __future__ import annotations

import ctypes
from typing import Optional, Sequence

import torch

from . import _lib
from . import gemm as _g
from . import graph as _graph

WIDTH = 128
ROWS = 128                                                   # rows of a tile of the kernel
_ACTS = (_g.ACT_GELU, _g.ACT_SILU, _g.ACT_RELU)


def _lib_mlp():
    """The library with the signatures of the two calls that are launched by themselves (by tests; a backward launches natively)."""
    lib = _lib.load(required=True)
    if not getattr(lib, "_mlp3_declared", False):
        c = ctypes
        vp, i, l = c.c_void_p, c.c_int, c.c_longlong
        lib.pnm_mlp3_bwd.argtypes = [vp, vp, vp, vp, vp, vp, vp, i, vp, vp, vp, vp, vp, l, vp]
        lib.pnm_segment_sum_split.argtypes = [vp, vp, vp, vp, l, l, i, vp]
        lib.pnm_mlp3_bwd.restype = lib.pnm_segment_sum_split.restype = i
        lib._mlp3_declared = True
    return lib


def supported(srcs: Sequence[torch.Tensor], segs: Sequence, weights, biases, acts, gamma, beta, post: Optional[int]) -> bool:
    """Three 128-wide layers with the same activation after the first two and a 128-wide affine LayerNorm, on aligned
    bf16 tables of one device."""
    if not 1 <= len(srcs) <= 3 or len(weights) != 3 or len(acts) != 3 or acts[0] not in _ACTS or acts[1] != acts[0] or acts[2] != _g.ACT_NONE:
        return False
    # bf16 tables of 128 columns whose rows start on 32-byte boundaries; parameters of the right shapes on the same device
    if not _lib.host().mlp3_operands_ok(srcs, weights, biases, gamma, beta):
        return False
    rows = None
    for t, s in zip(srcs, segs):
        n = t.shape[0]
        if s is not None:
            if s.num_segments != n:
                return False
            n = s.num_items
        if n == 0 or (rows is not None and rows != n):
            return False
        rows = n
    return post is None or segs[post] is None


def _forward(srcs, segs, weights, biases, act, gamma, beta, eps, post, save: bool):
    m = segs[0].num_items if segs[0] is not None else srcs[0].shape[0]
    # kept: h1, h2, x3, mean, rstd; z1 and z2 (whole tiles) but for ReLU
    res = _lib.host().mlp3_fwd(srcs, [None if s is None else s.index32 for s in segs], [_g._bf16_weight(w) for w in weights],
                               (*biases, gamma, beta), eps, act, post, m, save)
    _g.launch_count += 1
    return (res[0], res[1:]) if save else (res, ())


def _w_t(w: torch.Tensor) -> torch.Tensor:
    return _g._bf16_weight(w, transpose=True)


class _Mlp3LnFn(torch.autograd.Function):
    """``srcs`` come first among the tensor arguments; ``post`` names the (un-indexed) source that is added to the result.
    ``tables``: the indexed sources that read the same tensor, or ``None`` where there will be no backward."""

    @staticmethod
    def forward(ctx, segs, tables, act, eps, post, *tensors):
        n = len(segs)
        srcs, (w1, w2, w3, b1, b2, b3, gamma, beta) = tensors[:n], tensors[n:]
        y, kept = _forward(srcs, segs, (w1, w2, w3), (b1, b2, b3), act, gamma, beta, eps, None if post is None else srcs[post],
                           tables is not None)
        if tables is None:
            return y
        ctx.save_for_backward(*srcs, w1, w2, w3, gamma, *kept)
        ctx.segs, ctx.tables, ctx.act, ctx.post = segs, tables, act, post
        ctx.dtypes = [None if t is None else t.dtype for t in (w1, w2, w3, b1, b2, b3, gamma, beta)]
        return y

    @staticmethod
    def backward(ctx, dy):
        n = len(ctx.segs)
        saved = ctx.saved_tensors                            # read once: activation checkpointing allows no second time
        srcs, (w1, w2, w3, gamma, h1, h2, x3, mean, rstd, *z) = saved[:n], saved[n:]
        z1, z2 = z or (h1, h2)
        # An indexed source: the gradient is summed over the rows that read a table row FIRST (the products are linear), then one small
        # product per table instead of one per row of M.  The fp32 sums go into the products as a bf16 pair (hi + lo): every sum
        # against the table in one product, and the two halves of a sum are added afterwards.
        dsrc, *grads, launches = _lib.host().mlp3_bwd(dy, srcs, ctx.segs, ctx.tables, ctx.needs_input_grad[5:], ctx.post, ctx.act,
                                                      (_w_t(w1), _w_t(w2), _w_t(w3)), gamma, (h1, h2, x3, mean, rstd, z1, z2))
        _g.launch_count += launches
        grads = [None if dt is None else (t if t.dtype == dt else t.to(dt)) for t, dt in zip(grads, ctx.dtypes)]
        return (None, None, None, None, None, *dsrc, *grads)


_KINDS = (torch.nn.Linear, torch.nn.SiLU, torch.nn.ReLU, torch.nn.GELU, torch.nn.LayerNorm)


def module_call(model: torch.nn.Sequential, srcs, segs, post: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """The kernel's result for a call without gradients, straight from the modules; ``None`` where the general way has to decide."""
    if torch.is_grad_enabled() or _g.call_is_observed():
        return None
    y = _lib.host().mlp3_module(model._modules, srcs, segs, post, _g._wcache, _g._captured, _lib.stream(), _KINDS)
    if y is not None:
        _g.launch_count += 1
    return y


def mlp3_ln(srcs: Sequence[torch.Tensor], segs: Sequence[Optional["_graph.SegmentIndex"]], weights, biases, act: int, gamma, beta,
            eps: float, post: Optional[int]) -> torch.Tensor:
    """See the module docstring; ``segs[j]`` names the rows of ``srcs[j]`` (``None``: row by row), ``post`` the source that is
    added to the result.  Call after ``supported``."""
    params = (*weights, *biases, gamma, beta)
    tables = None
    if torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (*srcs, *params)):
        by_tensor = {}
        for j, (t, s) in enumerate(zip(srcs, segs)):
            if s is not None:
                by_tensor.setdefault(id(t), []).append(j)
        tables = tuple(by_tensor.values())
    elif not _g.call_is_observed():                          # the function call costs 14 us on the host, the launch 9 on the device
        return _forward(srcs, segs, weights, biases, act, gamma, beta, eps, None if post is None else srcs[post], False)[0]
    return _Mlp3LnFn.apply(tuple(segs), tables, act, float(eps), post, *srcs, *params)

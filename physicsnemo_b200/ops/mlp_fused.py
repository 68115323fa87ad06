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


def _vec(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """fp32 contiguous, 16-byte aligned values of a parameter vector, for a launch: the parameter itself where it is that already."""
    if t is None:
        return None
    t = _g._f32(t)
    return t if t.data_ptr() % 16 == 0 else t.detach().clone()


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
        segs, post = ctx.segs, ctx.post
        n = len(segs)
        saved = ctx.saved_tensors                            # read once: activation checkpointing allows no second time
        srcs, (w1, w2, w3, gamma, h1, h2, x3, mean, rstd, *z) = saved[:n], saved[n:]
        z1, z2 = z or (h1, h2)
        m, dev = x3.shape[0], x3.device
        dy = _g._aligned(dy.contiguous())
        lib = _lib_mlp()
        # all gradients of parameters in one zeroed buffer, and nothing else: it lives as long as they do
        sizes = [n * WIDTH * WIDTH, WIDTH * WIDTH, WIDTH * WIDTH] + [WIDTH] * 5
        dw1, dw2, dw3, db1, db2, db3, dgamma, dbeta = torch.zeros(sum(sizes), dtype=torch.float32, device=dev).split(sizes)
        dw1, dw2, dw3 = dw1.view(WIDTH, -1), dw2.view(WIDTH, WIDTH), dw3.view(WIDTH, WIDTH)
        block = [dw1[:, j * WIDTH:(j + 1) * WIDTH] for j in range(n)]            # of source j
        rows = torch.empty((2, m, WIDTH), dtype=torch.bfloat16, device=dev)
        dx3, g1 = rows[0], rows[1]
        scratch = torch.empty(lib.pnm_layernorm_bwd_scratch_floats(m, WIDTH), dtype=torch.float32, device=dev)
        code = lib.pnm_layernorm_bwd(dy.data_ptr(), x3.data_ptr(), _vec(gamma).data_ptr(), mean.data_ptr(), rstd.data_ptr(), None,
                                     dx3.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(), scratch.data_ptr(), m, WIDTH,
                                     _g._stream())
        _g._check(code, "pnm_layernorm_bwd")
        w3t, w2t = _w_t(w3), _w_t(w2)                        # held: the second look-up may empty the cache
        code = lib.pnm_mlp3_bwd(dx3.data_ptr(), z2.data_ptr(), z1.data_ptr(), h2.data_ptr(), h1.data_ptr(), w3t.data_ptr(), w2t.data_ptr(),
                                ctx.act, g1.data_ptr(), dw3.data_ptr(), dw2.data_ptr(), db3.data_ptr(), db2.data_ptr(), m, _g._stream())
        _g._check(code, "pnm_mlp3_bwd")
        _g.launch_count += 3
        need = ctx.needs_input_grad[5:]
        w1t = _w_t(w1)                                       # [128 n, 128]: rows j * 128 .. belong to source j
        dsrc = [None] * n
        summed_bias = False
        for j in range(n):
            if segs[j] is None:
                if need[j]:
                    own = {"aux": dy, "aux_mode": _g.AUX_ADD} if post == j else {}
                    dsrc[j] = _g.gemm_tn(g1, w1t[j * WIDTH:(j + 1) * WIDTH], **own)
                _g.gemm_nt(g1, srcs[j], out=block[j], colsum_out=None if summed_bias else db1)
                summed_bias = True
        # An indexed source: sum g1 over the rows that read a table row FIRST (the products are linear), then one small product
        # per table instead of one per row of M.  The fp32 sums go into the products as a bf16 pair (hi + lo).
        for js in ctx.tables:
            src, rows = srcs[js[0]], segs[js[0]].num_segments
            pairs = torch.empty((rows, 2 * WIDTH * len(js)), dtype=torch.bfloat16, device=dev)
            for k, j in enumerate(js):
                part = pairs[:, 2 * k * WIDTH:]
                code = lib.pnm_segment_sum_split(g1.data_ptr(), segs[j].perm.data_ptr(), segs[j].offsets.data_ptr(), part.data_ptr(),
                                                 pairs.stride(0), rows, WIDTH, _g._stream())
                _g._check(code, "pnm_segment_sum_split")
                _g.launch_count += 1
            # every sum against the table in one product; the two halves of a sum are added afterwards
            both = torch.zeros(pairs.shape[1] * (WIDTH + 1), dtype=torch.float32, device=dev)
            part = both[:pairs.shape[1] * WIDTH].view(-1, WIDTH)
            _g.gemm_nt(pairs, src, out=part, colsum_out=None if summed_bias else both[part.numel():])
            halves = part.view(len(js), 2, WIDTH, WIDTH)
            for k, j in enumerate(js):
                torch.add(halves[k, 0], halves[k, 1], out=block[j])
            if not summed_bias:
                db1 = both[part.numel():].view(len(js), 2, WIDTH)[0].sum(0)
                summed_bias = True
            if any(need[j] for j in js):
                wt = torch.cat([w1t[j * WIDTH:(j + 1) * WIDTH] for j in js for _ in range(2)], 1)
                dsrc[js[0]] = _g.gemm_tn(pairs, wt)
        grads = [dw1, dw2, dw3, db1, db2, db3, dgamma, dbeta]
        grads = [None if dt is None else (t if t.dtype == dt else t.to(dt)) for t, dt in zip(grads, ctx.dtypes)]
        return (None, None, None, None, None, *dsrc, *grads)


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

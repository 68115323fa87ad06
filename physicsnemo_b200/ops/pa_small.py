"""ctypes bindings of the four small-algebra kernels of the fused physics attention (``csrc/physics_attn_small.cu``)."""
from __future__ import annotations

import ctypes
import math
from typing import List, Optional, Sequence

import torch

from . import _lib
from . import gemm as _g

S = 64  # slices per head covered by the kernels


def _lib_pa():
    lib = _lib.load(required=True)
    if not getattr(lib, "_pasmall_declared", False):
        c = ctypes
        vp, i, u, ll, f, d = c.c_void_p, c.c_int, c.c_uint, c.c_longlong, c.c_float, c.c_double
        lib.pnm_pa_tokens_fwd.argtypes = [vp, i, i, ll, i, vp, vp, vp, vp, i, i, i, f, vp, i, u, ll, d, vp, vp]
        lib.pnm_pa_tokens_bwd.argtypes = [vp, i, i, vp, vp, vp, vp, vp, vp, vp, vp, i, i, i, f, f, vp, i, u, ll, d, vp, vp]
        for n in ("pnm_pa_tokens_fwd", "pnm_pa_tokens_bwd"):
            getattr(lib, n).restype = i
        lib._pasmall_declared = True
    return lib


def _st():
    return _lib.stream()


def _ptr_array(ptrs: Sequence[int]):
    return (ctypes.c_void_p * len(ptrs))(*ptrs)


def supported(H: int, D: int, slices: int, C: int, params: Sequence[torch.Tensor]) -> bool:
    return (slices == S and 0 < D <= 64 and 256 % D == 0 and (H * D) % 8 == 0 and C % 8 == 0
            and all(p.dtype == torch.float32 and p.is_cuda and p.is_contiguous() for p in params))      # read as they lie


def prepare_fwd(Wx, bx, Wfx, Ws, bs, temp, H: int, D: int):
    """``(Wc bf16 [H*S, C], bc [H*S], inv_t [H*S], Wfx bf16, Wback bf16 [C, H*S + H*D])``."""
    res = _lib.host().pa_prepare_fwd(Wx, bx, Wfx, Ws, bs, temp, H, D)
    _g.launch_count += 1
    return res


def _saved_shapes(H: int, D: int, Cout: int) -> tuple:
    """What the forward keeps, one after the other in one fp32 buffer: token, norm, q, k, v, probabilities, out, Wcomb."""
    t = (H, S, D)
    return t, (H, S), t, t, t, (H, S, S), t, (Cout, H * S)


def saved_parts(saved: torch.Tensor, H: int, D: int, Cout: int) -> List[torch.Tensor]:
    shapes = _saved_shapes(H, D, Cout)
    return [p.view(s) for p, s in zip(saved.split([math.prod(s) for s in shapes]), shapes)]


def tokens_fwd(src_ptrs: Sequence[int], norm_off: int, ld_tok: int, Wqkv, Wo, H: int, D: int, peer: Optional[tuple] = None):
    """``(Wcomb bf16 [Cout, H*S], saved)``; ``src_ptrs``: per rank the address of the [H*S, ld_tok] token-sum matrix.

    ``peer``: ``PeerRuntime.peer_args(epoch)`` when the sources are peers' buffers whose flags must be awaited.
    """
    _g.launch_count += 1
    if peer is None and len(src_ptrs) == 1:
        return _lib.host().pa_tokens_fwd(src_ptrs[0], norm_off, ld_tok, Wqkv, Wo, H, D)
    Cout = Wo.shape[0]
    saved = torch.empty(sum(math.prod(s) for s in _saved_shapes(H, D, Cout)), dtype=torch.float32, device=Wo.device)
    wcomb16 = torch.empty(Cout, H * S, dtype=torch.bfloat16, device=Wo.device)
    bases, rank, _w, epoch, cap, budget, ebase = peer if peer is not None else (None, 0, 1, 0, 0, 1.0, None)
    err = _lib_pa().pnm_pa_tokens_fwd(_ptr_array(src_ptrs), len(src_ptrs), int(peer is not None), norm_off, ld_tok, Wqkv.data_ptr(), Wo.data_ptr(),
                                      wcomb16.data_ptr(), _ptr_array([t.data_ptr() for t in saved_parts(saved, H, D, Cout)]), H, D, Cout,
                                      float(D) ** -0.5, bases, rank, epoch, cap, budget, ebase, _st())
    _g._check(err, "pnm_pa_tokens_fwd")
    return wcomb16, saved


def tokens_bwd(src_ptrs: Sequence[int], Wqkv, Wo, saved, H: int, D: int, share: float, peer: Optional[tuple] = None):
    """``(dWo, dWqkv, d_norm [H*S], Bcat bf16 [H*S, Cout + H*D], BdT bf16 [H*D, H*S])``."""
    _g.launch_count += 1
    if peer is None and len(src_ptrs) == 1:
        return _lib.host().pa_tokens_bwd(src_ptrs[0], Wqkv, Wo, saved, H, D, share)
    Cout = Wo.shape[0]
    dev = Wo.device
    inner = H * D
    dWo = torch.empty(Cout, inner, dtype=torch.float32, device=dev)
    dWqkv = torch.zeros(3 * D, D, dtype=torch.float32, device=dev)
    d_norm = torch.empty(H * S, dtype=torch.float32, device=dev)
    Bcat = torch.empty(H * S, Cout + inner, dtype=torch.bfloat16, device=dev)
    BdT = torch.empty(inner, H * S, dtype=torch.bfloat16, device=dev)
    bases, rank, _w, epoch, cap, budget, ebase = peer if peer is not None else (None, 0, 1, 0, 0, 1.0, None)
    err = _lib_pa().pnm_pa_tokens_bwd(_ptr_array(src_ptrs), len(src_ptrs), int(peer is not None), Wqkv.data_ptr(), Wo.data_ptr(),
                                      _ptr_array([t.data_ptr() for t in saved_parts(saved, H, D, Cout)]), dWo.data_ptr(), dWqkv.data_ptr(),
                                      d_norm.data_ptr(), Bcat.data_ptr(), BdT.data_ptr(), H, D, Cout, float(D) ** -0.5,
                                      float(share), bases, rank, epoch, cap, budget, ebase, _st())
    _g._check(err, "pnm_pa_tokens_bwd")
    return dWo, dWqkv, d_norm, Bcat, BdT


def prepare_bwd(dW, db, grp, Wx, bx, Ws, temp, H: int, D: int):
    """``(dWx, dbx, dWfx, dbfx, dWs, dbs, dtemp)`` from the gradients of the combined projection and, below them, of the values' projection."""
    res = _lib.host().pa_prepare_bwd(dW, db, grp, Wx, bx, Ws, temp, H, D)
    _g.launch_count += 1
    return res

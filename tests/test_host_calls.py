"""Calls without gradients go to an autograd function's ``forward`` directly; the native host calls refuse what the Python code refused."""
import pytest
import torch

from physicsnemo_b200.ops import _lib
from physicsnemo_b200.ops import gemm as G


class _Twice(torch.autograd.Function):
    contexts: list = []

    @staticmethod
    def forward(ctx, x, k):
        _Twice.contexts.append(type(ctx).__name__)
        ctx.save_for_backward(x)
        ctx.k = k
        return x * k

    @staticmethod
    def backward(ctx, g):
        return g * ctx.k, None


def test_apply_function_takes_the_graph_where_a_gradient_is_wanted():
    x = torch.randn(3, requires_grad=True)
    _Twice.contexts.clear()
    G.apply_function(_Twice, x, 2.0).sum().backward()
    assert torch.equal(x.grad, torch.full((3,), 2.0)) and _Twice.contexts[-1] != "_NoContext"
    with torch.no_grad():
        y = G.apply_function(_Twice, x, 2.0)
    assert torch.equal(y, 2 * x) and not y.requires_grad and _Twice.contexts[-1] == "_NoContext"
    y = G.apply_function(_Twice, x.detach(), 2.0)                        # gradients enabled, none wanted
    assert not y.requires_grad and _Twice.contexts[-1] == "_NoContext"
    with torch.autograd.forward_ad.dual_level(), torch.no_grad():        # a level is open: the function object says what it can do
        G.apply_function(_Twice, x, 2.0)
    assert _Twice.contexts[-1] != "_NoContext"


@pytest.mark.skipif(not _lib._HOST_PATH.exists(), reason="the kernel library is not built")
def test_host_calls_refuse_bad_operands():
    host, t = _lib.host(), torch.randn(4, 128).bfloat16()
    assert not host.mlp3_operands_ok([t], [torch.randn(128, 128)] * 3, [None] * 3, torch.ones(128), None)     # not on a GPU
    with pytest.raises(TypeError):
        host.gemm_nt(t, None, False, None, None, 0)
    with pytest.raises(TypeError):
        host.gemm_nt(t)
    with pytest.raises(AssertionError):                                  # different numbers of rows
        host.gemm_nt(t, t[:3], False, None, None, 0)
    with pytest.raises(AssertionError):                                  # different numbers of columns
        host.gemm_tn(t, t[:, :64], None, None, 0, None, 0, None, None, False, None, None, False, 0, 0)
    with pytest.raises(AssertionError):                                  # not bf16
        host.gemm_tn(t.float(), t.float(), None, None, 0, None, 0, None, None, False, None, None, False, 0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,channels,side,groups,dtype", [(1, 128, 5, 32, torch.bfloat16),     # slices of fewer pixels than are loaded ahead
                                                             (2, 96, 33, 32, torch.bfloat16),     # three channels a group: values per channel
                                                             (1, 24, 7, 3, torch.bfloat16), (2, 64, 37, 32, torch.float32),
                                                             (1, 36, 19, 12, torch.float32), (1, 512, 8, 32, torch.bfloat16)])
def test_group_norm_channels_last_edges(batch, channels, side, groups, dtype):
    from physicsnemo_b200.ops import group_norm as gn

    gen = torch.Generator().manual_seed(channels + side)
    x, up = (torch.randn(batch, channels, side, side, generator=gen).to(dtype) for _ in range(2))
    ga, be = 1 + 0.1 * torch.randn(channels, generator=gen), 0.1 * torch.randn(channels, generator=gen)
    ref = [t.double().requires_grad_() for t in (x, ga, be)]
    y = torch.nn.functional.silu(torch.nn.functional.group_norm(ref[0], groups, *ref[1:], 1e-5))
    y.backward(up.double())
    dev = [x.cuda().contiguous(memory_format=torch.channels_last).requires_grad_(), ga.cuda().requires_grad_(), be.cuda().requires_grad_()]
    assert gn.supported(dev[0], groups)
    out = gn.group_norm(dev[0], groups, dev[1], dev[2], 1e-5, silu=True)
    out.backward(up.cuda().contiguous(memory_format=torch.channels_last))
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6       # one rounding of the result (2^-9), or sums of a few thousand fp32 terms
    for a, b in ((out, y), *((d.grad, r.grad) for d, r in zip(dev, ref))):
        assert float((a.detach().cpu().double() - b.detach()).norm() / b.detach().norm()) < tol

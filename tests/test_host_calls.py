"""Calls without gradients go to an autograd function's ``forward`` directly; the native host calls refuse what the Python code refused."""
import threading
import time

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


@pytest.mark.skipif(not _lib._HOST_PATH.exists(), reason="the kernel library is not built")
def test_host_calls_copy_operands_without_the_interpreters_lock():
    """Another thread runs while an operand is copied (or its memory allocated, which may wait for the device)."""
    host, b = _lib.host(), torch.zeros(8, 16).bfloat16()
    a = torch.zeros(8192, 8192).bfloat16().t()                           # read by columns: copied before its width is refused
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(1e-3)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        inside, threads = 0, torch.get_num_threads()
        torch.set_num_threads(1)
        for _ in range(3):
            began = time.perf_counter()
            with pytest.raises(AssertionError):
                host.gemm_tn(a, b, None, None, 0, None, 0, None, None, False, None, None, False, 0, 0)
            ended = time.perf_counter()
            margin = 0.25 * (ended - began)                              # an end of the call may overlap with a tick that began outside
            inside += sum(began + margin < t < ended - margin for t in ticks)
    finally:
        torch.set_num_threads(threads)
        stop.set()
        thread.join()
    assert inside > 0


def _forms(t):
    """The values of a matrix by columns, in rows of an odd stride, one element off a 16-byte boundary, and with a longer row stride."""
    m, n = t.shape
    odd, off, wide = t.new_empty(m, n + 1), t.new_empty(m * n + 1), t.new_empty(m, n + 8)
    odd[:, :n], off[1:], wide[:, 8:] = t, t.reshape(-1), t
    return [t.t().contiguous().t(), odd[:, :n], off[1:].view(m, n), wide[:, 8:]]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [3, 130])
def test_host_calls_copy_strided_and_misaligned_operands(rows):
    from physicsnemo_b200.ops import mlp_fused as mf

    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    a, a2, b, aux, bias = bf(rows, 64), bf(rows, 128), bf(72, 192), bf(rows, 72), torch.randn(72, device="cuda")
    want = G.gemm_tn(a, b, bias=bias, a2=a2, aux=aux, aux_mode=G.AUX_ADD)
    for x, x2, w, r in zip(_forms(a), _forms(a2), _forms(b), _forms(aux)):
        assert torch.equal(G.gemm_tn(x, w, bias=bias, a2=x2, aux=r, aux_mode=G.AUX_ADD), want)
    ref, sums = a.double().t() @ a2.double(), a.double().sum(0)
    for x, x2 in zip(_forms(a), _forms(a2)):
        got, got_sums = G.gemm_nt(x, x2, colsum=True)
        # exact products of bf16 values, at most 130 of them added in fp32
        assert float((got - ref).abs().max()) < 1e-4 and float((got_sums - sums).abs().max()) < 1e-4
    # parameter vectors of the one-kernel MLP: bf16, every other value of a longer vector, off a 16-byte boundary
    x, w = bf(rows, 128), [bf(128, 128) / 11 for _ in range(3)]
    vec = [torch.randn(128, device="cuda").bfloat16().float() for _ in range(5)]
    want = mf._forward([x], [None], w, vec[:3], 2, *vec[3:], 1e-5, None, False)[0]
    for form in (lambda v: v.bfloat16(), lambda v: v.repeat_interleave(2)[::2], lambda v: torch.cat([v[:1], v])[1:]):
        v = [form(t) for t in vec]
        assert torch.equal(mf._forward([x], [None], w, v[:3], 2, *v[3:], 1e-5, None, False)[0], want)


@pytest.mark.gpu
def test_host_calls_raise_for_tensors_without_storage():
    """The pointer is read where the interpreter's lock is released: its error arrives as an exception all the same."""
    host, idx = _lib.host(), torch.zeros(4, dtype=torch.int32, device="cuda")
    raised = []

    def inner(x):                                                        # x: a wrapper of vmap
        for call in (lambda: host.gather_rows(x, idx, None, None), lambda: host.gemm_nt(x, x, False, None, None, 0),
                     lambda: host.segment_sum(x, idx, idx, 3, False, False, None)):
            with pytest.raises(RuntimeError, match="storage"):
                call()
            raised.append(call)
        return x

    torch.vmap(inner)(torch.randn(2, 3, 8, device="cuda").bfloat16())
    assert len(raised) == 3


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


@pytest.mark.skipif(not _lib._HOST_PATH.exists(), reason="the kernel library is not built")
@pytest.mark.parametrize("batch,channels,groups,slices", [(1, 8, 1, 1), (3, 96, 32, 7), (2, 256, 256, 600)])
def test_group_norm_scratch_holds_the_counters_of_the_call(batch, channels, groups, slices):
    from physicsnemo_b200.ops import group_norm as gn

    # partials of every slice, folded sums, one counter per batch item (the last also where a group has a single channel)
    assert gn._lib_gn().pnm_groupnorm_scratch_floats(batch, channels, groups, slices) >= 2 * batch * slices * groups + 2 * batch * groups + batch


@pytest.mark.gpu
def test_group_norm_channels_last_on_two_streams():
    """Calls of different slice counts side by side give what they give one after the other."""
    from physicsnemo_b200.ops import group_norm as gn

    shapes = [(2, 128, 96, 32), (2, 64, 40, 32)]             # batch, channels, side, groups
    args = [(torch.randn(b, c, s, s, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last), g,
             torch.randn(c, device="cuda"), torch.randn(c, device="cuda")) for b, c, s, g in shapes]
    ups = [torch.randn_like(a[0]) for a in args]

    def step(k):
        x, g, ga, be = args[k]
        leaves = [t.clone().requires_grad_() for t in (x, ga, be)]
        y = gn.group_norm(leaves[0], g, *leaves[1:], 1e-5, silu=True)
        return [y.detach(), *torch.autograd.grad(y, leaves, ups[k])]

    serial = [step(k) for k in range(2)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    beside = [[], []]
    for _ in range(60):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                beside[k].append(step(k))
    torch.cuda.synchronize()
    for want, runs in zip(serial, beside):
        for got in runs:
            assert torch.equal(got[0], want[0])              # moments are folded in a fixed order
            # the backward adds a channel's pixels with fp32 atomics: a rounding of bf16 (2^-9) at most, parameter gradients in fp32
            assert float((got[1].double() - want[1].double()).norm() / want[1].double().norm()) < 2.0 ** -9
            assert all(float((a - b).norm() / b.norm()) < 1e-5 for a, b in zip(got[2:], want[2:]))


def test_build_passes_with_a_cpu_build_of_torch(monkeypatch):
    import __graft_entry__ as entry

    class Library:
        def pnm_version(self):
            return 100

    def no_host():
        raise RuntimeError("not built")

    monkeypatch.setattr(torch.version, "cuda", None)
    monkeypatch.setattr(_lib, "build", lambda force: _lib.lib_path())    # compiles the kernels only
    monkeypatch.setattr(_lib, "load", lambda required=False: Library())
    monkeypatch.setattr(_lib, "host", no_host)
    entry.build()


def _tree(tmp_path, monkeypatch):
    """A tree of empty sources and built files that are up to date; the compilers' command lines are recorded."""
    import os

    src, out, ran = tmp_path / "csrc", tmp_path / "lib", []
    src.mkdir()
    out.mkdir()
    monkeypatch.setattr(_lib, "_SRC_DIR", src)
    monkeypatch.setattr(_lib, "_LIB_DIR", out)
    monkeypatch.setattr(_lib, "_LIB_PATH", out / _lib._LIB_PATH.name)
    monkeypatch.setattr(_lib, "_HOST_PATH", out / _lib._HOST_PATH.name)
    monkeypatch.setattr(torch.version, "cuda", "12.8")
    for k, name in enumerate(("kernels.cu", "kernels.cuh", "pnm_api.h", "host_calls.cpp")):
        (src / name).touch()
        os.utime(src / name, (1000 + k, 1000 + k))

    def run(cmd, **kwargs):
        ran.append(cmd[0])
        target = next(t for f, t in zip(cmd, cmd[1:]) if f == "-o")
        open(target, "w").close()
        return type("Done", (), {"returncode": 0, "stdout": "", "stderr": ""})()

    monkeypatch.setattr(_lib.subprocess, "run", run)
    monkeypatch.setenv("NVCC", "nvcc")
    monkeypatch.setenv("CXX", "g++")
    _lib.build()
    assert ran == ["nvcc", "g++"] and not _lib.needs_build()
    ran.clear()
    return src, ran


@pytest.mark.parametrize("name,compilers", [("host_calls.cpp", ["g++"]), ("kernels.cuh", ["nvcc"]), ("pnm_api.h", ["nvcc", "g++"])])
def test_only_what_is_out_of_date_is_built(tmp_path, monkeypatch, name, compilers):
    import os

    src, ran = _tree(tmp_path, monkeypatch)
    later = time.time() + 60
    os.utime(src / name, (later, later))
    assert _lib.needs_build()
    _lib.build()
    assert ran == compilers


def test_host_calls_belong_to_one_python_and_one_torch(tmp_path, monkeypatch):
    """Another torch or Python has an extension of its own and leaves the other's in place; the wheel is for one Python."""
    import runpy
    import sysconfig
    from pathlib import Path

    import setuptools

    names = {_lib._HOST_PATH.name}
    get = sysconfig.get_config_var
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.1")
        names.add(_lib._host_path().name)
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-399-other" if name == "SOABI" else get(name))
        names.add(_lib._host_path().name)
    assert len(names) == 3
    src, ran = _tree(tmp_path, monkeypatch)
    monkeypatch.setattr(_lib, "_HOST_PATH", _lib._HOST_PATH.with_name(max(names - {_lib._HOST_PATH.name})))
    assert _lib.needs_build()
    _lib.build()
    assert ran == ["g++"] and len(list(_lib._LIB_DIR.glob("_pnm_host.*"))) == 2
    asked = {}
    monkeypatch.setattr(setuptools, "setup", lambda **kwargs: asked.update(kwargs))
    runpy.run_path(str(Path(__file__).resolve().parents[1] / "setup.py"))
    assert asked["distclass"]().has_ext_modules()


def test_declared_functions_are_called():
    """A function that the loader declares is called somewhere in the package (calls that went to the extension leave no declaration)."""
    import re
    from pathlib import Path

    class Recorder:
        def __getattr__(self, name):
            return self.__dict__.setdefault(name, type("Function", (), {})())

    lib = Recorder()
    _lib._declare(lib)
    own = Path(_lib.__file__)
    text = "\n".join(f.read_text() for f in own.parents[1].rglob("*.py") if f != own) + own.read_text().split("def load(")[1]
    entry = Path(__file__).resolve().parents[1] / "__graft_entry__.py"
    assert vars(lib) and [name for name in vars(lib) if not re.search(rf"\.{name}\b", text + entry.read_text())] == []


def test_mlps_with_an_identity_activation_stay_layer_by_layer():
    """The fused chain takes Linear / activation / ... / Linear: an Identity between two layers is refused, no error."""
    from torch import nn

    from physicsnemo_b200.nn.module.gnn_layers.mesh_graph_mlp import MeshGraphMLP, _layers

    lin = lambda: nn.Linear(8, 8)  # noqa: E731
    assert _layers(nn.Sequential(lin(), nn.Identity(), lin())) is None
    assert _layers(nn.Sequential(nn.SiLU(), lin())) is None and _layers(nn.Sequential(lin(), nn.SiLU(), nn.SiLU(), lin())) is None
    model = nn.Sequential(lin(), nn.SiLU(), lin(), lin(), nn.LayerNorm(8))
    weights, biases, acts, norm = _layers(model)
    assert acts == [2, 0, 0] and weights[1] is model[2].weight and biases[2] is model[3].bias and norm is model[4]
    m, x = MeshGraphMLP(8, 8, 8, 2, nn.Identity()), torch.randn(5, 8)
    assert torch.equal(m(x), m.model(x))

"""Loader / builder of the in-tree sm_100a kernel library ``libpnm_b200.so``.

The library is plain C ABI (see ``csrc/pnm_api.h``) bound through ``ctypes``: every
call passes raw device pointers and the current CUDA stream.  ``build()`` compiles the
single translation unit ``csrc/pnm_lib.cu`` with
``nvcc -gencode arch=compute_100a,code=sm_100a`` (cross-compiles without a GPU), and the CPython
extension ``_pnm_host.*.so`` from ``csrc/host_calls.cpp``: the host side of the hottest calls
(operand checks, allocation, launch), without ctypes.  The library serves any Python; the extension serves the Python and the torch
that its file name gives, and is built anew for others.
On a machine with a CUDA device a missing library is an error, never a silent
fallback.
"""
from __future__ import annotations

import ctypes
import os
import subprocess
import sysconfig
import threading
from pathlib import Path

import torch

_PKG_DIR = Path(__file__).resolve().parents[1]
_REPO = _PKG_DIR.parent
_SRC_DIR = _REPO / "csrc"
_LIB_DIR = _PKG_DIR / "lib"
_LIB_PATH = _LIB_DIR / "libpnm_b200.so"


def _host_path() -> Path:
    """The extension's binary interface is that of one Python and one torch: its name says which."""
    return _LIB_DIR / f"_pnm_host.torch-{torch.__version__}.{sysconfig.get_config_var('SOABI')}.so"


_HOST_PATH = _host_path()
_lock = threading.Lock()
_lib = None
_host = None
_load_error: str | None = None

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def lib_path() -> Path:
    return _LIB_PATH


def _sources():
    return sorted(list(_SRC_DIR.glob("*.cu")) + list(_SRC_DIR.glob("*.cuh")) + list(_SRC_DIR.glob("*.h")))


def _stale(target: Path, sources) -> bool:
    return not target.exists() or any(p.stat().st_mtime > target.stat().st_mtime for p in sources)


def _kernels_need_build() -> bool:
    return _stale(_LIB_PATH, _sources())


def _host_needs_build() -> bool:
    if torch.version.cuda is None:                           # nothing is launched without CUDA
        return False
    return _stale(_HOST_PATH, (_SRC_DIR / "host_calls.cpp", _SRC_DIR / "pnm_api.h"))


def needs_build() -> bool:
    return _kernels_need_build() or _host_needs_build()


def _build_host() -> None:
    top = Path(torch.__file__).resolve().parent
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    include = [top / "include", top / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", sysconfig.get_paths()["include"]]
    tmp_out = _LIB_DIR / f"._pnm_host.{os.getpid()}.so.tmp"
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{p}" for p in include], f"-I{_SRC_DIR}", "-o", str(tmp_out), str(_SRC_DIR / "host_calls.cpp"), f"-L{top / 'lib'}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-L{_LIB_DIR}", f"-l:{_LIB_PATH.name}",
           "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{top / 'lib'}"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        if tmp_out.exists():
            tmp_out.unlink()
        raise RuntimeError(f"{cmd[0]} failed:\n{proc.stdout}\n{proc.stderr}")
    os.replace(tmp_out, _HOST_PATH)


def _build_kernels(verbose: bool) -> None:
    nvcc = os.environ.get("NVCC", "nvcc")
    tmp_out = _LIB_DIR / f".libpnm_b200.{os.getpid()}.so.tmp"     # built aside, then moved into place in one step
    cmd = [nvcc, *NVCC_FLAGS, "-o", str(tmp_out), *[str(p) for p in sorted(_SRC_DIR.glob("*.cu"))]]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        if tmp_out.exists():
            tmp_out.unlink()
        raise RuntimeError(f"nvcc failed:\n{proc.stdout}\n{proc.stderr}")
    os.replace(tmp_out, _LIB_PATH)
    if verbose:
        print(proc.stderr)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile what is not up to date (``force``: all) of the kernel library and the host calls in-tree; returns the library's path."""
    if not _SRC_DIR.exists():
        raise FileNotFoundError(f"kernel sources not found at {_SRC_DIR}")
    _LIB_DIR.mkdir(parents=True, exist_ok=True)
    if force or _kernels_need_build():
        _build_kernels(verbose)
    if torch.version.cuda is not None and (force or _host_needs_build()):
        _build_host()                                        # links the library
    return _LIB_PATH


def _declare(lib):
    c = ctypes
    vp, i32, i64 = c.c_void_p, c.c_int, c.c_longlong
    sigs = {
        "pnm_version": ([], i32),
        "pnm_num_sms": ([], i32),
        "pnm_get_error": ([], i32),
        "pnm_reset_error": ([], i32),
        "pnm_gemm_tn_stacked": ([vp, i32, vp, i32, vp, i32, vp, i32, i32, i32, i32, i32, vp, i32, i32, i32, vp], i32),
        "pnm_gemm_nt_stacked": ([vp, i32, vp, i32, vp, vp, i32, i32, i32, i32, i32, vp], i32),
        "pnm_segment_sum": ([vp, i32, vp, vp, vp, i32, i64, i32, i32, i32, vp], i32),
        "pnm_layernorm_bwd_scratch_floats": ([i64, i32], i64),
        "pnm_layernorm_bwd": ([vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, vp], i32),
    }
    for name, (argtypes, restype) in sigs.items():
        try:
            fn = getattr(lib, name)
        except AttributeError:
            continue
        fn.argtypes = argtypes
        fn.restype = restype
    # optional symbols (added by later kernels) declare themselves in their wrappers


def load(required: bool = False):
    """Return the ctypes handle (or ``None`` when unavailable and not required)."""
    global _lib, _load_error
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is not None:
            return _lib
        try:
            if not _LIB_PATH.exists():
                raise FileNotFoundError(f"{_LIB_PATH} not built; run `python -c 'import __graft_entry__ as g; g.build()'`")
            lib = ctypes.CDLL(str(_LIB_PATH))
            _declare(lib)
            _lib = lib
        except Exception as exc:  # noqa: BLE001
            _load_error = str(exc)
            if required:
                raise RuntimeError(f"sm_100a kernel library unavailable: {exc}") from exc
            return None
    return _lib


def host():
    """The extension with the host side of the hottest calls (an error where it is missing: there is no second path)."""
    global _host
    if _host is None:
        import importlib.util

        load(required=True)
        with _lock:
            if _host is None:
                if not _HOST_PATH.exists():
                    raise RuntimeError(f"{_HOST_PATH} not built for this Python and torch; run "
                                       "`python -c 'import __graft_entry__ as g; g.build()'`")
                spec = importlib.util.spec_from_file_location("_pnm_host", _HOST_PATH)
                module = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(module)
                _host = module
    return _host


# absent from CPU builds of torch, where nothing is launched
_raw_stream, _current_device = getattr(torch._C, "_cuda_getCurrentRawStream", None), getattr(torch._C, "_cuda_getDevice", None)


def stream() -> int:
    """Handle of the current CUDA stream: ``torch.cuda.current_stream().cuda_stream`` without the stream object that it builds
    (a few microseconds of every launch)."""
    return _raw_stream(_current_device())


def available() -> bool:
    return load() is not None


def load_error() -> str | None:
    return _load_error

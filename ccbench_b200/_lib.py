"""Loader and builder of the native libraries (in-tree, never JIT-cached).

`libccb.so` holds the host runtime and every fused sm_100a kernel; it is built by
`build_native()` with plain nvcc and loaded with ctypes, so no torch extension and
no JIT cache is involved and the built file travels with the source tree.
"""
from __future__ import annotations

import ctypes
import functools
import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sysconfig
import warnings
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
NATIVE_DIR = Path(__file__).resolve().parent / "_native"
LIBCCB = NATIVE_DIR / "libccb.so"
CALLS, CALLS_SOURCE = NATIVE_DIR / "ccb_calls.so", ROOT / "csrc/py/ccb_calls.cpp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "--threads", "0",
]

RT_SOURCES = ["csrc/rt/ccb_rt.cu", "csrc/rt/ccb_bootstrap.cpp", "csrc/kernels/ccb_standalone.cu",
              "csrc/kernels/ccb_sz.cu", "csrc/kernels/ccb_moe.cu", "csrc/kernels/ccb_noalloc.cu", "csrc/kernels/ccb_pipe.cu",
              "csrc/kernels/ccb_lossless.cu", "csrc/kernels/ccb_local.cu",
              "csrc/kernels/ccb_local_f32.cu", "csrc/kernels/ccb_local_bf16.cu", "csrc/kernels/ccb_local_f16.cu"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libccb.so cannot be built")
    return exe


def _stale(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(s.exists() and s.stat().st_mtime > t for s in sources)


def build_native(force: bool = False, verbose: bool = False) -> Path:
    """Compile libccb.so for sm_100a if it is missing or older than its sources."""
    NATIVE_DIR.mkdir(parents=True, exist_ok=True)
    srcs = [ROOT / s for s in RT_SOURCES if (ROOT / s).exists()]
    deps = srcs + list((ROOT / "csrc").rglob("*.cuh")) + list((ROOT / "csrc").rglob("*.h")) + list((ROOT / "include").rglob("*.h"))
    if force or _stale(LIBCCB, deps):
        cmd = [_nvcc(), *NVCC_FLAGS, f"-I{ROOT / 'include'}", *map(str, srcs), "-o", str(LIBCCB)]
        if verbose:
            print(" ".join(cmd))
        subprocess.run(cmd, check=True, cwd=ROOT)
    return LIBCCB


def _calls_marks() -> list[str]:
    """What the native side of the frequent calls is compiled with and has to hold: the torch and the Python whose objects it
    reads by their layout, and its sources with the C API that it calls (where they are there to look at)."""
    import torch

    marks = [f"torch {torch.__version__} {torch.version.git_version} {importlib.machinery.EXTENSION_SUFFIXES[0]}"]
    if CALLS_SOURCE.exists():
        digest = hashlib.sha256()
        for f in [CALLS_SOURCE, *sorted((ROOT / "include").rglob("*.h"))]:
            digest.update(f.read_bytes())
        marks.append(f"sources {digest.hexdigest()}")
    return marks


def _calls_fit() -> bool:
    if not CALLS.exists():
        return False
    held = CALLS.read_bytes()
    return all(mark.encode() in held for mark in _calls_marks())


def build_calls(force: bool = False, verbose: bool = False) -> Path:
    """Compile the native side of the frequent calls (csrc/py/ccb_calls.cpp) against the torch that is installed, if it
    is missing or made for another torch or of other sources. Processes that build at once each make their own file."""
    import torch

    NATIVE_DIR.mkdir(parents=True, exist_ok=True)
    if force or not _calls_fit():
        home, cuda = Path(torch.__file__).parent, Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
        made = CALLS.with_name(f"{CALLS.name}.{os.getpid()}")
        include = [home / "include", home / "include/torch/csrc/api/include", sysconfig.get_paths()["include"], cuda / "include", ROOT / "include"]
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f'-DCCB_BUILT_FOR="{"; ".join(_calls_marks())}"', *(f"-I{i}" for i in include), str(CALLS_SOURCE), "-o", str(made), f"-L{home / 'lib'}",
               "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", f"-L{cuda / 'lib64'}", "-lcudart"]
        if verbose:
            print(" ".join(cmd))
        subprocess.run(cmd, check=True, cwd=ROOT)
        os.replace(made, CALLS)
    return CALLS


@functools.cache
def calls():
    """The native side of the frequent calls, or None where it cannot be had (made for another torch or of other
    sources, and no compiler to make it again; a libccb.so without what it calls): every call has a way without it, slower
    by some microseconds of the host. Said once."""
    import torch

    from . import constants as K

    try:
        if not _calls_fit():   # before it is loaded: it would read another torch's objects wrongly, not fail
            build_calls()
        spec = importlib.util.spec_from_file_location("ccb_calls", CALLS, loader=importlib.machinery.ExtensionFileLoader("ccb_calls", str(CALLS)))
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        L = lib()
        where = {name: ctypes.cast(getattr(L, name), ctypes.c_void_p).value for name in module.names().split()}
    except (ImportError, OSError, subprocess.CalledProcessError, AttributeError) as e:
        warnings.warn(f"calls from Python take their slower way: {CALLS.name} cannot be used ({e})", RuntimeWarning, stacklevel=2)
        return None
    module.setup(where, K.OPS, K.CODECS, K.ALGOS, torch.nn.Parameter)
    return module


_lib = None


def lib() -> ctypes.CDLL:
    """The loaded libccb.so (built on first use when missing)."""
    global _lib
    if _lib is None:
        if not LIBCCB.exists():
            build_native()
        _lib = ctypes.CDLL(str(LIBCCB))
        _declare(_lib)
    return _lib


def _declare(L: ctypes.CDLL) -> None:
    c_u64, c_int, c_vp = ctypes.c_uint64, ctypes.c_int, ctypes.c_void_p
    pp = ctypes.POINTER(ctypes.c_void_p)
    L.ccb_last_error.restype = ctypes.c_char_p
    L.ccb_launch_count.restype = c_u64
    L.ccb_comm_create.argtypes = [pp, c_int, c_int, ctypes.c_char_p, c_u64, c_int]
    L.ccb_comm_create_local.argtypes = [pp, c_int, c_u64]
    L.ccb_comm_destroy.argtypes = [c_vp]
    for f in ("ccb_comm_rank", "ccb_comm_nranks", "ccb_comm_nlocal", "ccb_comm_has_nvls"):
        getattr(L, f).argtypes = [c_vp]
    L.ccb_comm_arena_bytes.argtypes = [c_vp]
    L.ccb_comm_arena_bytes.restype = c_u64
    L.ccb_comm_set_timeout_ms.argtypes = [c_vp, c_u64]
    L.ccb_comm_set_max_ctas.argtypes = [c_vp, c_int]
    L.ccb_comm_status.argtypes = [c_vp, ctypes.POINTER(ctypes.c_uint32)]
    L.ccb_wire_bytes.argtypes = [c_int, c_int, c_u64]
    L.ccb_wire_bytes.restype = c_u64
    L.ccb_p2p.argtypes = [c_vp, c_vp, c_int, c_vp]
    L.ccb_link_probe.argtypes = [c_vp, c_int, c_int, c_u64, c_vp]
    L.ccb_fold.argtypes = [c_int, c_int, c_vp, c_u64, c_int, c_u64, c_vp, c_vp]
    L.ccb_all_reduce.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, c_int, pp, c_vp]
    L.ccb_reduce_scatter.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, pp, c_vp]
    L.ccb_reduce.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, c_int, c_vp]
    up = ctypes.POINTER(c_u64)
    L.ccb_exchange.argtypes = [c_vp, pp, pp, up, up, up, c_int, c_int, c_vp]
    L.ccb_all_gather.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_vp]
    L.ccb_broadcast.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, c_vp]
    L.ccb_all_to_all.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_vp]
    L.ccb_scatter.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, c_vp]
    L.ccb_gather.argtypes = [c_vp, pp, pp, c_u64, c_int, c_int, c_int, c_vp]

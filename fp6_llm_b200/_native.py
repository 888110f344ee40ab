"""Builds and loads libfp6_b200.so (the CUDA kernels behind the C interface in include/fp6_llm_b200.h) and the extension
fp6_b200_host (the layer call on torch tensors, csrc/torch_host.cpp).

The library is compiled in-tree with nvcc for sm_100a only.  There is no fallback of any kind: if the
library is missing or fails to load, every operator raises.  The extension only shortens the way to it: it is compiled against one
torch and one Python, which its file name carries, and without it the operators reach the same kernels through ctypes.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sysconfig
import warnings

_PKG = os.path.dirname(os.path.abspath(__file__))
_ROOT = os.path.dirname(_PKG)
_CSRC = os.path.join(_PKG, "csrc")
LIB_DIR = os.path.join(_PKG, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libfp6_b200.so")
HOST_SOURCE = "torch_host.cpp"
SOURCES = ("fpx_gemm.cu", "fpx_native.cu", "fpx_prepack.cu", "c_api.cu", "c_api_noalloc.cu")
HEADERS = ("fpx_codes.cuh", "fpx_epilogue.cuh", "fpx_internal.h", "fpx_layout.h", "ptx_sm100.cuh")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--threads", "4",
              "-Xcompiler", "-fPIC", "-shared"]

# every symbol include/fp6_llm_b200.h declares
C_SYMBOLS = (
    "fp6b200_version", "fp6b200_error_string", "fp6b200_linear", "fp6b200_linear_host_io",
    "fp6b200_workspace_bytes", "fp6b200_choose_split_k", "fp6b200_prepack", "fp6b200_prepack_host",
    "fp6b200_dequant", "fp6b200_dequant_host", "fp6b200_dequant_packed", "fp6b200_splitk_reduce",
    "fp6b200_device_status", "fp6b200_linear_static_scratch", "fp6b200_static_scratch_bytes",
    "fp6b200_linear_gather", "fp6b200_set_option", "fp6b200_get_option", "fp6b200_quantize_prepack", "fp6b200_row_scales",
    "fp6b200_linear_host_io_batch", "fp6b200_kernel_launches", "fp6b200_linear_ex", "fp6b200_linear_scratch",
    "fp6b200_native_supported", "fp6b200_native_preferred", "fp6b200_native_weight_bytes", "fp6b200_native_workspace_bytes",
    "fp6b200_native_repack", "fp6b200_linear_native", "fp6b200_native_kernel_launches", "fp6b200_linear_native_gather",
)


class HostCall(ctypes.Structure):
    """fp6b200_host_call of include/fp6_llm_b200.h."""
    _fields_ = [("e_bits", ctypes.c_int), ("m_bits", ctypes.c_int), ("weight_packed_dev", ctypes.c_void_p),
                ("scales_dev", ctypes.c_void_p), ("act_host", ctypes.c_void_p), ("out_host", ctypes.c_void_p),
                ("M", ctypes.c_size_t), ("N", ctypes.c_size_t), ("K", ctypes.c_size_t), ("split_k", ctypes.c_int),
                ("weight_native_dev", ctypes.c_void_p)]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: cannot build libfp6_b200.so")
    return cand


def host_path() -> str:
    """Where the extension for the running torch and Python is: its interface is that of their headers."""
    import torch
    return os.path.join(LIB_DIR, f"fp6_b200_host-torch{torch.__version__}{sysconfig.get_config_var('EXT_SUFFIX')}")


def _stale(path: str, sources) -> bool:
    if not os.path.exists(path):
        return True
    built = os.path.getmtime(path)
    deps = [os.path.join(_CSRC, f) for f in sources]
    deps += [os.path.join(_ROOT, "include", f) for f in ("fp6_llm_b200.h", "fp6_llm_b200_cxx.cuh")]
    return any(os.path.getmtime(d) > built for d in deps)


def _run(what: str, cmd) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + res.stdout + res.stderr)
    return res.stderr


def _build_host() -> None:
    """The Python binding of the layer call: plain C++ against torch's headers, linked to the library beside it."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-o", host_path(), os.path.join(_CSRC, HOST_SOURCE)]
    for inc in (os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]):
        cmd += ["-isystem", inc]
    cmd += ["-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python",
            "-L" + LIB_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN"]
    _run("g++", cmd)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library and its Python binding if they are missing or older than their sources.  Returns the library's
    path."""
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or _stale(LIB_PATH, SOURCES + HEADERS):
        cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH]
        out = _run("nvcc", cmd + [os.path.join(_CSRC, s) for s in SOURCES])
        if verbose:
            print(out)
    if force or _stale(host_path(), (HOST_SOURCE,)):
        _build_host()
    return LIB_PATH


_lib = None


def lib() -> ctypes.CDLL:
    """The loaded library with argument types set.  Raises if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise RuntimeError(
            f"{LIB_PATH} is missing: build it first (python -c 'import __graft_entry__ as g; g.build()' "
            "or fp6_llm_b200.build()); there is no fallback path")
    L = ctypes.CDLL(LIB_PATH)
    vp, sz, ci = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int
    L.fp6b200_version.restype = ci
    L.fp6b200_version.argtypes = []
    L.fp6b200_error_string.restype = ctypes.c_char_p
    L.fp6b200_error_string.argtypes = [ci]
    L.fp6b200_linear.restype = ci
    L.fp6b200_linear.argtypes = [ci, ci, vp, vp, vp, vp, vp, sz, sz, sz, vp, ci]
    L.fp6b200_linear_ex.restype = ci
    L.fp6b200_linear_ex.argtypes = [ci, ci, vp, vp, vp, vp, vp, sz, sz, sz, vp, ci, vp, ci]
    L.fp6b200_linear_scratch.restype = ci
    L.fp6b200_linear_scratch.argtypes = [ci, ci, vp, vp, vp, vp, vp, sz, sz, sz, vp, vp, vp, ci]
    L.fp6b200_native_supported.restype = ci
    L.fp6b200_native_supported.argtypes = [ci, ci, sz, sz, sz]
    L.fp6b200_native_preferred.restype = ci
    L.fp6b200_native_preferred.argtypes = [ci, ci, sz, sz, sz]
    L.fp6b200_native_weight_bytes.restype = sz
    L.fp6b200_native_weight_bytes.argtypes = [sz, sz]
    L.fp6b200_native_workspace_bytes.restype = sz
    L.fp6b200_native_workspace_bytes.argtypes = [sz, sz]
    L.fp6b200_native_repack.restype = ci
    L.fp6b200_native_repack.argtypes = [ci, ci, vp, vp, vp, sz, sz]
    L.fp6b200_linear_native.restype = ci
    L.fp6b200_linear_native.argtypes = [ci, ci, vp, vp, vp, vp, vp, sz, sz, sz, vp, vp, ci]
    L.fp6b200_linear_native_gather.restype = ci
    L.fp6b200_linear_native_gather.argtypes = [ci, ci, vp, vp, vp, vp, vp, vp, vp, ci, ci, sz, sz, sz, sz, sz, vp]
    L.fp6b200_native_kernel_launches.restype = ci
    L.fp6b200_native_kernel_launches.argtypes = [sz, sz, sz]
    L.fp6b200_linear_host_io.restype = ci
    L.fp6b200_linear_host_io.argtypes = [ci, ci, vp, vp, vp, vp, sz, sz, sz, ci]
    L.fp6b200_linear_host_io_batch.restype = ci
    L.fp6b200_linear_host_io_batch.argtypes = [ctypes.POINTER(HostCall), ci]
    L.fp6b200_kernel_launches.restype = ci
    L.fp6b200_kernel_launches.argtypes = [sz, sz, sz, ci]
    L.fp6b200_workspace_bytes.restype = sz
    L.fp6b200_workspace_bytes.argtypes = [sz, sz, sz, ci]
    L.fp6b200_choose_split_k.restype = ci
    L.fp6b200_choose_split_k.argtypes = [sz, sz, sz, ci]
    L.fp6b200_prepack.restype = ci
    L.fp6b200_prepack.argtypes = [ci, ci, vp, vp, vp, sz, sz]
    L.fp6b200_prepack_host.restype = ci
    L.fp6b200_prepack_host.argtypes = [ci, ci, vp, vp, sz, sz]
    L.fp6b200_dequant.restype = ci
    L.fp6b200_dequant.argtypes = [ci, ci, vp, vp, vp, vp, sz, sz]
    L.fp6b200_dequant_host.restype = ci
    L.fp6b200_dequant_host.argtypes = [ci, ci, vp, vp, sz, sz, vp]
    L.fp6b200_dequant_packed.restype = ci
    L.fp6b200_dequant_packed.argtypes = [ci, ci, vp, vp, vp, vp, sz, sz]
    L.fp6b200_splitk_reduce.restype = ci
    L.fp6b200_splitk_reduce.argtypes = [vp, vp, vp, sz, ci]
    L.fp6b200_linear_static_scratch.restype = ci
    L.fp6b200_linear_static_scratch.argtypes = [ci, ci, vp, vp, vp, vp, vp, sz, sz, sz]
    L.fp6b200_static_scratch_bytes.restype = sz
    L.fp6b200_static_scratch_bytes.argtypes = []
    L.fp6b200_linear_gather.restype = ci
    L.fp6b200_linear_gather.argtypes = [ci, ci, vp, vp, vp, vp, vp, vp, vp, ci, ci, sz, sz, sz, sz, sz, vp, ci]
    L.fp6b200_set_option.restype = ci
    L.fp6b200_set_option.argtypes = [ci, ci]
    L.fp6b200_get_option.restype = ci
    L.fp6b200_get_option.argtypes = [ci]
    L.fp6b200_quantize_prepack.restype = ci
    L.fp6b200_quantize_prepack.argtypes = [ci, ci, vp, vp, vp, vp, sz, sz]
    L.fp6b200_row_scales.restype = ci
    L.fp6b200_row_scales.argtypes = [vp, vp, vp, sz, sz, ctypes.c_float]
    L.fp6b200_device_status.restype = ci
    L.fp6b200_device_status.argtypes = [ctypes.POINTER(ci)]
    _lib = L
    return L


class _PythonForm:
    """Stands in for the extension: every call is left to the Python form of the same operator."""
    linear = native = layer = host_batch = unwatched = staticmethod(lambda *args: NotImplemented)


_host = None


def host():
    """The native host side of the layer call (csrc/torch_host.cpp); where it has not been built for this torch and Python, or does
    not load, a warning and a stand-in that declines every call."""
    global _host
    if _host is None:
        lib()
        import torch  # noqa: F401  (its libraries must be loaded first)
        path = host_path()
        try:
            loader = importlib.machinery.ExtensionFileLoader("fp6_b200_host", path)
            module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("fp6_b200_host", path, loader=loader))
            loader.exec_module(module)
        except ImportError as e:
            warnings.warn(f"no native host side for the layer calls ({e}): they go through ctypes, 20 - 30 us slower each; "
                          "fp6_llm_b200.build() compiles it", RuntimeWarning, stacklevel=3)
            module = _PythonForm
        _host = module
    return _host


def check(code: int, what: str) -> None:
    if code != 0:
        msg = lib().fp6b200_error_string(code)
        raise RuntimeError(f"{what} failed: CUDA error {code} ({msg.decode() if msg else '?'})")

"""ctypes binding of libaccelgcn.so -- the C ABI declared in include/accelgcn.h.

The library is the product; this module only loads it and declares the
prototypes.  There is no fallback of any kind: if the shared object is missing
or fails to load, importing a function from here raises.
"""
from __future__ import annotations

import ctypes
import functools
import importlib.machinery
import importlib.util
import os
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
DEFAULT_LIB = os.path.join(os.path.dirname(_HERE), "lib", "libaccelgcn.so")

OK, ERR_INVALID, ERR_CUDA, ERR_CAPACITY, ERR_RANGE = 0, -1, -2, -3, -4
DEG_BOUND = 384
PARTITION_NOALLOC_MAX_ROWS = 1 << 24

_vp, _i64, _int = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int

# name -> (restype, argtypes); every symbol include/accelgcn.h declares
PROTOTYPES = {
    "agcn_last_error": (ctypes.c_char_p, []),
    "agcn_version": (_int, []),
    "agcn_release_scratch": (_int, []),
    "agcn_partition_device": (_int, [_vp, _i64, _vp, _i64, ctypes.POINTER(_i64), _vp]),
    "agcn_partition_begin": (_int, [_vp, _i64, ctypes.POINTER(_vp), ctypes.POINTER(_i64), _vp]),
    "agcn_partition_finish": (_int, [_vp, _vp]),
    "agcn_partition_host": (_int, [_vp, _i64, _vp, _i64, ctypes.POINTER(_i64)]),
    "agcn_partition_device_noalloc": (_int, [_vp, _i64, _vp, _i64, ctypes.POINTER(_i64), _vp]),
    "agcn_degree_sort_device": (_int, [_vp, _vp, _vp, _i64, _i64, _int, _vp, _vp, _vp, _vp, _vp]),
    "agcn_degree_sort_host": (_int, [_vp, _vp, _vp, _i64, _i64, _int, _vp, _vp, _vp, _vp]),
    "agcn_spmm_create": (_int, [ctypes.POINTER(_vp), _vp, _i64, _vp, _i64, _i64, _i64, _vp]),
    "agcn_spmm_run": (_int, [_vp, _vp, _vp, _vp, _i64, _vp, _i64, _int, _vp]),
    "agcn_spmm_run_act": (_int, [_vp, _vp, _vp, _vp, _i64, _vp, _i64, _int, _int, _vp]),
    "agcn_spmm_once": (_int, [_vp, _i64, _vp, _vp, _i64, _i64, _i64, _vp, _i64, _vp, _i64, _int, _vp]),
    "agcn_spmm_destroy": (_int, [_vp]),
    "agcn_gemm_tf32": (_int, [_vp, _i64, _vp, _vp, _i64, _i64, _int, _int, _vp]),
    "agcn_spmm_plan_info": (_int, [_vp, ctypes.POINTER(_i64), ctypes.POINTER(_i64), ctypes.POINTER(_i64),
                                  ctypes.POINTER(_int)]),
    "agcn_spmm_plan_hot_column": (_int, [_vp, _int, ctypes.POINTER(_i64)]),
    "agcn_host_ctx_create": (_int, [ctypes.POINTER(_vp)]),
    "agcn_host_ctx_destroy": (_int, [_vp]),
    "agcn_host_set_graph": (_int, [_vp, _vp, _i64, _vp, _vp, _i64, _i64, _i64]),
    "agcn_host_spmm": (_int, [_vp, _vp, _vp, _int]),
    "agcn_spmm_host": (_int, [_vp, _vp, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _int]),
    "agcn_host_spmm_batch": (_int, [_vp, _int, _vp, _vp, _vp]),
    "agcn_spmm_host_batch": (_int, [_vp, _vp, _i64, _vp, _vp, _i64, _i64, _i64, _int, _vp, _vp, _vp]),
    "agcn_host_last_timing": (_int, [_vp, _vp]),
    "agcn_spmm_tiled_create": (_int, [ctypes.POINTER(_vp), _vp, _vp, _vp, _i64, _i64, _i64, _vp, _int, _vp]),
    "agcn_spmm_tiled_run": (_int, [_vp, _vp, _i64, _vp, _i64, _int, _int, _vp]),
    "agcn_spmm_tiled_run_range": (_int, [_vp, _int, _vp, _i64, _vp, _i64, _int, _int, _vp]),
    "agcn_spmm_tiled_destroy": (_int, [_vp]),
    "agcn_spmm_tiled_info": (_int, [_vp, ctypes.POINTER(_int), ctypes.POINTER(_i64), _vp, ctypes.POINTER(_int)]),
    "agcn_spmm_tiled_suggest": (_int, [_i64, _i64, _i64, _int]),
    "agcn_gemm_tf32_async": (_int, [_vp, _i64, _vp, _vp, _i64, _i64, _int, _int, _vp, _vp]),
    "agcn_gemm_tf32_pair_async": (_int, [_vp, _vp, _vp, _vp, _i64, _vp, _vp]),
    "agcn_gemm_tf32_selftest_timeout": (_int, [_vp, _i64, _vp, _vp, _i64, _i64, _vp]),
    "agcn_gemm_tf32_pair_selftest_timeout": (_int, [_vp, _vp, _vp, _vp, _i64, _vp]),
    "agcn_gcn_fused_layer": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _vp, _vp]),
    "agcn_balanced_blocks": (_int, [_vp, _i64, _int, _vp, ctypes.POINTER(_i64)]),
    "agcn_dist_unique_id": (_int, [_vp]),
    "agcn_dist_create": (_int, [ctypes.POINTER(_vp), _int, _int, _vp]),
    "agcn_dist_destroy": (_int, [_vp]),
    "agcn_dist_set_graph": (_int, [_vp, _vp, _vp, _vp, _i64, _i64, _int, _int, _vp]),
    "agcn_dist_info": (_int, [_vp, ctypes.POINTER(_i64), ctypes.POINTER(_i64), ctypes.POINTER(_i64),
                             ctypes.POINTER(_i64), ctypes.POINTER(_int), ctypes.POINTER(_int)]),
    "agcn_dist_block_rows": (_int, [_vp, _int, _vp, _vp]),
    "agcn_dist_gather_begin": (_int, [_vp, _int, _vp, _int, _vp]),
    "agcn_dist_spmm_gathered": (_int, [_vp, _int, _vp, _int, _int, _vp]),
    "agcn_dist_spmm_step": (_int, [_vp, _vp, _vp, _int, _int, _vp]),
    "agcn_dist_wait_gathered": (_int, [_vp, _int, _vp]),
    "agcn_dist_spmm_on_gathered": (_int, [_vp, _vp, _vp, _int, _int, _vp]),
    "agcn_dist_gathered": (_int, [_vp, _int, ctypes.POINTER(_vp), ctypes.POINTER(_i64)]),
    "agcn_gcn2_forward_create": (_int, [ctypes.POINTER(_vp), _vp, _vp, _vp]),
    "agcn_gcn2_forward_run": (_int, [_vp, _vp, _vp, _vp]),
    "agcn_gcn2_forward_status": (_int, [_vp, _vp]),
    "agcn_gcn2_forward_launches": (_int, [_vp, ctypes.POINTER(_int)]),
    "agcn_gcn2_forward_paired": (_int, [_vp, ctypes.POINTER(_int)]),
    "agcn_gcn2_forward_destroy": (_int, [_vp]),
    "agcn_probe_gather_bandwidth": (_int, [_i64, _int, _i64, _int, _int, ctypes.POINTER(ctypes.c_double)]),
}
DIST_ID_BYTES = 128
MAX_WORLD = 64

_lib = None
_call = None


class AccelGcnError(RuntimeError):
    """A call into libaccelgcn.so returned a negative status."""

    def __init__(self, code: int, message: str):
        super().__init__(f"libaccelgcn error {code}: {message}")
        self.code = code


def lib_path() -> str:
    return os.environ.get("ACCELGCN_LIB", DEFAULT_LIB)


def load():
    """Load the shared library (once) and declare every prototype."""
    global _lib
    if _lib is None:
        path = lib_path()
        if not os.path.exists(path):
            raise FileNotFoundError(
                f"{path} not found: build it with `python iccad-accel-gcn_b200/build.py` "
                "(there is no CPU or PyTorch fallback for this library)")
        lib = ctypes.CDLL(path)
        for name, (res, args) in PROTOTYPES.items():
            fn = getattr(lib, name)          # AttributeError if the symbol is not exported
            fn.restype, fn.argtypes = res, args
        _lib = lib
    return _lib


def call():
    """The native caller `call(address, *integers) -> int` (csrc/pycall.c): what the hot paths use in place of
    ctypes.  No fallback: it is built with the library."""
    global _call
    if _call is None:
        path = os.path.join(os.path.dirname(DEFAULT_LIB), "agcn_call" + sysconfig.get_config_var("EXT_SUFFIX"))
        if not os.path.exists(path):
            raise FileNotFoundError(f"{path} not found: build it with `python iccad-accel-gcn_b200/build.py` under this Python")
        loader = importlib.machinery.ExtensionFileLoader("agcn_call", path)
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("agcn_call", loader))
        loader.exec_module(module)
        _call = module.call
    return _call


@functools.lru_cache(maxsize=None)
def address(name: str) -> int:
    """Address of a library function, for `call`."""
    return ctypes.cast(getattr(load(), name), ctypes.c_void_p).value


def raw_stream(index: int) -> int:
    """The cudaStream_t of the current stream of device `index` (torch.cuda.current_stream builds an object for it)."""
    import torch
    return torch._C._cuda_getCurrentRawStream(index)


class _Here:
    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_HERE_ALREADY = _Here()


def on_device(index: int):
    """Makes device `index` current for a `with` block; nothing is done where it already is."""
    import torch
    return _HERE_ALREADY if torch._C._cuda_getDevice() == index else torch.cuda.device(index)


def device_index(device) -> int:
    import torch
    return device.index if device.index is not None else torch.cuda.current_device()


def release_scratch() -> None:
    """Gives back what the library keeps between calls: the current device's scratch pool (up to 2 GB, which torch's
    allocator does not see) and the pinned pieces of the host copies.  Waits for the device."""
    check(load().agcn_release_scratch())


def check(code: int) -> None:
    if code != OK:
        raise AccelGcnError(code, load().agcn_last_error().decode("utf-8", "replace"))

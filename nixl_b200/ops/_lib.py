"""ctypes access to ``libnixl_kernels.so`` (the fused sm_100a kernels with a C ABI).

The library is built in-tree by ``make -C csrc``.  Importing this module on a machine with a
GPU but without the library is an error: the ops never fall back to eager PyTorch.
"""
import ctypes
import os

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(os.path.dirname(_HERE), "lib", "libnixl_kernels.so")

_lib = None


def lib() -> ctypes.CDLL:
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise ImportError(f"{LIB_PATH} is missing; build it with `make -C csrc -j8`")
        _lib = ctypes.CDLL(LIB_PATH)
    return _lib


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise RuntimeError(f"{what} failed with CUDA error {rc}")


def raw_stream(device: torch.device) -> ctypes.c_void_p:
    """The current stream's ``cudaStream_t`` on a device (torch's raw accessor: 0.2 us, where the Stream object takes 2)."""
    get = getattr(torch._C, "_cuda_getCurrentRawStream", None)
    if get is None:
        return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)
    return ctypes.c_void_p(get(device.index if device.index is not None else torch.cuda.current_device()))


def launch_on(device: torch.device, fn, ref, stream: ctypes.c_void_p, what: str) -> None:
    """Calls a launcher with ``device`` current; entering the device context costs half a launch, so only when needed."""
    if device.index is None or torch.cuda.current_device() == device.index:
        rc = fn(ref, stream)
    else:
        with torch.cuda.device(device):
            rc = fn(ref, stream)
    check(rc, what)


def read_u64(address: int) -> int:
    """Volatile read of a host word (a pinned flag written by a kernel)."""
    return ctypes.c_uint64.from_address(address).value

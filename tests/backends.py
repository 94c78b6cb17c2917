"""Where the test buffers live: CUDA tensors for the real library, numpy arrays for the
g++-compiled emulation build (tests/emu).  Both expose the same four calls so a parity case
is written once and runs through the same C ABI on either."""
from __future__ import annotations

import ctypes as C
import os
import sys

import numpy as np

from cerium_b200 import _capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class EmuBackend:
    """Kernel sources compiled for the host (index arithmetic / orchestration checks)."""

    name = "emu"

    def __init__(self):
        sys.path.insert(0, os.path.join(ROOT, "tests", "emu"))
        import build_emu
        self.lib = _capi.Library(build_emu.build())
        self._keep = []

    def to_dev(self, a: np.ndarray):
        b = self.empty(a.shape, a.dtype)
        b[...] = a
        return b

    def empty(self, shape, dtype):
        # as aligned as an allocation on the device: numpy's own lie 16 bytes past a page
        count = int(np.prod(shape))
        raw = np.zeros(count * np.dtype(dtype).itemsize + 256, dtype=np.uint8)
        at = -raw.ctypes.data % 256
        return raw[at:at + count * np.dtype(dtype).itemsize].view(dtype).reshape(shape)

    def ptr(self, buf) -> int:
        return buf.ctypes.data

    def to_host(self, buf) -> np.ndarray:
        return buf.copy()

    def sync(self):
        pass

    def launches(self, call) -> int:
        """Kernels that call(stream) launches."""
        count = self.lib.dll.cerium_emu_launches
        count.restype = C.c_long
        before = count()
        call(0)
        return count() - before


class CudaBackend:
    """The shipped CUDA library on cuda:0."""

    name = "cuda"

    def __init__(self):
        import torch
        self.torch = torch
        if not torch.cuda.is_available():
            raise RuntimeError("CUDA backend requested without a GPU")
        self.lib = _capi.load()
        self.dev = torch.device("cuda:0")

    def _tdtype(self, dtype):
        return {np.dtype(np.uint64): self.torch.int64, np.dtype(np.uint32): self.torch.int32}[np.dtype(dtype)]

    def to_dev(self, a: np.ndarray):
        a = np.ascontiguousarray(a)
        signed = a.view(np.int64 if a.dtype == np.uint64 else np.int32)
        return self.torch.from_numpy(signed.copy()).to(self.dev)

    def empty(self, shape, dtype):
        return self.torch.zeros(shape, dtype=self._tdtype(dtype), device=self.dev)

    def ptr(self, buf) -> int:
        return buf.data_ptr()

    def to_host(self, buf) -> np.ndarray:
        self.torch.cuda.synchronize()
        a = buf.cpu().numpy()
        return a.view(np.uint64 if a.dtype == np.int64 else np.uint32).copy()

    def sync(self):
        self.torch.cuda.synchronize()

    def launches(self, call) -> int:
        """Kernels that call(stream) launches: captured into a graph and counted, not run."""
        from cuda.bindings import runtime as rt
        stream = self.torch.cuda.Stream()
        (err,) = rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
        assert err == rt.cudaError_t.cudaSuccess, err
        try:
            call(stream.cuda_stream)
        finally:
            err, graph = rt.cudaStreamEndCapture(stream.cuda_stream)
        assert err == rt.cudaError_t.cudaSuccess, err
        err, _, count = rt.cudaGraphGetNodes(graph)
        assert err == rt.cudaError_t.cudaSuccess, err
        rt.cudaGraphDestroy(graph)
        return count

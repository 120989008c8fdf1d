"""For tests that look at what an op hands to its kernel without a GPU: CPU tensors that take the ops' CUDA branch, and
the native library with the launches replaced by a recorder."""
import ctypes

import torch


class AsCuda(torch.Tensor):
    """A CPU tensor that takes the CUDA branch of the ops."""
    is_cuda = True


def as_cuda(t):
    return torch.Tensor._make_subclass(AsCuda, t)


class Recorder:
    """``lib``, except that the GEMM launches only leave a copy of their argument block in ``calls``."""

    def __init__(self, lib):
        self._lib, self.calls = lib, []

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def _keep(self, ref):
        kept = type(ref._obj)()
        ctypes.memmove(ctypes.byref(kept), ref, ctypes.sizeof(kept))
        self.calls.append(kept)
        return 0

    fluxb_dense_gemm = fluxb_ulysses_gemm = fluxb_moe_grouped_gemm = _keep


def record_launches():
    """Installs a recorder for the rest of the process (for ranks that run in a process of their own)."""
    from tempname_new_b200 import _native
    from tempname_new_b200.ops import _dense
    rec = Recorder(_native.lib())
    _native.lib, _dense.current_stream_ptr = lambda: rec, lambda device=None: 0
    return rec

"""Helpers for the GPU parity tests (skip when no CUDA device)."""
import pytest

torch = pytest.importorskip("torch")


def own_stream():
    """A stream outside torch's round-robin pool, so that no later test is given
    it (and the library handle with grown scratch that belongs to it)."""
    import ctypes
    cu = ctypes.CDLL("libcuda.so.1")
    torch.cuda.current_stream().synchronize()
    s = ctypes.c_void_p()
    assert cu.cuStreamCreate(ctypes.byref(s), 1) == 0      # non-blocking
    return torch.cuda.ExternalStream(s.value)


def need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sslablu_gb300 import _lib
    _lib.lib()  # raises if libslablu.so is missing: no silent fallback

"""The library in a second driver context of the device: its contractions run in
either, and alternating between the two does not keep more and more memory."""
import ctypes

import numpy as np
import pytest

from pyheartsim_b200 import _lib

pytestmark = pytest.mark.gpu


class _Context:
    """A driver context of device 0 of its own, current inside ``with``."""

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.h = ctypes.c_void_p()
        self._do("cuInit", 0)
        self._do("cuCtxCreate_v2", ctypes.byref(self.h), ctypes.c_uint(0), ctypes.c_int(0))
        self._do("cuCtxPopCurrent_v2", ctypes.byref(ctypes.c_void_p()))

    def _do(self, name, *a):
        rc = getattr(self.cu, name)(*a)
        assert rc == 0, f"{name}: {rc}"

    def __enter__(self):
        self._do("cuCtxPushCurrent_v2", self.h)
        return self

    def __exit__(self, *a):
        self._do("cuCtxPopCurrent_v2", ctypes.byref(ctypes.c_void_p()))

    def put(self, a):
        p = ctypes.c_uint64()
        self._do("cuMemAlloc_v2", ctypes.byref(p), ctypes.c_size_t(a.nbytes))
        self._do("cuMemcpyHtoD_v2", p, ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.nbytes))
        return p

    def get(self, p, like):
        out = np.empty_like(like)
        self._do("cuCtxSynchronize")
        self._do("cuMemcpyDtoH_v2", ctypes.c_void_p(out.ctypes.data), p, ctypes.c_size_t(out.nbytes))
        return out

    def free_bytes(self):
        f, t = ctypes.c_size_t(), ctypes.c_size_t()
        self._do("cuCtxSynchronize")
        self._do("cuMemGetInfo_v2", ctypes.byref(f), ctypes.byref(t))
        return f.value

    def destroy(self):
        self._do("cuCtxDestroy_v2", self.h)


def _contract(V, M, out):
    """egm = V M^T of device arrays given by address, on the default stream."""
    T, n, ne = 600, 4000, 512
    _lib.check(_lib.lib().phs_egm_contract_f64(T, n, ne, V, n, M, out, None), "phs_egm_contract_f64")


def test_contractions_in_two_contexts(cuda_device):
    import torch
    rng = np.random.default_rng(0)
    V, M = rng.normal(size=(600, 4000)), rng.normal(size=(512, 4000))
    want = V @ M.T
    tv, tm = torch.as_tensor(V, device=cuda_device), torch.as_tensor(M, device=cuda_device)
    to = torch.empty((600, 512), dtype=torch.float64, device=cuda_device)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _contract(p(tv), p(tm), p(to))                     # the process's context first
    np.testing.assert_allclose(to.cpu().numpy(), want, rtol=0, atol=1e-10)
    ctx = _Context()
    try:
        with ctx:
            dv, dm, do = ctx.put(V), ctx.put(M), ctx.put(np.zeros_like(want))
            _contract(ctypes.c_void_p(dv.value), ctypes.c_void_p(dm.value), ctypes.c_void_p(do.value))
            # rounding of 4000 terms of size 1 in another order
            np.testing.assert_allclose(ctx.get(do, want), want, rtol=0, atol=1e-10)
            free = ctx.free_bytes()
        for _ in range(50):                            # each takes some 10 MB of partial sums
            _contract(p(tv), p(tm), p(to))
            torch.cuda.synchronize()
            with ctx:
                _contract(ctypes.c_void_p(dv.value), ctypes.c_void_p(dm.value), ctypes.c_void_p(do.value))
                ctx.get(do, want)
        with ctx:
            # one pool each: nothing grows with the number of switches (a pool keeps 32 MB steps)
            assert free - ctx.free_bytes() < 200 << 20
    finally:
        ctx.destroy()
    _contract(p(tv), p(tm), p(to))
    np.testing.assert_allclose(to.cpu().numpy(), want, rtol=0, atol=1e-10)

"""The device pointers that the engine hands out can be exported to other
processes, and handing them out changes nothing about the run."""
import ctypes

import numpy as np
import pytest

from pyheartsim_b200 import _lib
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.instance import compile_instance
from tests import gpu_cases

pytestmark = pytest.mark.gpu


def _cudart():
    import torch  # noqa: F401  (loads the runtime)
    with open("/proc/self/maps") as f:
        paths = {line.split()[-1] for line in f if "libcudart.so" in line}
    if not paths:
        pytest.skip("no shared CUDA runtime in the process")
    return ctypes.CDLL(sorted(paths)[0])


def _handle(rt, ptr):
    h = (ctypes.c_char * 64)()
    rt.cudaIpcGetMemHandle.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    rc = rt.cudaIpcGetMemHandle(ctypes.byref(h), ctypes.c_void_p(ptr))
    rt.cudaGetLastError()
    return rc, bytes(h)


def _ptrs(eng, slot):
    p = [ctypes.c_void_p(), ctypes.c_void_p(), _lib.c_int32_p()]
    _lib.check(_lib.lib().phs_instance_device_ptrs(eng._h, slot, *(ctypes.byref(x) for x in p)),
               "phs_instance_device_ptrs")
    return [p[0].value, p[1].value, ctypes.cast(p[2], ctypes.c_void_p).value]


@pytest.mark.parametrize("fast", [True, False])
def test_pointers_can_be_exported(fast, cuda_device):
    import torch
    rt = _cudart()
    x = torch.zeros(1 << 20, device=cuda_device)
    if _handle(rt, x.data_ptr())[0] != 0:
        pytest.skip("no inter-process handles on this machine")
    (n, P, geom, sp, ap), pdur = gpu_cases.small_shell_ms()
    kw = dict(full_cycles=False, tol=1e-7, restart=20) if fast else {}
    inst = compile_instance(n, P, geom, dict(sp), dict(ap), pacing_duration=pdur, max_steps=60, **kw)
    prec = _lib.PREC_F32 if fast else _lib.PREC_F64
    with BatchedEngine(prec) as plain, BatchedEngine(prec) as eng:
        s, r = eng.add(inst), plain.add(inst)
        other = eng.add(inst)                          # its arrays stay where they are
        for e in (eng, plain):
            e.advance(30)
        p = _ptrs(eng, s)
        handles = [_handle(rt, q) for q in p]
        assert [rc for rc, _ in handles] == [0, 0, 0]
        assert len({h for _, h in handles}) == 3 or len(set(p)) == 3
        for e in (eng, plain):
            e.advance(30)
        assert _ptrs(eng, s) == p                      # stable from then on

        class _U:
            __cuda_array_interface__ = {"data": (p[0], False), "shape": (n,), "typestr": "<f4" if fast else "<f8",
                                        "version": 3, "strides": None}

        u_dev = inst.to_caller(torch.as_tensor(_U(), device=cuda_device).cpu().numpy())
        want = plain.state(r)
        np.testing.assert_array_equal(u_dev, want[0])
        for k in (s, other):
            for a, b in zip(eng.state(k), want):
                np.testing.assert_array_equal(a, b)
            np.testing.assert_array_equal(eng.history(k), plain.history(r))
            np.testing.assert_array_equal(eng.history_host(k), plain.history(r))
        eng.remove(s)
        np.testing.assert_array_equal(eng.state(other)[0], want[0])

"""Engines advanced on streams that do not wait for the legacy stream, on which
the engine allocates and fills its launch plans: every plan (one per change of
the instance set, per automatic re-split and per tile length) is in place when
the launch reads it."""
import numpy as np
import pytest

from pyheartsim_b200 import _lib
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.instance import compile_instance
from tests import gpu_cases

pytestmark = pytest.mark.gpu


def _instances(steps):
    out = []
    for name in ("sheet_ms", "slab_ap", "small_shell_ms", "small_shell_ms_fibres"):
        (n, P, geom, sp, ap), pdur = getattr(gpu_cases, name)()
        out.append(compile_instance(n, P, geom, dict(sp), dict(ap), pacing_duration=pdur, max_steps=steps,
                                    full_cycles=False, tol=1e-7, restart=20))
    return out


def _run(insts, stream, launches, per):
    """Instances that come one by one, a few steps after each change of the plan."""
    with BatchedEngine(_lib.PREC_F32) as eng:
        slots = []
        for x in insts:
            slots.append(eng.add(x))
            eng.advance(per, stream=stream, sync=False)
            eng.configure(variant=3)                  # another plan, nothing waited for in between
            eng.advance(per, stream=stream, sync=False)
            eng.configure(variant=-1)
        for _ in range(launches):
            eng.advance(per, stream=stream, sync=True)
        return [eng.state(s) for s in slots]


def test_plans_on_a_non_blocking_stream(cuda_device):
    import torch
    insts = _instances(60)
    want = _run(insts, torch.cuda.default_stream(), 30, 3)
    stream = torch.cuda.Stream()                      # does not wait for the legacy stream
    for _ in range(3):
        for a, b in zip(_run(insts, stream, 30, 3), want):
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x, y)

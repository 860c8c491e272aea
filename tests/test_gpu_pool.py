"""Instances placed in device memory that earlier instances used: the results
do not depend on what the memory held before."""
import numpy as np
import pytest

from pyheartsim_b200 import _lib
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.instance import compile_instance
from tests import gpu_cases

pytestmark = pytest.mark.gpu


def _instance(case, fast, steps):
    (n, P, geom, sp, ap), pdur = getattr(gpu_cases, case)()
    kw = dict(full_cycles=False, tol=1e-7, restart=20) if fast else {}
    return compile_instance(n, P, geom, dict(sp), dict(ap), pacing_duration=pdur, max_steps=steps, **kw)


def _run(eng, inst, steps):
    s = eng.add(inst)
    eng.advance(steps)
    out = (eng.history(s), *eng.state(s))
    eng.remove(s)
    return out


@pytest.mark.parametrize("fast", [True, False])
def test_reused_memory_gives_the_same_results(fast, cuda_device):
    steps = 60 if fast else 10
    prec = _lib.PREC_F32 if fast else _lib.PREC_F64
    names = ["small_shell_ms", "slab_ap", "small_shell_ms_fibres", "sheet_ms"]
    insts = [_instance(c, fast, steps) for c in names]
    first = []
    for x in insts:                       # each in an engine of its own
        with BatchedEngine(prec) as eng:
            first.append(_run(eng, x, steps))
    with BatchedEngine(prec) as eng:      # one after another in one engine, largest and smallest alternating
        for k in (0, 1, 2, 3, 0, 2, 1, 0):
            for a, b in zip(_run(eng, insts[k], steps), first[k]):
                np.testing.assert_array_equal(a, b)

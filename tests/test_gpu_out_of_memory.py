"""A call that finds no device memory fails by itself: the next ones run."""
import numpy as np
import pytest

from pyheartsim_b200 import _lib
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.instance import compile_instance
from tests import gpu_cases

pytestmark = pytest.mark.gpu


def _instance():
    (n, P, geom, sp, ap), pdur = gpu_cases.sheet_ms()
    return compile_instance(n, P, geom, dict(sp), dict(ap), pacing_duration=pdur, max_steps=40, full_cycles=False,
                            tol=1e-7, restart=20)


def test_an_instance_too_large_leaves_the_engine_as_it_was(cuda_device):
    huge = _instance()
    huge.n_samples = 1 << 30                       # a history of 6.9 TB
    with BatchedEngine(_lib.PREC_F32) as eng, BatchedEngine(_lib.PREC_F32) as other:
        a = eng.add(_instance())
        with pytest.raises(_lib.PhsError) as e:
            eng.add(huge)
        assert e.value.status == _lib.PHS_ERR_OOM
        b = eng.add(_instance())                   # the first call after it
        eng.advance(40)
        c = other.add(_instance())
        other.advance(40)
        for x, y, z in zip(eng.state(a), eng.state(b), other.state(c)):
            np.testing.assert_array_equal(x, z)
            np.testing.assert_array_equal(y, z)

"""Device memory of removed instances and closed engines, beyond what the
library's pool keeps, is free for other allocators when the call returns."""
import pytest

from pyheartsim_b200 import _lib, synthetic
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.instance import compile_instance

pytestmark = pytest.mark.gpu

KEEP_ENGINE, KEEP_IDLE = 4 << 30, 512 << 20      # the pool's bounds
SLACK = 128 << 20                                # tables, and the driver's 32 MB steps


def test_memory_is_given_back(cuda_device):
    import torch
    free = lambda: torch.cuda.mem_get_info(cuda_device)[0]
    ijk = synthetic.sheet(200, 200)
    n, P, geom, sp, ap = synthetic.make_case(ijk, 0.4, 0, 0.05, 42000.0, [0], flag=4)    # 42,000 samples
    inst = compile_instance(n, P, geom, sp, ap, full_cycles=False, tol=1e-7, restart=20, save_h=False)
    size = inst.n_samples * n * 4
    assert size > KEEP_ENGINE + (2 << 30)
    torch.cuda.synchronize()
    before = free()
    eng = BatchedEngine(_lib.PREC_F32)
    for _ in range(2):
        slot = eng.add(inst)
        assert before - free() > size - KEEP_ENGINE - SLACK
        eng.remove(slot)
        assert before - free() < KEEP_ENGINE + SLACK
    eng.add(inst)
    eng.close()
    assert before - free() < KEEP_IDLE + SLACK

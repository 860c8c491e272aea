"""The neighbour table at the edges of its bit words and chunks of words."""
import numpy as np
import pytest

from pyheartsim_b200 import geometry_gpu
from pyheartsim_b200.geometry import lattice_neighbors

pytestmark = pytest.mark.gpu


# boxes (with the padding) of less than a word, of words that rows cross, of one
# chunk (65,536 cells), one more, and of several hundred chunks
@pytest.mark.parametrize("span,count", [((1, 1, 1), 1), ((2, 1, 1), 2), ((30, 1, 1), 30), ((31, 3, 2), 100),
                                        ((62, 30, 30), 9000), ((63, 31, 31), 255), ((64, 32, 32), 257),
                                        ((400, 300, 200), 40000)])
def test_random_subsets(span, count, cuda_device):
    rng = np.random.default_rng(sum(span) + count)
    cells = rng.choice(int(np.prod(span)), size=count, replace=False)
    ijk = np.stack(np.unravel_index(cells, span), axis=1) - np.array([7, 300, -20])
    nb, order = geometry_gpu.lattice_neighbors(ijk.astype(np.int32))
    np.testing.assert_array_equal(nb.cpu().numpy(), lattice_neighbors(ijk))
    np.testing.assert_array_equal(order.cpu().numpy(), np.lexsort((ijk[:, 0], ijk[:, 1], ijk[:, 2])))
    nb2, none = geometry_gpu.lattice_neighbors(ijk.astype(np.int32), order=False)
    assert none is None and bool((nb2 == nb).all())

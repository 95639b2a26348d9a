"""The order inside the cells where a warp takes several positions per lane and
several tiles, and the scatter several particles per thread and trip: about a
million particles, cells of 1 to 256 of them side by side with crowded ones, on a
grid that is scanned and scattered in one launch, on a larger one, and on one whose
strip is planned in pieces of 1024 columns.  State
bitwise equal to the oracle, alone and in a batch."""
import numpy as np
import pytest

from amsc_b200.batch import Batch
from amsc_b200.dampm import Solver
from oracle.oracle import Oracle
from test_gpu_sort_paths import FIELDS, _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ney,nex,spread", [(97, 101, 256), (150, 140, 90), (9, 1101, 256)])
def test_mixed_cells_in_wide_tiles(cuda_lib, ney, nex, spread):
    rng = np.random.default_rng(ney)
    sizes = rng.integers(1, spread + 1, ney * nex)
    sizes[rng.random(sizes.size) < 0.1] = 1
    edge = rng.permutation(sizes.size)[:200]
    sizes[edge] = np.resize([255, 256, 257, 600], edge.size)
    d = _data(ney, nex, 0.5, rng, [(c, int(m)) for c, m in enumerate(sizes)])
    assert 0.8e6 < d.np < 1.5e6
    o = Oracle(d, threads=8)
    o.run(2)
    with Solver(d, capacity=d.np) as s, Batch(d.np, 2 * d.nnodes, 1) as b:
        h = b.add(d)
        s.step(2)
        b.step(2)
        for k in FIELDS:
            np.testing.assert_array_equal(s.download(k), o.get(k), err_msg=k)
            np.testing.assert_array_equal(b.download(h, k), o.get(k), err_msg=k)

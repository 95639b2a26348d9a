"""An addition's arrays reach the device in pieces of 131072 values (13107
particles): scenarios around the edges of a piece, in both precisions."""
import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.batch import Batch
from amsc_b200.dampm import Solver
from amsc_b200.data import PARTICLE_KEYS

pytestmark = pytest.mark.gpu


def _cropped(cells, particles):
    d = scenarios.mudflow(N=cells)
    for k in PARTICLE_KEYS:
        d.arrays[k] = d.arrays[k][:particles].copy()
    d.arrays["mom_px"] = np.linspace(-1.0, 1.0, particles)  # read by the first step
    d.arrays["mom_py"] = np.linspace(2.0, -1.0, particles)
    return d


# 361^2 and 363^2 nodes: one piece of terrain and two
@pytest.mark.parametrize("cells, particles", [(360, 1), (362, 13107), (362, 13108),
                                              (362, 3 * 13107 + 5)])
def test_pieces(cuda_lib, cells, particles):
    d = _cropped(cells, particles)
    small = scenarios.dam_break_flat()
    with Batch(d.np + small.np, d.nnodes + small.nnodes, 2) as b, Solver(d) as s:
        b.add(small)  # the scenario does not start at the arrays' start
        h = b.add(d)
        for k in ("x", "y", "Mp", "Vp", "hp", "vpx", "mom_px", "mom_py"):
            np.testing.assert_array_equal(b.download(h, k), d.arrays[k], err_msg=k)
        b.step(2)
        s.step(2)
        for k in ("x", "y", "vpx", "vpy", "hp", "F_11", "F_12", "F_22"):
            np.testing.assert_array_equal(b.download(h, k), s.download(k), err_msg=k)
    with Batch(d.np, d.nnodes, 1, precision="fp32") as b:
        h = b.add(d)
        for k in ("x", "y", "Mp", "Vp", "hp", "mom_px", "mom_py"):
            np.testing.assert_array_equal(b.download(h, k),
                                          d.arrays[k].astype(np.float32).astype(np.float64),
                                          err_msg=k)

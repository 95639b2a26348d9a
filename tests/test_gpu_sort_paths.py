"""The paths of a pass's sort and planner: grids up to 16384 cells are scanned
and scattered in one launch, larger ones in tiles; warps cut the strips, several
each where there are more strips than warps, in pieces where a strip is long.
Cells on both sides of 256 particles, up to which a warp counts over the indices
of a particle's cell and above which a block orders the cell.  State bitwise equal
to the oracle, alone and in a batch."""
import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.batch import Batch
from amsc_b200.data import DATA
from amsc_b200.dampm import Solver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vpx", "vpy", "hp", "F_11", "F_12", "F_22")
SIZES = (1, 2, 15, 16, 17, 32, 33, 255, 256, 257, 600)


def _scenario(ney, nex, h=0.5):
    """Cells of SIZES particles over the whole grid, the corners among them."""
    rng = np.random.default_rng(ney * 7919 + nex)
    n = min(4 * len(SIZES), ney * nex)
    cells = np.unique(np.concatenate([[0, ney * nex - 1], rng.integers(0, ney * nex, n)]))
    return _data(ney, nex, h, rng, [(c, SIZES[k % len(SIZES)])
                                    for k, c in enumerate(rng.permutation(cells))])


def _data(ney, nex, h, rng, cells):
    """m particles in each cell c of (c, m), in random order."""
    x, y, ap = [], [], []
    for c, m in cells:
        x.append((c // ney + rng.uniform(0.02, 0.98, m)) * h)
        y.append((c % ney + rng.uniform(0.02, 0.98, m)) * h)
        ap.append(np.full(m, h * h / m))
    x, y, ap = (np.concatenate(v) for v in (x, y, ap))
    order = rng.permutation(x.size)
    x, y, ap = x[order], y[order], ap[order]
    hp, z = rng.uniform(0.9, 1.1, x.size), np.zeros(x.size)
    arrays = {"x": x, "y": y, "Mp": 1000.0 * ap * hp, "Ap": ap, "vpx": z, "vpy": z, "hp": hp,
              "mom_px": z, "mom_py": z, "Vp": ap * hp}
    for k in ("Z", "dZdx", "dZdy"):
        arrays[k] = np.zeros((ney + 1) * (nex + 1))
    return DATA(arrays, scenarios._base_scalars(
        Nex=nex, Ney=ney, hx=h, hy=h, rho=1000.0, tauy=500.0, BINGHAM_ON=1.0, FRICTION_ON=1.0,
        BC_FLAG=1, MERGE_SPLIT_ON=0, eq_level=0.0, DT_FIXED=1e-4, NSTEPS=100))


@pytest.mark.parametrize("ney,nex", [(1, 1), (1, 40), (61, 5), (64, 64), (128, 128), (127, 130),
                                     (16384, 1), (16400, 1), (2, 8300)])
def test_sort_and_units_on_every_path(cuda_lib, ney, nex):
    _check(_scenario(ney, nex))


@pytest.mark.parametrize("ney,nex", [(8, 600), (100, 300)])
def test_units_beyond_the_planner_s_buffer(cuda_lib, ney, nex):
    """Every column holds particles and is a unit of its own: a strip's units are
    appended to the list in several pieces, a crowded column among the heavy ones."""
    rng = np.random.default_rng(nex)
    cells = [(c, 1) for c in range(ney * nex)]
    cells[ney * (nex // 2)] = (ney * (nex // 2), 2500)
    _check(_data(ney, nex, 0.5, rng, cells))


def _check(d):
    steps = 6
    o = Oracle(d, threads=2)
    o.run(steps)
    with Solver(d) as s, Batch(d.np, 8 * d.nnodes, 1) as b:
        h = b.add(d)
        s.step(steps)
        b.step(steps)
        assert s.status()["it"] == steps
        for k in FIELDS:
            np.testing.assert_array_equal(s.download(k), o.get(k), err_msg=k)
            np.testing.assert_array_equal(b.download(h, k), o.get(k), err_msg=k)
        # (per unit, then over the units: round-off of the order)
        np.testing.assert_allclose(s.ledgers()[:6], o.ledger()[:6], rtol=1e-11, atol=1e-9)

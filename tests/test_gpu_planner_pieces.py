"""Strips planned in pieces of 512 columns: grids at the edges of a piece, flows
that lie inside one piece or across two, strips of many pieces and many strips of
one; with the pieces cut one by one and several at a time.  State bitwise equal to
the oracle, alone and in a batch, ledger to the round-off of its order."""
import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.batch import Batch
from amsc_b200.dampm import Solver
from test_gpu_sort_paths import FIELDS, _check, _data
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _columns(ney, nex, lo, hi, crowd=()):
    """One to four particles in some cells of columns [lo, hi), 700 in one of each
    column of `crowd`."""
    rng = np.random.default_rng(nex * 31 + lo)
    n = min(3000, ney * (hi - lo))
    cells = np.unique(rng.integers(ney * lo, ney * hi, n))
    cells = [(int(c), int(m)) for c, m in zip(cells, rng.integers(1, 5, cells.size))]
    return _data(ney, nex, 0.5, rng, cells + [(c * ney + ney // 2, 700) for c in crowd])


CASES = [(40, 511, 0, 511, (510,)), (40, 512, 0, 512, (511,)), (40, 513, 0, 513, (511, 512)),
         (40, 1025, 500, 530, (511,)), (31, 1025, 1000, 1025, (1023, 1024)),
         (31, 1600, 512, 1024, (512, 1023)), (29, 1600, 511, 512, ()), (2, 5000, 0, 5000, (2048,)),
         (9000, 3, 0, 3, (1,))]


@pytest.mark.parametrize("case", CASES)
def test_pieces(cuda_lib, case):
    _check(_columns(*case))


@pytest.mark.parametrize("col_weight", [4, 64, 100000])
def test_several_pieces_at_a_time(cuda_lib, col_weight):
    """The lighter a column, the more pieces one warp takes: 1, 2, 32 of them."""
    ds = [_columns(*CASES[k]) for k in (2, 5, 7)]
    with Batch(sum(d.np for d in ds), sum(d.nnodes for d in ds), 3) as b:
        hs = [b.add(d) for d in ds]
        b.tune(col_weight=col_weight)
        b.step(4)
        for h, d in zip(hs, ds):
            o = Oracle(d, threads=2)
            o.run(4)
            for k in FIELDS:
                np.testing.assert_array_equal(b.download(h, k), o.get(k), err_msg=k)
            np.testing.assert_allclose(b.ledgers(h)[:6], o.ledger()[:6], rtol=1e-11, atol=1e-9)


@pytest.mark.parametrize("case", [CASES[0], CASES[8]])  # 2 and 301 pieces
def test_ledger_of_every_step(cuda_lib, case):
    """A block of G2P sums the ledger, or a launch of its own where the pieces are
    many: the log holds every step's row, replayed from a graph or not."""
    d = _columns(*case)
    o = Oracle(d, threads=2)
    with Solver(d) as s:
        s.step(19)
        log = s.ledger_history(1, 19)
        for it in range(1, 20):
            o.run(1)
            led = o.ledger()
            assert log[it - 1][0] == pytest.approx(it * 1e-4 - 1e-4, abs=1e-12)
            np.testing.assert_allclose(log[it - 1][1:], led[6:8], rtol=0, atol=1e-12)
        np.testing.assert_allclose(s.ledgers()[:6], o.ledger()[:6], rtol=1e-11, atol=1e-9)
        assert tuple(s.ledgers()[[8, 6, 7]]) == tuple(log[18])
    # in a batch, beside one of the other kind (which a graph's passes take along)
    e = _columns(*CASES[3])
    with Batch(d.np + e.np, d.nnodes + e.nnodes, 2) as b:
        hd, he = b.add(d), b.add(e)
        b.step(19)
        np.testing.assert_allclose(b.ledgers(hd)[:6], o.ledger()[:6], rtol=1e-11, atol=1e-9)
        o = Oracle(e, threads=2)
        o.run(19)
        np.testing.assert_allclose(b.ledgers(he)[:6], o.ledger()[:6], rtol=1e-11, atol=1e-9)


def test_units_of_a_large_batch(cuda_lib):
    """More than 4096 particles per CTA: the units stay at that weight, the state is
    that of the scenario alone."""
    d = scenarios.mudflow(N=2048)
    with Solver(d, capacity=d.np) as s, Batch(d.np, d.nnodes, 1) as b:
        h = b.add(d)
        s.step(4)
        b.step(4)
        for k in FIELDS:
            np.testing.assert_array_equal(b.download(h, k), s.download(k), err_msg=k)
        np.testing.assert_allclose(b.ledgers(h)[:6], s.ledgers()[:6], rtol=1e-12, atol=1e-6)

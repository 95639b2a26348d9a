"""The step's begin and end live inside other kernels (the unit plan, the next
pass, the call's last launch): the loop state and the fields are the oracle's
however the passes are split into calls, and when the loop condition fails in
the middle of one."""
import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.batch import Batch
from amsc_b200.dampm import Solver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vpx", "vpy", "hp", "F_11", "F_12", "F_22")


def _fixed():
    return scenarios.dam_break_flat(nsteps=37)


def _adaptive():
    d = scenarios.well_balance(nE=20, DX=0.41)
    d.scalars["T"] = 0.02
    return d


@pytest.mark.parametrize("make", [_fixed, _adaptive])
@pytest.mark.parametrize("calls", [(1, 1, 1), (16,), (17, 3), (64,), (40, 1, 16), (5, 48)])
def test_loop_state_after_split_calls(cuda_lib, make, calls):
    d = make()
    o = Oracle(d)
    b_np, b_nn = d.np, d.nnodes
    with Solver(d) as s, Batch(b_np, b_nn, 1) as b:
        h = b.add(d)
        for n in calls:
            o.run(n)
            s.step(n)
            b.step(n)
            st, q = s.status(), b.query(h)
            assert (st["it"], st["t"], st["dt"]) == (o.it, o.t, o.dt)
            assert (q["it"], q["t"], q["dt"]) == (o.it, o.t, o.dt)
        for k in FIELDS:
            np.testing.assert_array_equal(s.download(k), o.get(k), err_msg=k)
            np.testing.assert_array_equal(b.download(h, k), o.get(k), err_msg=k)

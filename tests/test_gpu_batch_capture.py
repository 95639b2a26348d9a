"""A batch whose stream the caller captures: an addition is refused (it would
run at the graph's launches and not before the steps that count on it), and the
batch goes on as if it had not been asked for."""
import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.batch import Batch
from amsc_b200.dampm import DampmError, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_addition_during_capture_is_refused(cuda_lib, precision):
    import torch
    d = scenarios.dam_break_flat(nsteps=500)
    st = torch.cuda.Stream()
    with Batch(2 * d.np, 2 * d.nnodes, 4, stream=st.cuda_stream, precision=precision) as b:
        first = b.add(d)
        b.step(3)
        b.sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            g.capture_begin(capture_error_mode="thread_local")
            b.step(2)
            with pytest.raises(DampmError):
                b.add(d)
            g.capture_end()
        assert b.usage()["live"] == 1
        second = b.add(d)
        b.step(3)
        assert b.query(first)["it"] == 6 and b.query(second)["it"] == 3
        got = {h: b.download(h, "hp") for h in (first, second)}
        if precision == "fp64":
            for h, n in ((first, 6), (second, 3)):
                with Solver(d) as s:
                    s.step(n)
                    np.testing.assert_array_equal(got[h], s.download("hp"))

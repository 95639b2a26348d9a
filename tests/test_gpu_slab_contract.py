"""What the slab calls accept: reference indices that repeat (each slab's
particles numbered from 0, or all alike) or have the top bit set (they count as
unsigned), and a first half of a step that no second half follows."""
import ctypes as C

import numpy as np
import pytest

from amsc_b200 import scenarios
from amsc_b200.dampm import Solver, _ptr
from amsc_b200.slabs import local_run

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vpx", "vpy", "hp", "F_11", "F_12", "F_22")


def _set_index(e, idx):
    idx = np.ascontiguousarray(idx, dtype=np.int32)
    e.s._check(e.lib.dampm_slab_set_index(e.h, idx.ctypes.data_as(C.POINTER(C.c_int))))


def _marked(d):
    """Every particle with a mass of its own, which no step changes."""
    d = d.copy()
    m = d.arrays["Mp"]
    d.arrays["Mp"] = m * (1.0 + 1e-6 * np.arange(m.size) / m.size)
    assert np.unique(d.arrays["Mp"]).size == m.size
    return d


def _by_mass(run, k):
    v = np.concatenate([e.download(k)[0] for e in run.E.values()])
    m = np.concatenate([e.download("Mp")[0] for e in run.E.values()])
    return v[np.argsort(m)], np.sort(m)


@pytest.mark.parametrize("numbering", ["from_zero", "all_alike"])
def test_equal_indices_lose_no_particle(cuda_lib, numbering):
    steps = 40
    d = _marked(scenarios.mudflow(N=256))
    d.scalars["BINGHAM_ON"] = 0.0  # (a yield stress turns round-off into another plug)
    with Solver(d) as s:
        s.step(steps)
        ref = {k: s.download(k) for k in FIELDS[:5]}
        order = np.argsort(s.download("Mp"))
    run = local_run(d, 2)
    try:
        for e in run.E.values():
            n = e.status()["np"]
            _set_index(e, np.arange(n) if numbering == "from_zero" else np.zeros(n))
        run.step(steps)
        # every particle once, and where it was to move up to the order of the
        # sums: one of 1e-16 a step, which a flow amplifies by less than 10 in 50
        # steps (a perturbation in the 13th digit comes out as 5e-13)
        for k in ref:
            v, m = _by_mass(run, k)
            np.testing.assert_array_equal(m, np.sort(d.arrays["Mp"]))
            scale = np.abs(ref[k]).max()
            np.testing.assert_allclose(v, ref[k][order], rtol=0, atol=1e-9 * scale, err_msg=k)
    finally:
        run.close()


def test_equal_indices_follow_in_storage_order(cuda_lib):
    """The storage after an upload is DATA order: the first step of particles
    that are all numbered alike is the plain step."""
    d = scenarios.bench_slab(10000, nsteps=1)
    with Solver(d) as s:
        s.step(1)
        ref = {k: s.download(k) for k in FIELDS}
    plain, alike = local_run(d, 1), local_run(d, 1)
    try:
        _set_index(alike.E[0], np.zeros(d.np))
        plain.step(1)
        alike.step(1)
        place = plain.E[0].download("x")[1]  # which particle lies where, in both
        for k in FIELDS:
            np.testing.assert_array_equal(alike.E[0].download(k)[0], ref[k][place], err_msg=k)
    finally:
        plain.close()
        alike.close()


def test_indices_with_the_top_bit_set_come_last(cuda_lib):
    """Indices count as unsigned numbers, in plain cells as in crowded ones: the
    run is that of the particles listed in that order."""
    d = scenarios.bench_slab(10000, nsteps=30)
    rng = np.random.default_rng(3)
    x, y, h = d.arrays["x"].copy(), d.arrays["y"].copy(), float(d.scalars["hx"])
    pick = rng.permutation(x.size)[:600]  # a crowded cell too
    x[pick] = 40.3 * h + 0.2 * h * rng.random(600)
    y[pick] = 5.3 * h + 0.2 * h * rng.random(600)
    d.arrays["x"], d.arrays["y"] = x, y
    idx = (rng.permutation(d.np) - d.np // 2).astype(np.int32)
    order = np.argsort(idx.view(np.uint32))
    listed = d.copy()
    for k in ("x", "y", "Mp", "Ap", "vpx", "vpy", "hp", "mom_px", "mom_py", "Vp"):
        listed.arrays[k] = np.ascontiguousarray(d.arrays[k][order])
    with Solver(listed) as s:
        s.step(30)
        ref = {k: s.download(k) for k in FIELDS}
    run = local_run(d, 1)
    try:
        e = run.E[0]
        _set_index(e, idx)
        run.step(30)
        for k in FIELDS:
            v, ix = e.download(k)
            v = v[np.argsort(ix.astype(np.int32).view(np.uint32))]
            np.testing.assert_array_equal(v, ref[k], err_msg=k)
    finally:
        run.close()


@pytest.mark.parametrize("cells", [64, 256])  # one launch for scan and scatter, two
def test_upload_after_half_a_step(cuda_lib, cells):
    """A caller that gives a step up after its first half and uploads again gets
    the run of a fresh context: P2G's work list does not keep the units of the
    half that was given up."""
    d = scenarios.dam_break_flat(nsteps=100) if cells == 64 else scenarios.mudflow(N=cells)
    with Solver(d) as s:
        s.step(10)
        ref = {k: s.download(k) for k in FIELDS}
        led = s.ledgers()
    run = local_run(d, 1)
    try:
        e = run.E[0]
        arrs = [_ptr(d.arrays[k]) for k in ("x", "y", "Mp", "Ap", "vpx", "vpy", "hp", "mom_px",
                                            "mom_py", "Vp")]
        for _ in range(3):
            e.pass_(0)
            e.s._check(e.lib.dampm_upload_particles(e.h, d.np, *arrs))
        run.step(10)
        for k in FIELDS:
            np.testing.assert_array_equal(run.gather(k), ref[k], err_msg=k)
        np.testing.assert_allclose(run.ledgers()[:6], led[:6], rtol=1e-12, atol=1e-9)
    finally:
        run.close()

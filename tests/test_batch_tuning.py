"""Where Batch.autotune starts from, on the CPU against a stand-in library: the
setting in force, which it keeps unless a candidate is faster by the margin."""
import os
import re

import pytest

from amsc_b200 import batch as batch_mod


class _Library:
    """Every call succeeds; the settings of dampm_batch_tune are noted."""

    def __init__(self):
        self.settings = []

    def __getattr__(self, name):
        if name == "dampm_batch_tune":
            return lambda h, u, w, g: self.settings.append((u, w)) or 0
        return lambda *a: 0


@pytest.fixture
def batch(monkeypatch):
    monkeypatch.setattr(batch_mod, "load_library", _Library)
    # a clock by which every measurement takes the same time: nothing is faster
    now = iter(range(1 << 20))
    monkeypatch.setattr(batch_mod.time, "perf_counter", lambda: float(next(now)))
    b = batch_mod.Batch(1000, 1000, 4)
    b.h = 1
    yield b
    b.h = None


def _library_default():
    src = open(os.path.join(os.path.dirname(batch_mod.__file__), "csrc", "dampm_kernels.h")).read()
    units = int(re.search(r"kBatchUnitsPerCta = (\d+)", src).group(1))
    weight = int(re.search(r"#define DAMPM_COL_WEIGHT (\d+)", src).group(1))
    return units, weight


def test_autotune_starts_from_the_library_s_setting(batch):
    info = batch.autotune()
    assert info["trials"][0][:2] == _library_default()
    assert (info["units_per_cta"], info["col_weight"]) == _library_default()
    assert batch.lib.settings[-1] == _library_default()


def test_autotune_starts_from_the_setting_last_given(batch):
    batch.tune(units_per_cta=4)
    batch.tune(col_weight=64, graphs=False)
    batch.tune(graphs=True)
    info = batch.autotune(units=(1, 2), weights=(192,))
    assert info["trials"][0][:2] == (4, 64)
    assert (info["units_per_cta"], info["col_weight"]) == (4, 64)

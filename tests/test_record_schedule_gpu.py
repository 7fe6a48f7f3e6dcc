"""Rows of interval records across launches of every depth (the per-launch
schedule holds 32 steps a word): the rows taken and their values equal the
FP64 oracle's, with few records and with more than a tile lists."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("fp32", 1e-5)])
@pytest.mark.parametrize("depth", [1, 31, 33, 64, 200])
def test_interval_records(native, depth, prec, tol, many):
    from mbsolve_gb300 import lib as mb, setups
    mb.material.clear_library()
    n, steps = 900, 450
    dev, sce = setups.sit_2lvl(n, steps, phase=0.5)
    sce.set_ic_electric(mb.ic_field_random(amplitude=1e8, seed=5))
    dt = sce.get_endtime() / (steps - 1)
    length = dev.get_length()
    for interval in (1.0, 2.7, 31.9, 40.0, 129.3):
        sce.add_record(mb.record("e", interval * dt))
        if many:
            sce.add_record(mb.record("h", interval * dt, 0.4 * length))
    if prec == "fp32":
        # smooth fields: FP32 differences of white noise say nothing
        x = np.linspace(0.0, 1.0, n)
        sce.set_ic_electric(mb.ic_field_random(seed=5))
        sce.get_ic_electric()._cache[n] = 1e8 * np.exp(-((x - 0.5) / 0.1) ** 2)
    _, want = helpers.oracle_results("cvr-rodr", 2, dev, sce)
    _, got = helpers.gpu_results("gpu-fdtd-2lvl-cvr-rodr-" + prec, dev, sce,
                                 helpers.tuning(4, 256, depth))
    for a, b in zip(got, want):
        assert a.shape == b.shape
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)

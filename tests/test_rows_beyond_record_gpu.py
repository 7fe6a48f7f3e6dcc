"""Steps due beyond a record's last row (floor(dt / interval * step) against
floor(endtime / interval) + 1 rows, each as rounded) are no part of the results:
a NaN at such a step alone is not reported, one at a recorded step is."""
import ctypes as C
import math

import numpy as np
import pytest

from tests.test_failure_gpu import _add_nan_source

pytestmark = pytest.mark.gpu


def _grid(native, dev, sce):
    from mbsolve_gb300 import _native, capi_types as T, lib as mb
    g = T.mbg_grid()
    b = mb.to_pod(dev, sce)
    _native.check(native.mbg_scenario_grid(C.byref(b.device), C.byref(b.scenario), C.byref(g)))
    return g.timestep_size, g.num_timesteps


def _interval(dt, steps, endtime):
    """An interval with one step more due, the last, than rows."""
    for k in range(2, 40):
        interval = endtime / k
        for _ in range(8):
            rows = math.floor(endtime / interval) + 1
            if interval > dt and math.floor((dt / interval) * (steps - 1)) == rows:
                return interval
            interval = math.nextafter(interval, math.inf)
    return None


def _cases(kind):
    from mbsolve_gb300 import lib as mb, setups
    for steps in range(200, 260):
        mb.material.clear_library()
        if kind == "point":
            from tests.test_point_runs_gpu import _case
            dev, sce = _case(3, steps)
            out = mb.scenario("p", 1, sce.get_endtime(), sce.get_ic_density(), mb.ic_field_const(0.0),
                              mb.ic_field_const(0.0), steps)
            yield dev, out
        else:
            yield setups.sit_2lvl(256, steps)


@pytest.mark.parametrize("kind,name", [("grid", "2lvl-cvr-rodr-fp32"), ("grid", "2lvl-cvr-rodr-fp64"),
                                       ("point", "3lvl-reg-cayley-fp64")])
def test_only_recorded_rows_are_checked(native, kind, name):
    from mbsolve_gb300 import lib as mb, solvergpu
    for dev, sce in _cases(kind):
        dt, steps = _grid(native, dev, sce)
        interval = _interval(dt, steps, sce.get_endtime())
        if interval is not None:
            break
    assert interval is not None
    sce.add_record(mb.record("e", interval, 0.0))
    _add_nan_source(native, dev, sce, steps - 1)
    s = solvergpu.solver_gpu_fdtd(dev, sce, "gpu-fdtd-" + name)
    s.run()
    e = s.get_results()[-1].as_array()
    assert e.shape[0] == math.floor(sce.get_endtime() / interval) + 1 and np.isfinite(e).all()
    # and the check itself works
    sce.add_record(mb.record("e", 0.0, 0.0))
    s = solvergpu.solver_gpu_fdtd(dev, sce, "gpu-fdtd-" + name)
    with pytest.raises(RuntimeError, match="non-finite value"):
        s.run()

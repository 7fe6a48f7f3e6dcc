"""A tensor-core completion wait that runs out (made to give up without
polling, in the launch per level and in the persistent kernel) ends the run
with an error the host reads; no further product is issued, the outstanding
one is waited for before its tensor memory is given back, and the GPU goes
on: the same case then runs and equals the run before."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _solver(algo, levels, persistent):
    from mbsolve_gb300 import lib as mb, setups, solvergpu
    mb.material.clear_library()
    dev, sce = setups.random_nlvl(levels, 2000, 120, seed=2)
    return solvergpu.solver_gpu_fdtd(dev, sce, "gpu-fdtd-%dlvl-%s-fp32" % (levels, algo),
                                     helpers.tuning(1, 128, 8, persistent=persistent))


@pytest.mark.parametrize("persistent", [1, 2])
@pytest.mark.parametrize("levels", [4, 6])
@pytest.mark.parametrize("algo", ["cvr-rodr", "reg-cayley"])
def test_wait_runs_out_and_gpu_goes_on(native, monkeypatch, algo, levels, persistent):
    s = _solver(algo, levels, persistent)
    s.run()
    want = s.get_results()[0].as_array()
    monkeypatch.setenv("MBG_TEST_STALL_TC", "1")
    s = _solver(algo, levels, persistent)
    with pytest.raises(RuntimeError, match="tensor-core or bulk-copy completion wait ran out"):
        s.run()
    monkeypatch.delenv("MBG_TEST_STALL_TC")
    s = _solver(algo, levels, persistent)
    s.run()
    assert np.isfinite(want).all()
    assert np.array_equal(s.get_results()[0].as_array(), want)

"""A persistent kernel asked for without a launch shape runs, wherever a shape
of the solver has one: the autotuner picks among those shapes."""
import pytest

from tests import helpers
from tests.test_diagonal_media_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("by", ["tuning", "environment"])
@pytest.mark.parametrize("diagonal", [False, True])
@pytest.mark.parametrize("levels", [4, 5, 6])
@pytest.mark.parametrize("algo", ["cvr-rodr", "reg-cayley"])
def test_persistent_is_honoured(native, monkeypatch, algo, levels, diagonal, by):
    from mbsolve_gb300 import ensemble
    if by == "environment":
        monkeypatch.setenv("MBG_PERSISTENT", "1")
    e = ensemble.ensemble("gpu-fdtd-%dlvl-%s-fp32" % (levels, algo), [_case(levels, diagonal)],
                          helpers.tuning(persistent=1) if by == "tuning" else None)
    assert e.info()["persistent"] == 1
    e.run()
    assert e.status() == 0
    e.close()

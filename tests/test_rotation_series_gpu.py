"""FP64 field rotation over the ranges of its series (angles per step below
2^-9, below 1/4 and beyond) against the FP64 oracle, for the sparse and the
dense 2-level block and for 3 and 6 levels."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


# the angle of a step is about 2.9e-12 m/V times the field (2 levels)
@pytest.mark.parametrize("field", [1e8, 1e10, 7e10, 3e11])
@pytest.mark.parametrize("levels,setup", [(2, "sit"), (2, "random"), (3, "random"), (6, "random")])
def test_fp64_rotation_against_oracle(native, field, levels, setup):
    from mbsolve_gb300 import lib as mb, setups
    mb.material.clear_library()
    if setup == "sit":
        dev, sce = setups.sit_2lvl(150, 60)
        sce.set_ic_electric(mb.ic_field_const(field))
        sce.set_ic_density(mb.ic_density_const(mb.qm_operator([0.7, 0.3])))
    else:
        dev, sce = setups.random_nlvl(levels, 150, 60, seed=3, e_seed=field,
                                      length=setups.LENGTH_2LVL * 149 / 16383)
    sce.add_record(mb.record("d11", mb.record.density, 1, 1, 0.0, -1.0))
    _, want = helpers.oracle_results("cvr-rodr", levels, dev, sce)
    mb_name = "gpu-fdtd-%dlvl-cvr-rodr-fp64" % levels
    _, got = helpers.gpu_results(mb_name, dev, sce)
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)

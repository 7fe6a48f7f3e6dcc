"""Results of records of every size class of the copy (below and beyond one
pinned chunk, a chunk exactly, ragged ends), FP32 and FP64, real and complex:
the values of the whole equal those recorded point by point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("points", [4096, 32768, 32769, 131072, 300001])
def test_copied_records_equal_their_probes(native, points, prec):
    from mbsolve_gb300 import ensemble, lib as mb, setups
    mb.material.clear_library()
    dev, sce = setups.sit_2lvl(points, 5, phase=0.5)
    rng = np.random.default_rng(points)
    sce.set_ic_electric(mb.ic_field_random(amplitude=1e8, seed=1))
    sce.set_ic_density(mb.ic_density_const(mb.qm_operator([0.6, 0.4], [0.1 + 0.2j])))
    sce.add_record(mb.record("e", 0.0))
    sce.add_record(mb.coherence_record("c12", 1, 2, 0.0))
    at = sorted({0, points - 1, *rng.integers(0, points, 3).tolist()})
    dx = dev.get_length() / (points - 1)
    for i in at:
        sce.add_record(mb.record("e", 0.0, i * dx))
        sce.add_record(mb.coherence_record("c12", 1, 2, 0.0, i * dx))
    e = ensemble.ensemble("gpu-fdtd-2lvl-cvr-rodr-" + prec, [(dev, sce)])
    e.run()
    res = e.results(0)
    e.close()
    field = res[1].as_array()
    coh = res[2].get_data_complex().reshape(5, points)
    assert field.shape == (5, points) and np.all(np.isfinite(field))
    assert not res[1].get_data_imag().any()
    for k, i in enumerate(at):
        np.testing.assert_array_equal(field[:, i], res[3 + 2 * k].get_data_real())
        np.testing.assert_array_equal(coh[:, i], res[4 + 2 * k].get_data_complex())
    assert np.abs(coh.imag).max() > 0

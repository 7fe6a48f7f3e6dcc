"""The precompute by one CTA per material and by one thread per material
(what ensembles of more than 2,048 materials take) give the same constants:
the same runs give the same results from both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["cvr-rodr", "reg-cayley"])
@pytest.mark.parametrize("levels", [3, 5])
def test_cta_and_thread_form_agree(native, algo, levels):
    from mbsolve_gb300 import ensemble, lib as mb, setups
    got = []
    for count in (3, 2049):
        mb.material.clear_library()
        runs = []
        for i in range(count):
            dev, sce = setups.random_nlvl(levels, 16, 40, seed=i % 3,
                                          e_seed=1e6)
            sce.add_record(mb.record("d11", mb.record.density, 1, 1, 0.0, 0.0))
            runs.append((dev, sce))
        e = ensemble.ensemble("gpu-fdtd-%dlvl-%s-fp64" % (levels, algo), runs,
                              ensemble.tuning(1, 128, 4))
        e.run()
        got.append([r.as_array() for i in range(3) for r in e.results(i)])
        e.close()
    for a, b in zip(*got):
        # one order of operations, contracted to fma by two compilations
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)

"""Ensembles on both sides of the line between the precompute by one CTA and
by one thread per material give the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo,levels,line", [("cvr-rodr", 3, 1024), ("cvr-rodr", 4, 2048), ("cvr-rodr", 5, 4096),
                                              ("reg-cayley", 3, 2048), ("reg-cayley", 4, 2048),
                                              ("reg-cayley", 5, 4096)])
def test_both_sides_of_the_line_agree(native, algo, levels, line):
    from mbsolve_gb300 import ensemble, lib as mb, setups
    got = []
    for count in (line, line + 1):
        mb.material.clear_library()
        three = [setups.random_nlvl(levels, 16, 40, seed=i, e_seed=1e6) for i in range(3)]
        for _, sce in three:
            sce.add_record(mb.record("d11", mb.record.density, 1, 1, 0.0, 0.0))
        e = ensemble.ensemble("gpu-fdtd-%dlvl-%s-fp64" % (levels, algo), [three[i % 3] for i in range(count)],
                              ensemble.tuning(1, 128, 4))
        e.run()
        got.append([r.as_array() for i in range(3) for r in e.results(i)])
        e.close()
    for a, b in zip(*got):
        # one order of operations, contracted to fma by two compilations
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)

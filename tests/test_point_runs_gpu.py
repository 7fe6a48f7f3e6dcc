"""FP64 Cayley runs of a single grid point (one warp per point) against the
FP64 oracle: 2 to 5 levels on random media with complex couplings, sources of
both kinds, field, population, inversion, coherence and interval records,
more records than a tile lists, step counts at and beside a launch's 256;
several points in one ensemble; a second run() continuing the first; and the
tile kernel's results with the launch shape given."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _case(levels, steps, seed=1, many=False):
    from mbsolve_gb300 import lib as mb, setups
    rng = np.random.default_rng(seed)
    dev, sce = setups.random_nlvl(levels, 16, 40, seed=seed)
    region = dev.get_regions()[0]
    point = mb.device("point")
    point.add_region(mb.region("point", region.get_material(), 0, 0))
    pops = rng.dirichlet(np.ones(levels))
    out = mb.scenario("point", 1, 2e-17 * (steps - 1),
                      mb.ic_density_const(mb.qm_operator(list(pops))),
                      mb.ic_field_const(1e8), mb.ic_field_const(0.0), steps)
    out.add_source(mb.sech_pulse("hard", 0.0, mb.source.hard_source, 5e8,
                                 2e14, 1.0, 1e15))
    out.add_source(mb.sech_pulse("soft", 0.0, mb.source.soft_source, 2e8,
                                 3e14, 0.5, 1e15))
    for k in range(1, levels + 1):
        out.add_record(mb.record("d%d%d" % (k, k), mb.record.density, k, k, 0.0, 0.0))
    out.add_record(mb.record("e", 0.0, 0.0))
    out.add_record(mb.record("inv12", 5.3e-17))
    if many:
        for k in range(9):
            out.add_record(mb.record("p", 2e-17 * (k + 0.5), 0.0))
    return point, out


@pytest.mark.parametrize("steps", [2, 255, 256, 257, 700])
@pytest.mark.parametrize("levels", [2, 3, 4, 5])
def test_against_oracle(native, levels, steps):
    from mbsolve_gb300 import lib as mb
    mb.material.clear_library()
    dev, sce = _case(levels, steps, many=steps == 257)
    _, want = helpers.oracle_results("reg-cayley", levels, dev, sce)
    _, got = helpers.gpu_results("gpu-fdtd-%dlvl-reg-cayley-fp64" % levels, dev, sce)
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert a.shape == b.shape
        assert np.linalg.norm(a - b) <= 1e-9 * max(np.linalg.norm(b), 1e-300)


def test_ensemble_rerun_coherence_and_tile_kernel(native):
    from mbsolve_gb300 import ensemble, lib as mb, solvergpu
    name = "gpu-fdtd-3lvl-reg-cayley-fp64"
    mb.material.clear_library()
    runs = [_case(3, 300 + 40 * k, seed=k) for k in range(5)]
    for _, sce in runs:
        sce.add_record(mb.coherence_record("c13", 1, 3, 0.0, 0.0))
        sce.add_record(mb.coherence_record("c31", 3, 1, 0.0, 0.0))
    a = ensemble.ensemble(name, runs)
    b = ensemble.ensemble(name, runs, ensemble.tuning(1, 128, 8))
    assert (a.info()["threads"], b.info()["threads"]) == (32, 128)
    a.run()
    b.run()
    for r in range(5):
        for x, y in zip(a.results(r), b.results(r)):
            x, y = x.get_data_complex(), y.get_data_complex()
            assert np.linalg.norm(x) > 0
            assert np.linalg.norm(x - y) <= 1e-10 * np.linalg.norm(y)
    # a checkpoint of one form continues in the other
    c = ensemble.ensemble(name, runs)
    d = ensemble.ensemble(name, runs, ensemble.tuning(1, 128, 8))
    c.advance(123)
    d.load_state(c.save_state())
    c.run()
    d.run()
    for r in range(5):
        for x, y in zip(c.results(r), d.results(r)):
            x, y = x.get_data_complex(), y.get_data_complex()
            assert np.linalg.norm(x - y) <= 1e-10 * np.linalg.norm(y)
    for e in (a, b, c, d):
        e.close()
    # run() twice continues from the state of the first
    dev, sce = runs[0]
    s = solvergpu.solver_gpu_fdtd(dev, sce, name)
    t = solvergpu.solver_gpu_fdtd(dev, sce, name, helpers.tuning(1, 128, 8))
    for q in (s, t):
        q.run()
        q.run()
    for x, y in zip(s.get_results(), t.get_results()):
        x, y = x.get_data_complex(), y.get_data_complex()
        assert np.linalg.norm(x - y) <= 1e-10 * np.linalg.norm(y)

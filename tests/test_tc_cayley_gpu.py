"""FP32 Cayley steps with the field-free product on the tensor cores, 4 to 6
levels: against the FP64 oracle and the CUDA-core kernel, on uniform tiles,
tiles that mix two media and vacuum, a device end inside a tile and a mirror
wall, launch per level and persistent."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _case(levels, points, mirror):
    from mbsolve_gb300 import lib as mb, setups
    mb.material.clear_library()
    dx = 2.0 ** -27   # positions exact: the last point is the device's end
    cut = [int(0.45 * points) * dx, int(0.5 * points) * dx, (points - 1) * dx]
    a, _ = setups.random_nlvl(levels, 16, 40, seed=3)
    b, _ = setups.random_nlvl(levels, 16, 40, seed=4)
    mats = [d.get_regions()[0].get_material() for d in (a, b)]
    vac = setups._material("vacuum")
    dev = mb.device("two media", mb.bc_field_mirror(0.5, 0.3) if mirror else None)
    dev.add_region(mb.region("a", mats[0], 0.0, cut[0]))
    dev.add_region(mb.region("v", vac, cut[0], cut[1]))
    dev.add_region(mb.region("b", mats[1], cut[1], cut[2]))
    rng = np.random.default_rng(levels)
    sce = mb.scenario("s", points, setups._courant_endtime(points, dev.get_length(), 300),
                      mb.ic_density_const(mb.qm_operator(list(rng.dirichlet(np.ones(levels))))),
                      mb.ic_field_random(), mb.ic_field_const(0.0))
    x = np.linspace(0.0, 1.0, points)
    sce.get_ic_electric()._cache[points] = 1e8 * np.exp(-((x - 0.5) / 0.1) ** 2)
    for name in ("e", "h", "p"):
        sce.add_record(mb.record(name, 1e-16))
    for k in range(1, levels + 1):
        sce.add_record(mb.record("d", mb.record.density, k, k, 1e-16, -1.0))
    return dev, sce


@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("points", [97, 128, 700])
@pytest.mark.parametrize("levels", [4, 5, 6])
def test_against_oracle_and_cuda_cores(native, levels, points, mirror):
    dev, sce = _case(levels, points, mirror)
    _, want = helpers.oracle_results("reg-cayley", levels, dev, sce)
    name = "gpu-fdtd-%dlvl-reg-cayley-fp32" % levels
    for tun in (helpers.tuning(1, 128, 8, persistent=2), helpers.tuning(1, 128, 8, persistent=1),
                helpers.tuning(1, 128, 16, persistent=2),
                helpers.tuning(1, 192 if levels == 4 else 256, 8, persistent=2)):
        dev, sce = _case(levels, points, mirror)
        _, got = helpers.gpu_results(name, dev, sce, tun)
        for a, b in zip(got, want):
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)

"""The FP32 Cayley steps with the field-free product on the tensor cores on a
coarse grid, where a step's increments are large: the error against the FP64
oracle after many steps is that of rounding errors that average out.

Bound: a step turns the coherences by up to phi = 0.038 (50 meV, 500 points
on 150 um); its increment carries about two roundings of 2^-24 of itself, in
2,000 steps sqrt(2000) x 2 x 2^-24 x phi = 2e-7 of the density matrix, and as
much again through the field. A truncating accumulation, whose error grows
with the number of steps itself, exceeds it."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _case(levels, seed):
    from mbsolve_gb300 import lib as mb, setups
    mb.material.clear_library()
    dev, sce = setups.random_nlvl(levels, 500, 2000, seed=seed)
    rng = np.random.default_rng(seed)
    sce.set_ic_density(mb.ic_density_const(mb.qm_operator(list(rng.dirichlet(np.ones(levels))))))
    sce.set_ic_electric(mb.ic_field_random())
    x = np.linspace(0.0, 1.0, 500)
    sce.get_ic_electric()._cache[500] = 1e7 * np.exp(-((x - 0.4) / 0.07) ** 2)
    for k in range(1, levels + 1):
        sce.add_record(mb.record("d", mb.record.density, k, k, 0.9 * sce.get_endtime(), -1.0))
    return dev, sce


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("levels", [4, 5, 6])
def test_error_on_a_coarse_grid(native, levels, seed):
    dev, sce = _case(levels, seed)
    _, want = helpers.oracle_results("reg-cayley", levels, dev, sce)
    errs = []
    for nt in (128, 192 if levels == 4 else 256):
        dev, sce = _case(levels, seed)
        _, got = helpers.gpu_results("gpu-fdtd-%dlvl-reg-cayley-fp32" % levels, dev, sce,
                                     helpers.tuning(1, nt, 8))
        errs.append(max(np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in zip(got[1:], want[1:])))
    print("levels %d seed %d: tensor cores %.2e, CUDA cores %.2e" % (levels, seed, *errs))
    assert max(errs) <= 4e-7

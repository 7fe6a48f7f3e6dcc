"""FP32 Cayley runs of 4 to 6 levels at 1 x 128: media with diagonal
Hamiltonians take the CUDA-core kernel (bit for bit the state of the wider
CUDA-core shape, low words included), persistent, by default and beside
vacuum; with one dense medium in the ensemble all take the tensor-core kernel,
whose state differs in its rounding."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu

WIDE = {4: 192, 5: 256, 6: 256}


def _case(levels, diagonal=True, seed=1):
    from mbsolve_gb300 import lib as mb, setups
    dev, sce = setups.random_nlvl(levels, 1500, 200, seed=seed, e_seed=1e7)
    qm = dev.get_regions()[0].get_material().get_qm()
    if diagonal:
        qm = mb.qm_description(1e24, mb.qm_operator(list(qm.get_hamiltonian().get_main_diagonal())),
                               qm.get_dipole_operator(), qm.get_relaxation_superop())
    length = dev.get_length()
    out = mb.device("device")
    out.add_region(mb.region("vacuum", setups._material("vacuum"), 0.0, 0.2 * length))
    out.add_region(mb.region("active", setups._material("active%d%d" % (diagonal, seed), qm), 0.2 * length, length))
    sce.add_record(mb.record("d", mb.record.density, 1, 1, 0.0, 0.7 * length))
    return out, sce


def _traces(levels, runs, *tuning, persistent=0):
    from mbsolve_gb300 import ensemble, lib as mb
    mb.material.clear_library()
    t = helpers.tuning(*tuning, persistent=persistent) if tuning else None
    e = ensemble.ensemble("gpu-fdtd-%dlvl-reg-cayley-fp32" % levels, runs(), t)
    e.run()
    out = [r.as_array() for r in e.results(0)] + [np.frombuffer(bytes(e.save_state()), np.uint8)]
    info = e.info()
    e.close()
    return out, info


@pytest.mark.parametrize("levels", [4, 5, 6])
def test_diagonal_media_take_the_cuda_cores(native, monkeypatch, levels):
    def one():
        return [_case(levels)]
    want, _ = _traces(levels, one, 1, WIDE[levels], 8)
    for persistent in (1, 2):
        got, info = _traces(levels, one, 1, 128, 8, persistent=persistent)
        assert info["persistent"] == (persistent == 1)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
    monkeypatch.setenv("MBG_AUTOTUNE", "0")
    got, info = _traces(levels, one)
    assert info["threads"] == 128
    wide, _ = _traces(levels, one, 1, WIDE[levels], info["depth"])
    for a, b in zip(got, wide):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("levels", [4, 6])
def test_a_dense_medium_beside_a_diagonal_one(native, levels):
    def two():
        return [_case(levels), _case(levels, False, 2)]
    got, _ = _traces(levels, two, 1, 128, 8)
    want, _ = _traces(levels, two, 1, WIDE[levels], 8)
    assert not np.array_equal(got[-1], want[-1])
    # rounding only: 200 steps of 2^-24 of increments below 1
    for a, b in zip(got[:-1], want[:-1]):
        assert np.linalg.norm(a - b) <= 200 * 2.0 ** -24 * np.linalg.norm(b)

"""The grid of the tensor-core Cayley product's leading words is that of the
field-free matrix's largest entry, which the precompute stores. CPU only."""
import numpy as np
import pytest

from mbsolve_gb300 import lib as mb, setups
from tests.test_precompute import _constants


@pytest.mark.parametrize("levels", [2, 4, 6])
def test_largest_entry_of_the_field_free_matrix(native, levels):
    from mbsolve_gb300 import _native
    dev, sce = setups.random_nlvl(N=levels, num_gridpoints=16, num_timesteps=10, seed=levels)
    L = _native.material_layout("reg-cayley", levels)
    c = _constants(native, "reg-cayley", mb.to_pod(dev, sce).device.materials[0], 2.5e-17)
    n2 = levels * levels
    B0 = c[L["B0"]:L["B0"] + n2 * L["NP"]].reshape(n2, L["NP"])[:, :n2]
    assert c[L["maxB0"]] == np.abs(B0).max() > 0

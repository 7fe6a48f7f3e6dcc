"""The allocation-free precompute allocates nothing on its launch either: the
device's free memory stays as it was but for the module's own code and arrays
(a stack frame beyond the context's limit would make the driver allocate it
for every thread the GPU can hold, hundreds of megabytes)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROG = """
import ctypes as C, sys
sys.path.insert(0, %r)
import torch
from mbsolve_gb300 import _native, lib as mb, setups
L = _native.load()
algo, levels = sys.argv[1].encode(), int(sys.argv[2])
dev, _ = setups.random_nlvl(levels, 16, 40)
b = mb.to_pod(dev, _)
mat = b.device.materials[0]
n = C.c_size_t()
_native.check(L.mbg_material_constants_noalloc(algo, C.byref(mat), 2.5e-17, None, 0, C.byref(n), None))
buf = torch.zeros(n.value, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
_native.check(L.mbg_material_constants_noalloc(algo, C.byref(mat), 2.5e-17, buf.data_ptr(), n.value, C.byref(n), None))
torch.cuda.synchronize()
print(before - torch.cuda.mem_get_info()[0])
""" % ROOT


@pytest.mark.parametrize("algo,levels", [("cvr-rodr", 2), ("cvr-rodr", 6), ("reg-cayley", 3), ("reg-cayley", 6)])
def test_launch_allocates_nothing(native, algo, levels):
    out = subprocess.run([sys.executable, "-c", PROG, algo, str(levels)], check=True, capture_output=True,
                         text=True, cwd=ROOT).stdout
    assert int(out.split()[-1]) <= 64 << 20

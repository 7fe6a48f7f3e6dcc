"""The autotuner's entries are told apart by what decides the pick: dense and
diagonal media, small and large grids, a persistent kernel asked for, and the
set of kernels (an entry in the form of an earlier set is not read)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROG = """
import sys
sys.path.insert(0, %r)
from mbsolve_gb300 import ensemble, lib as mb, setups
from tests import helpers
def medium(diagonal):
    dev, sce = setups.random_nlvl(6, 8000, 300)
    if diagonal:
        qm = dev.get_regions()[0].get_material().get_qm()
        m = setups._material("diagonal", mb.qm_description(
            1e24, mb.qm_operator(list(qm.get_hamiltonian().get_main_diagonal())),
            qm.get_dipole_operator(), qm.get_relaxation_superop()))
        length = dev.get_length()
        dev = mb.device("diagonal")
        dev.add_region(mb.region("active", m, 0.0, length))
    return dev, sce
def tune(name, run, tuning=None):
    e = ensemble.ensemble("gpu-fdtd-" + name, [run], tuning)
    print(e.info())
    e.close()
for kind in sys.argv[1:]:
    if kind in ("dense", "diagonal"):
        tune("6lvl-reg-cayley-fp32", medium(kind == "diagonal"))
    elif kind == "forced":
        tune("6lvl-reg-cayley-fp32", medium(False), helpers.tuning(persistent=1))
    else:
        tune("2lvl-cvr-rodr-fp32", setups.sit_2lvl(int(kind), 300))
""" % ROOT


def _entries(tmp_path, *kinds, before=()):
    path = tmp_path / "tune.txt"
    path.write_text("".join(line + "\n" for line in before))
    subprocess.run([sys.executable, "-c", PROG] + list(kinds), check=True, cwd=ROOT,
                   env=dict(os.environ, MBG_TUNE_CACHE=str(path)))
    return [line for line in path.read_text().split("\n") if line.strip()]


@pytest.mark.parametrize("kinds", [("dense", "diagonal"), ("100", "60000"), ("dense", "forced")])
def test_own_entries(native, tmp_path, kinds):
    lines = _entries(tmp_path, *kinds, *kinds)
    assert len(lines) == 2
    assert len({line.split()[0] for line in lines}) == 2


def test_entries_of_another_kernel_set(native, tmp_path):
    key = _entries(tmp_path, "dense")[0].split()[0]
    gpu = key.split(":")[0]
    # the form without media, size class and kernel set
    old = "%s:2:6:s0:32:0:1:256 1 256 1 8" % gpu
    lines = _entries(tmp_path, "dense", before=[old])
    assert len(lines) == 2 and lines[0] == old and lines[1].split()[0] == key

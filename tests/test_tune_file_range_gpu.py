"""Lines of an MBG_TUNE_CACHE file out of the engine's range (a depth beyond the
kernels' 256 step schedule entries, no launches per graph) are left out: the
run is tuned anew and appends its own."""
import pytest

from tests.test_tune_key_gpu import _entries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["8 256 512 8", "8 256 257 8", "2 128 16 0", "2 128 16 -2", "2 128 0 8"])
def test_lines_out_of_range(native, tmp_path, bad):
    key = _entries(tmp_path, "20000")[0].split()[0]
    lines = _entries(tmp_path, "20000", before=["%s %s" % (key, bad)])
    assert len(lines) == 2 and lines[1].split()[0] == key
    assert 1 <= int(lines[1].split()[3]) <= 256

"""Several threads reading the large FP32 records of one ensemble at a time get
the records, each its own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_read_their_own_records(native):
    from mbsolve_gb300 import ensemble, lib as mb, setups
    mb.material.clear_library()
    runs = []
    for k in range(4):
        dev, sce = setups.sit_2lvl(300000 + 1000 * k, 4, phase=0.5)
        sce.set_ic_electric(mb.ic_field_random(amplitude=1e8, seed=k))
        sce.add_record(mb.record("e", 0.0))
        runs.append((dev, sce))
    e = ensemble.ensemble("gpu-fdtd-2lvl-cvr-rodr-fp32", runs)
    e.run()
    want = [e.results(r)[1].as_array() for r in range(4)]
    wrong = []

    def read(r):
        for _ in range(8):
            if not np.array_equal(e.results(r)[1].as_array(), want[r]):
                wrong.append(r)

    threads = [threading.Thread(target=read, args=(r,)) for r in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    e.close()
    assert not wrong

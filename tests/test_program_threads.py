"""One recorded sequence of surrogate launches run by several threads, each with
its own input: every native call sees the input of its thread. CPU only (the
native call is replaced)."""
import threading
import time

import pytest

torch = pytest.importorskip("torch")


def test_every_run_sees_its_own_input(monkeypatch):
    from mbsolve_gb300 import surrogate_kernels as K
    seen = []

    class native:
        @staticmethod
        def mbg_fno_run(ops, count, stream):
            time.sleep(0.002)   # as the native call does, let other threads run
            seen.append((threading.get_ident(), count, ops[0].in_[0]))
            return 0

    monkeypatch.setattr(K, "_lib", lambda: native)
    monkeypatch.setattr(K, "_stream", lambda: None)
    monkeypatch.setattr(K._native, "check", lambda rc: None)
    x0, y = torch.zeros(64), torch.zeros(64, dtype=torch.bfloat16)
    p = K.Program()
    p.input("x", x0)
    with p:
        K.cast_bf16(x0, y)
    inputs = {}

    def work():
        x = torch.zeros(64)
        inputs[threading.get_ident()] = x
        for _ in range(20):
            p.run(x=x)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(seen) == 80
    assert all(count == 1 and at == inputs[who].data_ptr() for who, count, at in seen)

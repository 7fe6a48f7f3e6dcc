"""The surrogate's launches as laid-out programs: a second batch of inputs
through the same program, inputs at another address, a copied network, a
changed batch size and refused inputs give what separate networks give."""
import copy
import pickle

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ARGS = dict(S=256, W=16, Mo=8, L=2, F=9, Hq=32)


def _data(B, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(B, 256, 9, generator=g).cuda(), torch.randn(B, 256, generator=g).cuda()


def _net():
    from mbsolve_gb300 import surrogate
    return surrogate.FNO(surrogate.Shapes(**ARGS), seed=2)


def _step(net, X, t):
    # (before the step: the networks' Adam moments differ)
    y = net.infer(X).clone()
    loss = float(net.train_step(X, t, lr=1e-3).item())
    return loss, net.grad.clone(), y


def _same(a, b):
    # split-K sums meet in any order
    assert a[0] == pytest.approx(b[0], rel=1e-4)
    for x, y in zip(a[1:], b[1:]):
        assert (x - y).norm() <= 1e-3 * y.norm()


def test_programs_follow_their_inputs(native):
    net = _net()
    for B, seed in [(8, 1), (8, 2), (16, 3), (8, 4)]:
        X, t = _data(B, seed)
        fresh = _net()
        fresh.load_params(net.theta)
        _same(_step(net, X, t), _step(fresh, X, t))
    # an input whose storage starts elsewhere, and one that is not contiguous
    X, t = _data(8, 5)
    pad = torch.zeros(X.numel() + 3, device="cuda")
    pad[3:] = X.reshape(-1)
    want = net.forward(X).clone()
    assert (net.forward(pad[3:].view_as(X)) - want).norm() <= 1e-4 * want.norm()
    assert (net.forward(X.transpose(0, 1).contiguous().transpose(0, 1)) - want).norm() <= 1e-4 * want.norm()
    with pytest.raises(ValueError):
        net.forward(X.cpu())
    with pytest.raises(ValueError):
        net.infer(X.double())
    assert (net.forward(X) - want).norm() <= 1e-4 * want.norm()


def test_copies_own_their_programs(native):
    net = _net()
    X, t = _data(8, 1)
    _step(net, X, t)
    before = net.infer(X).clone()
    other = copy.deepcopy(net)
    other.load_params(torch.zeros_like(other.theta))
    assert float(other.infer(X).abs().max()) == 0.0
    assert torch.equal(net.infer(X), before)
    # (a pickled network's parameter views no longer share theta's storage)
    other = pickle.loads(pickle.dumps(net))
    del net
    assert torch.equal(other.infer(X), before)


def test_operation_layout(tmp_path):
    import ctypes as C
    import os
    import shutil
    import subprocess
    from mbsolve_gb300 import capi_types as T
    if shutil.which("gcc") is None:
        pytest.skip("no C compiler")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    names = [("kind", "kind"), ("i", "i"), ("n", "n"), ("in_", "in"), ("out", "out"), ("desc", "desc")]
    src = tmp_path / "op.c"
    src.write_text("#include <stdio.h>\n#include <stddef.h>\n#include \"mbsolve_fno.h\"\nint main(void) {"
                   "printf(\"%zu\", sizeof(mbg_fno_op));" +
                   "".join("printf(\" %%zu\", offsetof(mbg_fno_op, %s));" % c for _, c in names) +
                   "return 0; }\n")
    subprocess.run(["gcc", "-std=c99", "-I", os.path.join(root, "include"), str(src), "-o",
                    str(tmp_path / "op")], check=True)
    got = subprocess.run([str(tmp_path / "op")], check=True, capture_output=True, text=True).stdout
    assert [int(x) for x in got.split()] == [C.sizeof(T.mbg_fno_op)] + \
        [getattr(T.mbg_fno_op, p).offset for p, _ in names]

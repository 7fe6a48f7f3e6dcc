"""Copied and pickled surrogate networks: the parameter and gradient views are
views of the copy's own flat vectors, so that loading and training reach what
the passes read."""
import copy
import pickle

import pytest

torch = pytest.importorskip("torch")

ARGS = dict(S=256, W=16, Mo=8, L=2, F=9, Hq=32)
COPIES = [copy.copy, copy.deepcopy, lambda net: pickle.loads(pickle.dumps(net))]


@pytest.mark.parametrize("how", COPIES)
def test_views_follow_the_flat_vectors(how):
    from mbsolve_gb300 import surrogate
    net = surrogate.FNO(surrogate.Shapes(**ARGS), seed=2, device="cpu")
    other = how(net)
    assert torch.equal(other.theta, net.theta)
    other.load_params(torch.arange(other.theta.numel()))
    other.grad.fill_(3.0)
    at = 0
    for name, _ in other.sh.param_spec():
        p = other.p[name]
        assert torch.equal(p, torch.arange(at, at + p.numel()).float())
        assert bool((other.g[name] == 3.0).all())
        at += p.numel()


@pytest.mark.gpu
@pytest.mark.parametrize("how", COPIES[1:])
def test_a_copy_trains_as_the_original(native, how):
    from mbsolve_gb300 import surrogate
    net = surrogate.FNO(surrogate.Shapes(**ARGS), seed=2)
    g = torch.Generator().manual_seed(1)
    X, t = torch.randn(8, 256, 9, generator=g).cuda(), torch.randn(8, 256, generator=g).cuda()
    net.train_step(X, t, lr=1e-3)
    other = how(net)
    for n in (net, other):
        n.train_step(X, t, lr=1e-3)
    # split-K sums meet in any order
    assert (net.grad - other.grad).norm() <= 1e-3 * net.grad.norm()
    assert float(other.infer(X).abs().max()) > 0
    other.load_params(torch.zeros_like(other.theta))
    assert float(other.infer(X).abs().max()) == 0.0

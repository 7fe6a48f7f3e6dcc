"""Column sums at the edges of their forms: one column to more than a warp's
32, row counts below, at and beyond a slice, row strides beyond the columns.
Inputs are small integers, whose sums are exact in any order."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("cols", [1, 2, 3, 7, 8, 15, 16, 17, 31, 32, 33, 64, 100])
@pytest.mark.parametrize("rows", [1, 5, 31, 32, 33, 1000, 40001])
def test_sums_are_exact(native, rows, cols, pad):
    from mbsolve_gb300 import surrogate_kernels as K
    g = torch.Generator().manual_seed(rows * 128 + cols)
    x = torch.randint(-8, 9, (rows, cols + pad), generator=g).float().cuda()
    out = torch.ones(cols, device="cuda")
    K.colsum(x, rows, cols, cols + pad, out)
    assert torch.equal(out, x[:, :cols].double().sum(0).float() + 1.0)

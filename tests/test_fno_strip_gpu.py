"""Operands of the general product that 16-byte loads cannot read whole: rows
adjacent with an odd K stride (a thread takes one row), K contiguous with an
odd row stride (some rows aligned, some not), neither, batches an odd number
of elements apart, segments of different forms inside one K block; against
float64 products of the same BF16-rounded operands."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 2e-5   # FP32 accumulation of exact BF16 products, relative to max |C|


def _operand(g, batch, rows, k, form, dtype):
    sr, sk = {"rows": (1, rows + 1 - rows % 2), "k": (k + 1 - k % 2, 1), "any": (3, 3 * rows + 1)}[form]
    sz = (rows - 1) * sr + (k - 1) * sk + 2
    v = torch.randn(batch, rows, k, generator=g)
    t = torch.zeros(1 + batch * sz)
    i = 1 + (torch.arange(batch) * sz)[:, None, None] + (torch.arange(rows) * sr)[:, None] + torch.arange(k) * sk
    t[i] = v
    return t.to(dtype).cuda(), sr, sk, sz, v.to(torch.bfloat16).double()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fa", ["rows", "k", "any"])
@pytest.mark.parametrize("fb", ["rows", "k", "any"])
def test_unaligned_operands(native, fa, fb, dtype):
    from mbsolve_gb300 import surrogate_kernels as K
    g = torch.Generator().manual_seed(11)
    other = {"rows": "k", "k": "any", "any": "rows"}
    for batch, m, n, ks in [(1, 128, 64, (64,)), (2, 129, 65, (65,)), (3, 1, 1, (1,)), (1, 7, 200, (130,)),
                            (2, 131, 63, (8, 40, 17))]:
        segs, want = [], 0.0
        for i, k in enumerate(ks):
            a, am, ak, az, av = _operand(g, batch, m, k, fa if i != 1 else other[fa], dtype)
            b, bn, bk, bz, bv = _operand(g, batch, n, k, fb if i != 2 else other[fb], dtype)
            segs.append(K.Seg(a, 1, am, ak, az, b, 1, bn, bk, bz, k, negate=i == 1))
            want = want + (-1.0 if i == 1 else 1.0) * av @ bv.transpose(1, 2)
        c = torch.zeros(batch, m, n, device="cuda")
        K.gemm(m, n, segs, c, 0, n, 1, m * n, batch=batch)
        err = (c.double().cpu() - want).abs().max() / want.abs().max()
        assert err < TOL, (batch, m, n, ks, float(err))
    assert K.status() == 0

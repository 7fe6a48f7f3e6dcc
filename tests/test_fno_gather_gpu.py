"""Operand forms of the general product's gather path (16-byte loads along K,
along the rows with a transpose in registers, element by element) against
float64 products of the same BF16-rounded operands: both storage types, sizes
at and beside multiples of 8 and of a tile, unaligned bases, several segments
inside one K block, negation; and the epilogue by fours (pre, gate, atomic)
beside its scalar form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 2e-5   # FP32 accumulation of exact BF16 products, relative to max |C|


@pytest.fixture(scope="module")
def K(native):
    from mbsolve_gb300 import surrogate_kernels
    return surrogate_kernels


def _operand(g, rows, k, form, dtype, shift):
    """(tensor, offset, row stride, k stride, FP64 values) of a rows x k
    operand stored K-contiguous ("k"), row-contiguous ("r") or with neither
    stride 1 ("any"), starting `shift` elements into its tensor."""
    v = torch.randn(rows, k, generator=g)
    pad = lambda n: (n + 7) // 8 * 8  # noqa: E731
    sr, sk = {"k": (pad(k), 1), "r": (1, pad(rows)), "any": (2 * k + 1, 2)}[form]
    t = torch.zeros(shift + (rows - 1) * sr + (k - 1) * sk + 1)
    i = shift + torch.arange(rows)[:, None] * sr + torch.arange(k)[None, :] * sk
    t[i] = v
    return t.to(dtype).cuda(), shift, sr, sk, v.to(torch.bfloat16).double()


@pytest.mark.parametrize("shift", [0, 8, 1])
@pytest.mark.parametrize("fa,fb", [("k", "r"), ("r", "k"), ("r", "r"), ("any", "r"), ("k", "any")])
@pytest.mark.parametrize("ta,tb", [("f", "b"), ("b", "f"), ("b", "b")])
def test_operand_forms(K, fa, fb, ta, tb, shift):
    ty = {"f": torch.float32, "b": torch.bfloat16}
    g = torch.Generator().manual_seed(7)
    for m, n, ks in [(128, 64, (64,)), (136, 72, (72,)), (127, 63, (65,)),
                     (9, 1, (7,)), (200, 80, (8, 48, 33))]:
        segs, want = [], 0.0
        for i, k in enumerate(ks):
            a, ao, am, ak, av = _operand(g, m, k, fa, ty[ta], shift)
            b, bo, bn, bk, bv = _operand(g, n, k, fb, ty[tb], shift)
            neg = i == 1
            segs.append(K.Seg(a, ao, am, ak, 0, b, bo, bn, bk, 0, k, negate=neg))
            want = want + (-1.0 if neg else 1.0) * (av @ bv.T)
        c = torch.zeros(m, n, device="cuda")
        K.gemm(m, n, segs, c, 0, n, 1)
        err = (c.double().cpu() - want).abs().max() / want.abs().max()
        assert err < TOL, (m, n, ks, float(err))
    assert K.status() == 0


@pytest.mark.parametrize("n,ld", [(64, 64), (68, 68), (64, 65), (66, 68)])
@pytest.mark.parametrize("kind", ["atomic", "pre", "gate", "accum"])
def test_epilogue_by_fours(K, kind, n, ld):
    from mbsolve_gb300 import capi_types as T
    g = torch.Generator().manual_seed(3)
    m, k = 150, 200
    a = torch.randn(m, k, generator=g)
    b = torch.randn(n, k, generator=g)
    c0 = torch.randn(m, ld, generator=g)
    want = a.to(torch.bfloat16).double() @ b.to(torch.bfloat16).double().T
    seg = [K.Seg(a.cuda(), 0, k, 1, 0, b.cuda(), 0, k, 1, 0, k)]
    c = c0.clone().cuda()
    if kind == "atomic":
        K.gemm(m, n, seg, c, 0, ld, 1, mode=T.MBG_GEMM_ATOMIC, split_k=4)
        want = c0[:, :n].double() + want
    elif kind == "accum":
        K.gemm(m, n, seg, c, 0, ld, 1, mode=T.MBG_GEMM_ACCUM)
        want = c0[:, :n].double() + want
    elif kind == "pre":
        pre = torch.zeros(m, ld, device="cuda")
        bias = torch.randn(n, generator=g)
        K.gemm(m, n, seg, c, 0, ld, 1, bias=bias.cuda(), pre=pre, act=T.MBG_ACT_GELU)
        want = want + bias.double()
        assert (pre[:, :n].double().cpu() - want).abs().max() < TOL * want.abs().max()
        want = torch.nn.functional.gelu(want)
    else:
        gate = torch.randn(m, ld, generator=g)
        K.gemm(m, n, seg, c, 0, ld, 1, gate=gate.cuda(), act=T.MBG_ACT_GELU_BWD)
        x = gate[:, :n].double()
        want = want * (0.5 * (1 + torch.erf(x / 2 ** 0.5)) +
                       x * torch.exp(-0.5 * x * x) / (2 * np.pi) ** 0.5)
    assert (c[:, :n].double().cpu() - want).abs().max() < TOL * want.abs().max()
    if ld > n:
        assert torch.equal(c[:, n:].cpu(), c0[:, n:])

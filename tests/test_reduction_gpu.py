"""The split-k reduction in both of its tile widths (32 x 8, and 32 x 32 from four tiles per SM on): sizes
around the tiles, both orders of D, C beside D and in place, more slabs than are read at a
time, and the same kernel without slabs (k == 0).  Integer results are exact; f32 ones are the same
bits whatever the order of D."""
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import STORAGE, layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,split", [(33, 9, 1024, 2), (100, 63, 4096, 9), (300, 1000, 2048, 5), (784, 800, 512, 2),
                                         (769, 801, 1280, 10), (1025, 1023, 640, 3), (40, 20000, 512, 4), (20000, 33, 512, 4),
                                         (801, 769, 0, 0), (65, 7, 0, 0)])
@pytest.mark.parametrize("c_rm", [True, False])
@pytest.mark.parametrize("beta,in_place", [(0, False), (-2, False), (1, True)])
def test_int8(gpu, m, n, k, split, c_rm, beta, in_place):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randint(0, 256, (m, max(k, 1)), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, max(k, 1)), dtype=torch.int8, device="cuda", generator=g)
    shape = (m, n + 1) if c_rm else (n, m + 1)
    C = torch.randint(-1000, 1000, shape, dtype=torch.int32, device="cuda", generator=g)
    D = C if in_place else torch.full(shape, 77, dtype=torch.int32, device="cuda")
    inside = (lambda t: t[:, :n]) if c_rm else (lambda t: t[:, :m].T)
    # |sums| < 2^53: exact in f64
    want = beta * inside(C).clone()
    if k:
        want = want + (A.double() @ B.double().T).to(torch.int32)
    gap = D[:, -1].clone()
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, layout(c_rm))
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, max(k, 1)), c.TensorRef(B, max(k, 1)), c.TensorRef(C, shape[1]),
                         c.TensorRef(D, shape[1]), c.LinearCombination(1, beta), split))
    assert st == c.Status.kSuccess, _capi.last_error()
    assert torch.equal(inside(D), want)
    assert torch.equal(D[:, -1], gap)


@pytest.mark.parametrize("m,n,k,split", [(300, 200, 2048, 6), (801, 769, 1280, 10)])
def test_mx_same_bits_in_both_orders(gpu, m, n, k, split):
    P = W.mx_problem(_capi.FMT_E4M3, m, n, k, True, seed=3)
    A, B, SA, SB = (torch.from_numpy(x).cuda() for x in (P.A, P.B, P.SA, P.SB))
    out = []
    for c_rm in (True, False):
        D = torch.full((m, n) if c_rm else (n, m), float("nan"), device="cuda")
        op = c.GemmMx(STORAGE[P.fmt_a], STORAGE[P.fmt_b], layout(c_rm))
        st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, SA, P.lda, P.ldsa), c.MxTensorRef(B, SB, P.ldb, P.ldsb),
                             c.TensorRef(D, D.shape[1]), c.TensorRef(D, D.shape[1]), c.LinearCombination(1.0, 0.0), split))
        assert st == c.Status.kSuccess, _capi.last_error()
        assert _capi.last_plan().slices == split
        out.append(D if c_rm else D.T)
    assert torch.equal(out[0], out[1])

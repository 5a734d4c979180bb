"""How a call without a forced plan cuts a deep k: wide tiles in slices, where one wave of 64-wide tiles or
of unsplit ones would run twice as many k-blocks one after the other; and no slices where one
wave is short.  Integer results are exact, MX ones those of the same call unsplit."""
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import MX_TOL, STORAGE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,split", [(640, 1024, 16384, True), (1024, 1024, 32768, True), (2560, 256, 16384, True),
                                         (1024, 1024, 1024, False), (128, 4096, 2048, False)])
def test_int8(gpu, m, n, k, split):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randint(0, 256, (m, k), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    D = torch.full((m, n), 77, dtype=torch.int32, device="cuda")
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, c.RowMajor)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, k), c.TensorRef(B, k), c.TensorRef(D, n), c.TensorRef(D, n),
                         c.LinearCombination(1, 0)))
    assert st == c.Status.kSuccess, _capi.last_error()
    plan = _capi.last_plan()
    assert (plan.slices > 1) == split and (plan.tile_n > 64 or not split), (plan.tile_n, plan.slices)
    # |sums| < 2^53: exact in f64
    assert torch.equal(D, (A.double() @ B.double().T).to(torch.int32))


@pytest.mark.parametrize("fmt,m,n,k,split", [
    (_capi.FMT_E4M3, 640, 1024, 16384, True), (_capi.FMT_E4M3, 512, 1024, 32768, True), (_capi.FMT_E4M3, 2560, 256, 16384, True),
    (_capi.FMT_E2M1, 640, 1024, 32768, True), (_capi.FMT_E2M1, 1024, 704, 32768, True), (_capi.FMT_E4M3, 512, 2048, 1024, False),
    (_capi.FMT_E2M1, 512, 2048, 1024, False)])
def test_mx(gpu, fmt, m, n, k, split):
    P = W.mx_problem(fmt, m, n, k, True, seed=k, scale_lo=114, scale_hi=120)
    A, B, SA, SB = (torch.from_numpy(x).cuda() for x in (P.A, P.B, P.SA, P.SB))
    op = c.GemmMx(STORAGE[fmt], STORAGE[fmt])
    out = []
    for slices in (0, 1):
        D = torch.full((m, n), float("nan"), device="cuda")
        st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, SA, P.lda, P.ldsa), c.MxTensorRef(B, SB, P.ldb, P.ldsb),
                             c.TensorRef(D, n), c.TensorRef(D, n), c.LinearCombination(1.0, 0.0), slices))
        assert st == c.Status.kSuccess, _capi.last_error()
        if slices == 0:
            plan = _capi.last_plan()
            assert (plan.slices > 1) == split and (plan.tile_n > 64 or not split), (plan.tile_n, plan.slices)
        out.append(D.double())
    # a running sum drops up to 6.3e-10 per element of k (1e-5 at 16384)
    assert ((out[0] - out[1]).norm() / out[1].norm()).item() <= MX_TOL * max(1.0, k / 16384)

"""MX scales read by the GEMM kernel itself (rows aligned to four or eight bytes) against the same problem
with its scales re-laid-out by a kernel in front of it (a leading dimension that is not a
multiple of four): the same bits, whatever the tile, slice and pair plan, for row counts around
the 128-row groups and k around the scale words of a k-block."""
import numpy as np
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import STORAGE, check_mx

pytestmark = pytest.mark.gpu

F8, F5, F4 = _capi.FMT_E4M3, _capi.FMT_E5M2, _capi.FMT_E2M1


def with_ld(scales, rows, ld, new_ld):
    """The same scale rows at another leading dimension; what follows a row's entries is NaN (255)."""
    out = torch.full((rows, new_ld), 255, dtype=torch.uint8)
    out[:, :ld] = torch.from_numpy(scales).reshape(rows, ld)
    return out.cuda()


@pytest.mark.parametrize("fmt,m,n,k,plan", [
    (F8, 129, 257, 512, {}), (F8, 128, 256, 2048, {}), (F8, 300, 500, 1000, {}), (F8, 70, 33, 513, {}),
    (F8, 1, 1, 33, {}), (F8, 257, 127, 31, {}), (F5, 1000, 1000, 1536, {}), (F8, 700, 900, 4096, {"split": 3}),
    (F8, 192, 320, 8192, {"split": 7}), (F4, 129, 257, 512, {}), (F4, 200, 300, 2000, {"split": 2}),
    (F4, 1000, 1000, 1056, {}), (F4, 2050, 3000, 288, {"pair": True}), (F8, 2050, 3000, 544, {"pair": True}),
    (F8, 300, 4097, 2080, {"pair": True, "tile_n": 192}), (F5, 520, 520, 16384, {"pair": True, "split": 5}),
    (F4, 520, 520, 16416, {"pair": True, "tile_n": 224}), (F8, 4500, 4500, 640, {}), (F4, 6000, 5000, 1024, {})])
def test_same_bits(gpu, oracle, fmt, m, n, k, plan):
    split = plan.get("split", 0)
    kg = (k + 31) // 32
    P = W.mx_problem(fmt, m, n, k, True, seed=m + n + k)
    A, B, C = (torch.from_numpy(x).cuda() for x in (P.A, P.B, P.C))
    op = c.GemmMx(STORAGE[fmt], STORAGE[fmt], tile_n=plan.get("tile_n", 0), pair=plan.get("pair"))
    got = []
    for ld in ((kg + 15) // 16 * 16, (kg + 7) // 8 * 8 + 8, kg + 1 if (kg + 1) % 4 else kg + 2):
        D = torch.full_like(C, float("nan"))
        before = c.launch_count()
        args = op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, with_ld(P.SA, m, P.ldsa, ld), P.lda, ld),
                            c.MxTensorRef(B, with_ld(P.SB, n, P.ldsb, ld), P.ldb, ld), c.TensorRef(C, P.ldc),
                            c.TensorRef(D, P.ldc), c.LinearCombination(1.0, 0.5), split)
        assert op(args) == c.Status.kSuccess, _capi.last_error()
        got.append((D, c.launch_count() - before))
    if m * n * k < 2 ** 28:
        check_mx(oracle, P, got[0][0].cpu().numpy(), 1.0, 0.5)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][0], got[2][0])
    assert not torch.isnan(got[0][0]).any()
    if m > 64 and not plan.get("pair"):
        # (smaller ones take the decode kernel; pairs re-lay the scales out, as 8-bit launches with
        # more work items than SMs over a long k do, of which there is none here)
        assert got[0][1] == got[1][1] == got[2][1] - 1, "the scales were not read by the GEMM kernel"


@pytest.mark.parametrize("a_fmt,b_fmt", [(F8, F5), (F5, F8)])
def test_two_formats(gpu, oracle, a_fmt, b_fmt):
    P = W.mx_problem(a_fmt, 300, 400, 512, True, seed=5, fmt_b=b_fmt)
    D = np.full_like(P.C, np.nan)
    op = c.GemmMx(STORAGE[a_fmt], STORAGE[b_fmt])
    st = op(op.Arguments(c.GemmCoord(P.m, P.n, P.k), c.MxTensorRef(P.A, P.SA, P.lda, P.ldsa),
                         c.MxTensorRef(P.B, P.SB, P.ldb, P.ldsb), c.TensorRef(P.C, P.ldc), c.TensorRef(D, P.ldc),
                         c.LinearCombination(1.0, 0.0)))
    assert st == c.Status.kSuccess, _capi.last_error()
    check_mx(oracle, P, D, 1.0, 0.0)


@pytest.mark.parametrize("fmt,m,n,k,ld_extra", [(F8, 192, 320, 16384, 0), (F8, 300, 300, 4096, 0), (F8, 256, 256, 2048, 1),
                                                (F5, 640, 1024, 4096, 0), (F8, 129, 65, 2080, 1), (F8, 100, 60, 8192, 0)])
def test_pieces_keep_the_precision_of_many_slices(gpu, fmt, m, n, k, ld_extra):
    """Small 8-bit problems that run in few slices sum k in pieces.  Against float64 a running
    sum is off by about 6.3e-10 per element of k, so 256 to 1024 elements give 2e-7 to 6.5e-7; one
    sum over all of k would give more than the bound in every case."""
    kg = (k + 31) // 32
    P = W.mx_problem(fmt, m, n, k, True, seed=k, scale_lo=114, scale_hi=120)
    A, B = (torch.from_numpy(x).cuda() for x in (P.A, P.B))
    SA, SB = with_ld(P.SA, m, P.ldsa, kg + ld_extra), with_ld(P.SB, n, P.ldsb, kg + ld_extra)
    D = torch.full((m, n), float("nan"), device="cuda")
    op = c.GemmMx(STORAGE[fmt], STORAGE[fmt])
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, SA, P.lda, kg + ld_extra),
                         c.MxTensorRef(B, SB, P.ldb, kg + ld_extra), c.TensorRef(D, n), c.TensorRef(D, n),
                         c.LinearCombination(1.0, 0.0)))
    assert st == c.Status.kSuccess, _capi.last_error()
    table = torch.arange(256, dtype=torch.uint8).view(
        torch.float8_e4m3fn if fmt == F8 else torch.float8_e5m2).double().cuda()

    def value(x, s):
        return table[x.reshape(-1, k).long()] * torch.exp2(s[:, :kg].double() - 127).repeat_interleave(32, 1)[:, :k]

    want = value(A, SA) @ value(B, SB).T
    error = ((D.double() - want).norm() / want.norm()).item()
    assert error <= 7e-7, error

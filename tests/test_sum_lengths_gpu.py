"""How long the tensor cores sum before an accumulator is taken down.  They drop the low bits of a
running sum: against float64 a result is off by up to 6.3e-10 per element of k summed in one
accumulator, and by about 2e-7 however short the sums are.  Plans that give a small output few
CTAs must not sum longer than the finer cut of k that every bound here states."""
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import STORAGE

pytestmark = pytest.mark.gpu

F8, F5, F4 = _capi.FMT_E4M3, _capi.FMT_E5M2, _capi.FMT_E2M1


def values(fmt, x, scales, rows, k, ld):
    """The (rows, k) matrix of elements times their scales, in float64."""
    x = x.reshape(rows, -1)
    if fmt == F4:
        positive = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
        v = torch.cat([positive, -positive])[torch.stack([x & 15, x >> 4], -1).reshape(rows, -1).long()]
    else:
        table = torch.arange(256, dtype=torch.uint8).view(torch.float8_e4m3fn if fmt == F8 else torch.float8_e5m2)
        v = table.double().cuda()[x.long()]
    s = torch.exp2(scales.reshape(rows, ld)[:, :(k + 31) // 32].double() - 127)
    return v[:, :k] * s.repeat_interleave(32, 1)[:, :k]


def error(fmt, m, n, k, lds, scale_lo, scale_hi, **options):
    """Normwise error of one call, scale rows `lds` apart."""
    P = W.mx_problem(fmt, m, n, k, True, lds=lds, seed=m + n + k, scale_lo=scale_lo, scale_hi=scale_hi)
    A, B, SA, SB = (torch.from_numpy(x).cuda() for x in (P.A, P.B, P.SA, P.SB))
    D = torch.full((m, n), float("nan"), device="cuda")
    op = c.GemmMx(STORAGE[fmt], STORAGE[fmt], **options)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, SA, P.lda, lds), c.MxTensorRef(B, SB, P.ldb, lds),
                         c.TensorRef(D, n), c.TensorRef(D, n), c.LinearCombination(1.0, 0.0)))
    assert st == c.Status.kSuccess, _capi.last_error()
    want = values(fmt, A, SA, m, k, lds) @ values(fmt, B, SB, n, k, lds).T
    return ((D.double() - want).norm() / want.norm()).item()


def bound(elements):
    return 2e-7 + 6.3e-10 * elements


def bound_e2m1(elements):  # (fewer of the products' bits fall off the end)
    return 1.2e-7 + 2.5e-10 * elements


# 160 k-blocks, once cut in seven (23 k-blocks at most), now in five slices of 32 and pieces of 22
@pytest.mark.parametrize("fmt,m,n,lo", [(F8, 1024, 704, 114), (F5, 2560, 256, 108), (F8, 1792, 384, 114)])
def test_a_plan_in_pieces_stays_with_one_cta_per_tile(gpu, fmt, m, n, lo):
    """As many work items as CTA pairs would want, but pairs sum in one piece."""
    e = error(fmt, m, n, 20480, 640, lo, lo + 6)
    assert _capi.last_plan().pair == 0
    assert e <= bound(23 * 128), e


# Once a CTA per SM shared the tiles' k-blocks evenly; now at most six share a tile and sum their part in
# pieces.  `longest`: k-blocks to a sum then.  One and four 16-column chunks, whole tiles and clusters.
@pytest.mark.parametrize("fmt,lo,m,n,k,longest", [
    (F8, 114, 32, 1024, 14336, 7), (F8, 114, 1, 512, 14336, 4), (F8, 114, 17, 1024, 8192, 4), (F5, 108, 64, 1536, 14336, 10),
    (F8, 114, 64, 4608, 14336, 28), (F8, 114, 8, 1000, 1024, 4), (F8, 114, 40, 1000, 1024, 4), (F8, 114, 33, 130, 2080, 4),
    (F8, 114, 32, 1024, 65536, 28)])
def test_decode_8_bit(gpu, fmt, lo, m, n, k, longest):
    e = error(fmt, m, n, k, -(-k // 512) * 16, lo, lo + 6)
    assert _capi.last_plan().decode == 1
    assert e <= bound(longest * 128), e


# Scales over 15 exponents: sums of e2m1 products no longer fit f32.
@pytest.mark.parametrize("m,n,k,longest", [(32, 1024, 28672, 7), (1, 512, 28672, 4), (64, 1000, 16384, 4), (16, 1000, 2048, 4)])
def test_decode_4_bit(gpu, m, n, k, longest):
    e = error(F4, m, n, k, -(-k // 512) * 16, 120, 134)
    assert _capi.last_plan().decode == 1
    assert e <= bound_e2m1(longest * 256), e


# `longest`: k-blocks of 256 elements to a sum when k was cut by an SM's share of HBM bandwidth.
@pytest.mark.parametrize("m,n,k,longest,lds_extra", [
    (512, 512, 8192, 4, 0), (192, 320, 16384, 3, 0), (256, 512, 16384, 4, 1), (1024, 1024, 8192, 16, 0), (640, 1024, 32768, 32, 0),
    (100, 60, 32768, 4, 0), (128, 128, 4096, 2, 0), (512, 1024, 16384, 13, 0)])
def test_general_4_bit(gpu, m, n, k, longest, lds_extra):
    """Scales over 15 exponents; scale rows that the kernel reads itself, and (an odd leading
    dimension) ones that are re-laid-out."""
    e = error(F4, m, n, k, k // 32 + lds_extra, 120, 134)
    assert e <= bound_e2m1(longest * 256), e

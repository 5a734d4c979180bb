"""256-wide tiles that all run at once go to CTA pairs when the k loop is long enough and no
pair would be half empty; every choice gives the exact integer product."""
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import STORAGE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,beta,pair", [
    (2048, 2048, 2048, 1, 1), (2048, 2048, 2048, 0, 0), (2048, 2048, 1920, 1, 0), (1024, 4096, 4096, 0, 1),
    (1000, 4090, 3200, 1, 1), (1024, 4096, 2944, 0, 0), (1100, 4096, 4096, 0, 0), (2048, 2304, 4096, 1, 1)])
def test_pairs_in_one_wave(gpu, m, n, k, beta, pair):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randint(0, 256, (m, k), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    C = torch.randint(-1000, 1000, (m, n), dtype=torch.int32, device="cuda", generator=g)
    D = torch.full((m, n), 77, dtype=torch.int32, device="cuda")
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, c.RowMajor)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, k), c.TensorRef(B, k), c.TensorRef(C, n),
                         c.TensorRef(D, n), c.LinearCombination(1, beta)))
    assert st == c.Status.kSuccess, _capi.last_error()
    assert (_capi.last_plan().tile_n, _capi.last_plan().pair) == (256, pair)
    # |sums| < 2^53: exact in f64
    assert torch.equal(D, (A.double() @ B.double().T).to(torch.int32) + beta * C)


@pytest.mark.parametrize("k,pair", [(4096, 0), (12160, 0), (12288, 1)])
def test_mx_pairs_in_one_wave(gpu, k, pair):
    """One CTA per tile reads the scales itself, which is worth more than the pair until k has 96
    k-blocks; the same bits in both forms."""
    m, n = 2048, 2304
    P = W.mx_problem(_capi.FMT_E4M3, m, n, k, True, seed=k, scale_lo=114, scale_hi=120)
    A, B, SA, SB = (torch.from_numpy(x).cuda() for x in (P.A, P.B, P.SA, P.SB))
    out = []
    for form in (None, not pair):
        D = torch.full((m, n), float("nan"), device="cuda")
        op = c.GemmMx(STORAGE[P.fmt_a], STORAGE[P.fmt_b], pair=form)
        st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, SA, P.lda, P.ldsa), c.MxTensorRef(B, SB, P.ldb, P.ldsb),
                             c.TensorRef(D, n), c.TensorRef(D, n), c.LinearCombination(1.0, 0.0)))
        assert st == c.Status.kSuccess, _capi.last_error()
        assert (_capi.last_plan().tile_n, _capi.last_plan().pair) == (256, pair if form is None else 1 - pair)
        out.append(D)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("m,n,k,tile_n", [(512, 512, 512, 64), (1000, 900, 300, 64), (129, 65, 128, 64), (1024, 1216, 512, 128),
                                          (128, 9472, 256, 64), (100, 200, 1500, 64), (60, 70, 333, 64)])
def test_narrow_tiles_in_one_wave(gpu, m, n, k, tile_n):
    """64-wide tiles while all of them run at once (1024 x 1216: 152 tiles on 148 SMs do not)."""
    k = (k + 15) // 16 * 16
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randint(0, 256, (m, k), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    C = torch.randint(-1000, 1000, (m, n), dtype=torch.int32, device="cuda", generator=g)
    D = torch.full((m, n), 77, dtype=torch.int32, device="cuda")
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, c.RowMajor)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, k), c.TensorRef(B, k), c.TensorRef(C, n),
                         c.TensorRef(D, n), c.LinearCombination(1, 1), 1))
    assert st == c.Status.kSuccess, _capi.last_error()
    assert (_capi.last_plan().tile_n <= 64) == (tile_n == 64)
    assert torch.equal(D, (A.double() @ B.double().T).to(torch.int32) + C)

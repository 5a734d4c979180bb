"""Device operands that TMA cannot address: C and D whose base or leading dimension is not a
multiple of 16 bytes (rows through the shared-memory ring by cp.async and plain stores), C
with contiguous columns (lane = row), one of the two addressable and the other not, and A and
B at odd addresses (copied into aligned rows first).  Sizes around the 32 x 32 chunks of the
epilogue and the 512-byte pieces of the copy.  Integer results must match the oracle bit for
bit, f32 ones the oracle's within the MX tolerance; what lies between the rows of D stays."""
import numpy as np
import pytest
import torch

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W
from tests.gpu_helpers import MX_TOL, STORAGE, gather, layout, normwise, run_int8_oracle, run_mx_oracle

pytestmark = pytest.mark.gpu


def on_device(x, shift):
    """A device copy of the flat array whose first element sits `shift` elements past a
    256-byte boundary."""
    t = torch.zeros(x.size + shift, dtype=torch.from_numpy(x[:1]).dtype, device="cuda")
    t[shift:] = torch.from_numpy(x).cuda()
    return t[shift:]


def call(op, m, n, k, a, b, C, ldc, beta, ldd, c_rm, shift, in_place):
    dC = on_device(C, shift)
    rows = m if c_rm else n
    D = dC if in_place else torch.full((rows * ldd + shift,), 77, dtype=dC.dtype, device="cuda")[shift:]
    before = D.clone()
    st = op(op.Arguments(c.GemmCoord(m, n, k), a, b, c.TensorRef(dC, ldc), c.TensorRef(D, ldc if in_place else ldd),
                         c.LinearCombination(3, beta)))
    assert st == c.Status.kSuccess, _capi.last_error()
    return D.cpu().numpy(), before.cpu().numpy(), (ldc if in_place else ldd)


def gaps_untouched(D, before, m, n, ld, c_rm):
    rows, cols = (m, n) if c_rm else (n, m)
    gap = np.ones(D.size, bool)
    for r in range(rows):
        gap[r * ld:r * ld + cols] = False
    assert np.array_equal(D[gap], before[gap]), "an element outside D was written"


# (m, n, k, row-major C, padding of the leading dimensions, element offset of the bases, in place)
CASES = [(129, 257, 513, True, 3, 0, False), (129, 257, 513, False, 3, 1, True), (33, 31, 1, True, 3, 1, True),
         (300, 1000, 97, True, 0, 1, False), (300, 1001, 529, True, 1, 0, True), (65, 32, 16, False, 3, 0, False),
         (1, 259, 1025, True, 3, 3, False), (1030, 1, 130, False, 2, 1, False), (1, 1, 5, True, 3, 1, True),
         (257, 4099, 300, True, 3, 0, False), (640, 96, 2000, True, 3, 0, False), (40, 333, 700, True, 3, 1, False)]


@pytest.mark.parametrize("a_rm,b_rm", [(True, True), (False, False), (True, False)])
@pytest.mark.parametrize("m,n,k,c_rm,pad,shift,in_place", CASES)
def test_int8(gpu, oracle, m, n, k, c_rm, pad, shift, in_place, a_rm, b_rm):
    P = W.int8_problem(m, n, k, a_rm, b_rm, c_rm, pad=pad, seed=m + n + k, full_range=True, c_range=1000)
    for beta in (0, -2):
        want = gather(run_int8_oracle(oracle, P, 3, beta), m, n, P.ldc, c_rm)
        op = c.GemmU8S8S32(layout(a_rm), layout(b_rm), layout(c_rm))
        D, before, ldd = call(op, m, n, k, c.TensorRef(on_device(P.A, shift), P.lda),
                              c.TensorRef(on_device(P.B, shift), P.ldb), P.C, P.ldc, beta, P.ldc + 2, c_rm, shift, in_place)
        assert np.array_equal(gather(D, m, n, ldd, c_rm), want)
        gaps_untouched(D, before, m, n, ldd, c_rm)


# one of C and D addressable by TMA, the other not; several tiles per CTA or pair
@pytest.mark.parametrize("c_pad,d_pad", [(0, 1), (1, 0), (1, 2)])
@pytest.mark.parametrize("m,n,k,pair", [(512, 768, 256, None), (4200, 4200, 1024, True), (2300, 4200, 256, False)])
def test_mixed_rings(gpu, m, n, k, pair, c_pad, d_pad):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.randint(0, 256, (m, k), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    C = torch.randint(-1000, 1000, (m, n + c_pad), dtype=torch.int32, device="cuda", generator=g)
    D = torch.full((m, n + d_pad), 77, dtype=torch.int32, device="cuda")
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, c.RowMajor, pair=pair)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, k), c.TensorRef(B, k), c.TensorRef(C, n + c_pad),
                         c.TensorRef(D, n + d_pad), c.LinearCombination(1, 1)))
    assert st == c.Status.kSuccess, _capi.last_error()
    # |sums| < 2^24 * 2: exact in f64
    want = (A.double() @ B.double().T).to(torch.int32) + C[:, :n]
    assert torch.equal(D[:, :n], want)
    assert bool((D[:, n:] == 77).all())


@pytest.mark.parametrize("m,n,k,pair", [(520, 771, 256, None), (4200, 4199, 512, True), (3000, 4097, 128, False)])
def test_rows_beside_tma_in_place(gpu, m, n, k, pair):
    """C == D with an aligned leading dimension and n not a multiple of four: C arrives by TMA in
    the buffers that D leaves by rows, and every warp refills each buffer many times."""
    ld = (n + 3) // 4 * 4
    g = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.randint(0, 256, (m, k), dtype=torch.uint8, device="cuda", generator=g)
    B = torch.randint(-128, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    C = torch.randint(-1000, 1000, (m, ld), dtype=torch.int32, device="cuda", generator=g)
    # |sums| < 2^53: exact in f64
    want = (A.double() @ B.double().T).to(torch.int32) + C[:, :n]
    gap = C[:, n:].clone()
    op = c.GemmU8S8S32(c.RowMajor, c.ColumnMajor, c.RowMajor, pair=pair)
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.TensorRef(A, k), c.TensorRef(B, k), c.TensorRef(C, ld),
                         c.TensorRef(C, ld), c.LinearCombination(1, 1)))
    assert st == c.Status.kSuccess, _capi.last_error()
    assert torch.equal(C[:, :n], want)
    assert torch.equal(C[:, n:], gap)


@pytest.mark.parametrize("fmt,k", [(_capi.FMT_E4M3, 200), (_capi.FMT_E2M1, 333), (_capi.FMT_E2M1, 1152)])
@pytest.mark.parametrize("c_rm,shift", [(True, 0), (True, 1), (False, 1)])
def test_mx(gpu, oracle, fmt, k, c_rm, shift):
    m, n = 193, 301
    P = W.mx_problem(fmt, m, n, k, c_rm, pad=3, seed=k, scale_lo=124, scale_hi=130)
    want = gather(run_mx_oracle(oracle, P, 3.0, 0.5), m, n, P.ldc, c_rm)
    op = c.GemmMx(STORAGE[fmt], STORAGE[fmt], layout(c_rm))
    a = c.MxTensorRef(on_device(P.A, shift), on_device(P.SA, shift), P.lda, P.ldsa)
    b = c.MxTensorRef(on_device(P.B, shift), on_device(P.SB, shift), P.ldb, P.ldsb)
    D, before, ldd = call(op, m, n, k, a, b, P.C, P.ldc, 0.5, P.ldc + 1, c_rm, shift, False)
    assert normwise(gather(D, m, n, ldd, c_rm), want) <= MX_TOL
    gaps_untouched(D, before, m, n, ldd, c_rm)

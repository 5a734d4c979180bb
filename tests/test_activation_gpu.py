"""Gelu and Silu over the whole range of f32: the large arguments on either side, where the
denominator overflows or the exponential vanishes, zeros, infinities and NaN, both in the
GEMM kernel's epilogue and in the element-wise kernel behind k == 0."""
import numpy as np
import pytest

import cpu_ops_b200 as c
from cpu_ops_b200 import _capi, workloads as W

pytestmark = pytest.mark.gpu

VALUES = np.concatenate([
    np.linspace(-100, 100, 4001), [0.0, -0.0, 1e-30, -1e-30, 1e30, -1e30, 87.2, -87.2, -87.4, 88.8, -88.8, 3.4e38],
    [np.inf, -np.inf, np.nan]]).astype(np.float32)


def want(name, v):
    """(value, factor on the argument's rounding error) in float64."""
    v = v.astype(np.float64)
    with np.errstate(all="ignore"):
        x = v if name == "silu" else 2.0 * np.float64(np.float32(0.7978845608028654)) * (
            v + np.float64(np.float32(0.044715)) * v * v * v)
        y = v / (1.0 + np.exp(-x))
    return y, np.abs(x) if name == "gelu" else np.zeros_like(x)


@pytest.mark.parametrize("name", ["silu", "gelu"])
@pytest.mark.parametrize("k", [0, 32])
def test_whole_range(gpu, name, k):
    m, n = 128, 256
    v = np.resize(VALUES, m * n).astype(np.float32)
    P = W.mx_problem(_capi.FMT_E4M3, m, n, max(k, 32), True, seed=1)
    A = np.zeros_like(P.A)  # acc = 0: the chain sees beta * C = C
    D = np.zeros_like(v)
    op = c.GemmMxE4M3()
    epi = c.LinearCombinationFused(1.0, 1.0, [c.Silu() if name == "silu" else c.Gelu()])
    st = op(op.Arguments(c.GemmCoord(m, n, k), c.MxTensorRef(A, P.SA, P.lda, P.ldsa),
                         c.MxTensorRef(P.B, P.SB, P.ldb, P.ldsb), c.TensorRef(v, n), c.TensorRef(D, n), epi))
    assert st == c.Status.kSuccess, _capi.last_error()
    y, slope = want(name, v)
    finite = np.isfinite(y)
    with np.errstate(all="ignore"):
        assert np.array_equal(np.isnan(D), np.isnan(y))
        assert np.array_equal(D[~finite & ~np.isnan(y)], y[~finite & ~np.isnan(y)].astype(np.float32))
    # expf 1 ulp (2 eps' with eps' = 2^-24), the sum, the reciprocal after its Newton step and the
    # product one rounding each, the step itself up to one more: 6 eps'; Gelu's argument carries
    # five roundings, which the exponential multiplies by |argument|.  Below -87.3 the result
    # (at most 88 / 2^126) is flushed to zero.
    eps = 2.0 ** -24
    bound = np.abs(y[finite]) * eps * (6 + 5 * np.minimum(slope[finite], 90)) + 88 / 2.0 ** 126
    err = np.abs(D[finite].astype(np.float64) - y[finite])
    worst = np.argmax(err / bound)
    assert np.all(err <= bound), (v[finite][worst], D[finite][worst], y[finite][worst])

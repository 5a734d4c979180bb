"""Gelu and Silu over the whole range of f32: the large arguments on either side, where the
denominator overflows or the exponential vanishes, zeros, infinities and NaN, both in the
GEMM kernel's epilogue and in the element-wise kernel behind k == 0."""
import numpy as np
import pytest
import torch

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
    # expf 1 ulp (2 eps' with eps' = 2^-24), the sum and the quotient one rounding each: Silu 4 eps' down
    # to the smallest normal number.  Gelu: the reciprocal one ulp, a product, and its argument's five
    # roundings, which the exponential multiplies by |argument|; above zero all of it only counts by
    # the part exp(-x) that is taken off, and below -87 the exponential itself is subnormal.
    eps = 2.0 ** -24
    x = slope[finite]
    if name == "silu":
        # (below -88.72 the exponential overflows f32 and the quotient is zero)
        bound = np.abs(y[finite]) * np.where(v[finite] < -88.72, 1, eps * 4) + 2.0 ** -126
    else:
        part = np.where(v[finite] > 0, np.exp(-x), 1.0)
        bound = np.abs(y[finite]) * eps * (1 + part * (6 + 5 * np.minimum(x, 90))) + 88 / 2.0 ** 126
    err = np.abs(D[finite].astype(np.float64) - y[finite])
    worst = np.argmax(err / bound)
    assert np.all(err <= bound), (v[finite][worst], D[finite][worst], y[finite][worst])


def run(v, chain):
    """The chain on the f32 matrix v, behind acc = 0 and beta = 1."""
    m, n = v.shape
    zero = lambda rows: torch.zeros(rows, 32, dtype=torch.uint8, device="cuda")  # noqa: E731
    scales = lambda rows: torch.full((rows, 4), 127, dtype=torch.uint8, device="cuda")  # noqa: E731
    D = torch.empty_like(v)
    op = c.GemmMxE4M3()
    st = op(op.Arguments(c.GemmCoord(m, n, 32), c.MxTensorRef(zero(m), scales(m), 32, 4),
                         c.MxTensorRef(zero(n), scales(n), 32, 4), c.TensorRef(v, n), c.TensorRef(D, n),
                         c.LinearCombinationFused(1.0, 1.0, chain)))
    assert st == c.Status.kSuccess, _capi.last_error()
    return D


def arguments(lo, hi):
    g = torch.Generator(device="cuda").manual_seed(1)
    return torch.rand((1024, 2048), device="cuda", generator=g) * (hi - lo) + lo


@pytest.mark.parametrize("lo,hi", [(-88.7, -80.0), (-80.0, -6.0), (-6.0, -1.0), (-1.0, 1.0), (1.0, 17.0), (17.0, 90.0)])
def test_silu_is_the_ieee_quotient(gpu, lo, hi):
    """v / (1 + exp(-v)) as torch divides it on the device, but for near ties (the corrected quotient is
    within half an ulp and a few 2^-24 ulp), and as close to float64."""
    v = arguments(lo, hi)
    got, quotient = run(v, [c.Silu()]), v / (1 + torch.exp(-v))
    exact = v.double() / (1 + torch.exp(-v.double()))
    assert (got != quotient).double().mean().item() <= 1e-5
    assert (got.view(torch.int32) - quotient.view(torch.int32)).abs().max().item() <= 1
    rms = lambda d: ((d.double() - exact) / exact).square().mean().sqrt().item()  # noqa: E731
    assert rms(got) <= rms(quotient) * 1.0001


@pytest.mark.parametrize("lo,hi", [(-6.0, -1.0), (-1.0, 1.0), (1.0, 6.0), (6.0, 30.0)])
def test_gelu_is_no_further_off_than_with_tanh(gpu, lo, hi):
    v = arguments(lo, hi)
    u = 0.7978845608028654 * (v + 0.044715 * v * v * v)
    x = v.double()
    exact = x / (1 + torch.exp(-2 * 0.7978845608028654 * (x + 0.044715 * x ** 3)))
    rms = lambda d: ((d.double() - exact) / exact).square().mean().sqrt().item()  # noqa: E731
    worst = lambda d: ((d.double() - exact) / exact).abs().max().item()  # noqa: E731
    got, tanh = run(v, [c.Gelu()]), 0.5 * (v * (1 + torch.tanh(u)))
    assert rms(got) <= rms(tanh) * 1.001
    assert worst(got) <= worst(tanh) * 1.05

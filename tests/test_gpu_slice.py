"""The FP64 product on digit planes (tensor cores) at the sizes where it can go wrong: edges of its 128-row and 16- or
64-column tiles, K remainders, split K, wide value ranges, infinities and NaN.

Bound: with z and x cut at 2^-63 of their scales (a power of two at most twice the largest entry of the row or vector)
and the digit pairs of levels 8 and up dropped (at most 7 x 2^14 x 2^48 of 2^124, all pairs below it less), a real
product is off by at most 2^-59 + 2 x 2^-63 < 2^-58 of the two scales, a complex entry's 2n products by 2n x 4 x 2^-58
of the maxima, and the result by its own rounding.  FP32: cut at 2^-31, levels 4 and up dropped (at most 3 x 2^14 x 2^16 of
2^60 and less below it): 2^-28 of the two scales."""
from fractions import Fraction

import numpy as np
import pytest

from emfa_gb300 import api

pytestmark = pytest.mark.gpu


def _run(ctx, z, x, mode="auto"):
    import torch
    return api.matvec(ctx, torch.from_numpy(z).cuda(), torch.from_numpy(x).cuda(), mode).cpu().numpy()


def _exact(zr, xr):
    re = im = Fraction(0)
    for a, b in zip(zr, xr):
        ar, ai, br, bi = Fraction(a.real), Fraction(a.imag), Fraction(b.real), Fraction(b.imag)
        re += ar * br - ai * bi
        im += ar * bi + ai * br
    return re, im


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("n,r", [(256, 4), (257, 8), (271, 9), (384, 33), (640, 65), (513, 130), (256, 520)])
@pytest.mark.parametrize("kind", ["normal", "graded", "extreme"])
def test_slice_product_against_exact_sums(ctx, n, r, kind):
    rng = np.random.default_rng(n * 1000 + r)
    z, x = _cplx(rng, n, n), _cplx(rng, r, n)
    if kind == "graded":  # rows over sixty decades, entries of a row over ten, a dominant diagonal
        z *= 10.0 ** rng.uniform(-30, 30, (n, 1)) * 10.0 ** rng.uniform(-10, 0, (n, n))
        x *= 10.0 ** rng.uniform(-30, 30, (r, 1))
        z[np.arange(n), np.arange(n)] *= 1e3
    if kind == "extreme":  # the largest digit sums: every entry the largest below a power of two, signs aligned
        z = np.full((n, n), 1 - 2.0 ** -53) * (1 + 1j)
        x = np.full((r, n), -(1 - 2.0 ** -53)) * (1 - 1j)
        z[1::3] *= 2.0 ** -1000
        x[1::2] *= 2.0 ** 900
        z[2::5] *= 0.0
    y = _run(ctx, z, x)
    for f, s in [(0, 0), (n - 1, r - 1), (n // 2, r // 2), (127, 0), (128, r - 1), (1, 1), (2, 2), (n - 2, r // 3)]:
        re, im = _exact(z[f], x[s])
        big = max(abs(z[f].real).max(), abs(z[f].imag).max()), max(abs(x[s].real).max(), abs(x[s].imag).max())
        tol = Fraction(2 * n * 4) * Fraction(big[0]) * Fraction(big[1]) / 2 ** 58
        for got, want in ((y[s, f].real, re), (y[s, f].imag, im)):
            assert abs(Fraction(got) - want) <= tol + abs(want) / 2 ** 52 + Fraction(1, 2 ** 1073), (f, s, got, float(want))


def test_slice_product_is_no_worse_than_the_cuda_core_one(ctx):
    """Entries of unit variance: both paths against sums of the FP64 products in extended precision."""
    rng = np.random.default_rng(5)
    z, x = _cplx(rng, 700, 700), _cplx(rng, 16, 700)
    rows = slice(0, 40)
    want = np.array([[complex(float(a), float(b)) for a, b in [_exact(z[f], xr)]][0] for xr in x[:4] for f in range(40)])
    a = _run(ctx, z, x)[:4, rows].reshape(-1)
    b = _run(ctx, z, x, "f64")[:4, rows].reshape(-1)
    assert np.linalg.norm(a - want) <= np.linalg.norm(b - want)


def test_slice_product_keeps_infinities_and_nans(ctx):
    rng = np.random.default_rng(6)
    z, x = _cplx(rng, 300, 300), _cplx(rng, 20, 300)
    z[7, 11] = np.inf
    z[130, 0] = complex(0, np.nan)
    x[3, 5] = complex(-np.inf, 0)
    x[17, 299] = np.nan
    a, b = _run(ctx, z, x), _run(ctx, z, x, "f64")
    for p in (np.real, np.imag):
        assert np.array_equal(np.isnan(p(a)), np.isnan(p(b)))
        assert np.array_equal(np.isposinf(p(a)), np.isposinf(p(b))) and np.array_equal(np.isneginf(p(a)), np.isneginf(p(b)))
    ok = np.isfinite(b)
    assert ok.sum() > 290 * 17
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12


def test_slice_product_of_two_shapes_in_turn(ctx):
    """The workspaces of a larger product serve a smaller one and the other way round."""
    rng = np.random.default_rng(7)
    ops = [(_cplx(rng, n, n), _cplx(rng, r, n)) for n, r in ((512, 96), (300, 5), (700, 31))]
    first = [_run(ctx, z, x) for z, x in ops]
    for (z, x), y in list(zip(ops, first))[::-1]:
        assert np.array_equal(_run(ctx, z, x), y)


@pytest.mark.parametrize("n,r", [(128, 17), (257, 18), (271, 17), (384, 64), (640, 65), (513, 130), (256, 520)])
@pytest.mark.parametrize("kind", ["normal", "graded", "extreme"])
def test_fp32_slice_product_against_exact_sums(ctx, n, r, kind):
    rng = np.random.default_rng(n * 1000 + r + 7)
    z, x = _cplx(rng, n, n), _cplx(rng, r, n)
    if kind == "graded":
        z *= 10.0 ** rng.uniform(-8, 8, (n, 1)) * 10.0 ** rng.uniform(-5, 0, (n, n))
        x *= 10.0 ** rng.uniform(-8, 8, (r, 1))
        z[np.arange(n), np.arange(n)] *= 1e3
    if kind == "extreme":
        z = np.full((n, n), 1 - 2.0 ** -24) * (1 + 1j)
        x = np.full((r, n), -(1 - 2.0 ** -24)) * (1 - 1j)
        z[1::3] *= 2.0 ** -60
        x[1::2] *= 2.0 ** 50
        z[2::5] *= 0.0
    z, x = z.astype(np.complex64), x.astype(np.complex64)
    y = _run(ctx, z, x)
    zd, xd = z.astype(np.complex128), x.astype(np.complex128)
    for f, s in [(0, 0), (n - 1, r - 1), (n // 2, r // 2), (127, 0), (min(128, n - 1), r - 1), (1, min(1, r - 1)), (n - 2, r // 3)]:
        re, im = _exact(zd[f], xd[s])
        big = max(abs(zd[f].real).max(), abs(zd[f].imag).max()), max(abs(xd[s].real).max(), abs(xd[s].imag).max())
        tol = Fraction(2 * n * 4) * Fraction(big[0]) * Fraction(big[1]) / 2 ** 28
        for got, want in ((y[s, f].real, re), (y[s, f].imag, im)):
            assert abs(Fraction(float(got)) - want) <= tol + abs(want) / 2 ** 23 + Fraction(1, 2 ** 148), (f, s, got, float(want))


def test_fp32_slice_product_keeps_infinities_and_nans(ctx):
    rng = np.random.default_rng(8)
    z, x = _cplx(rng, 300, 300).astype(np.complex64), _cplx(rng, 20, 300).astype(np.complex64)
    z[7, 11] = np.inf
    z[130, 0] = complex(0, np.nan)
    x[3, 5] = complex(-np.inf, 0)
    x[17, 299] = np.nan
    a, b = _run(ctx, z, x), _run(ctx, z, x, "f32")
    for p in (np.real, np.imag):
        assert np.array_equal(np.isnan(p(a)), np.isnan(p(b)))
        assert np.array_equal(np.isposinf(p(a)), np.isposinf(p(b))) and np.array_equal(np.isneginf(p(a)), np.isneginf(p(b)))
    ok = np.isfinite(b)
    assert ok.sum() > 290 * 17
    assert np.abs(a[ok] - b[ok]).max() <= 1e-3

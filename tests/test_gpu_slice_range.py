"""Products on digit planes over wide ranges: columns of Z scaled against x, components far apart, a row's largest entry
that meets a zero.  The error of every component is held against S, the sum of the magnitudes of that component's own
products, and not against the row's and the vector's maxima.

Bounds.  FP64: a digit result is kept where 2 n 2^-60.8 of the scales is at most (2 ceil(n / 32) + 5) 2^-52 S; a result
summed again is a chain of 2 ceil(n / 256) FMAs a thread, 5 additions across a warp and 7 across the warps, less than
that.  FP32: the digits' bound is (2 ceil(n / 32) + 5) 2^-23 S; the tiles' chain, of at most 2 n FMAs and eight parts, is
off by at most (2 n + 8) 2^-23 S (first order; the rounding is 2^-24, twice that covers the rest)."""
from fractions import Fraction

import numpy as np
import pytest

from emfa_gb300 import api

pytestmark = pytest.mark.gpu


def _run(ctx, z, x, mode="auto"):
    import torch
    return api.matvec(ctx, torch.from_numpy(z).cuda(), torch.from_numpy(x).cuda(), mode).cpu().numpy()


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _operands(rng, n, r, kind):
    z, x = _cplx(rng, n, n), _cplx(rng, r, n)
    if kind.startswith("scaled"):  # D Z D^p with x / D^p, D over some decades
        p, decades = {"scaled1": (1, 4), "scaled2": (2, 4), "scaled8": (2, 8), "scaled_half": (1, 1)}[kind]
        d = 10.0 ** rng.uniform(-decades / 2, decades / 2, n)
        z *= d[:, None] * d[None, :] ** p
        x /= d[None, :] ** p
    if kind == "components":  # real parts large, imaginary parts small, of either operand
        z, x = z.real + 1e-9j * z.imag, x.real + 1e-11j * x.imag
    if kind == "blind":  # the largest entry of every row meets the smallest of x
        z[:, 3] *= 1e9
        x[:, 3] *= 1e-10
    if kind == "empty":  # rows and right-hand sides with nothing or one entry
        z[5] = 0
        z[7] = 0
        z[7, n - 1] = 1e-30j
        x[2] = 0
        x[3] = 0
        x[3, 0] = 1e-25
    return z, x


KINDS = ["scaled_half", "scaled1", "scaled2", "scaled8", "components", "blind", "empty"]


@pytest.mark.parametrize("n,r", [(300, 40), (513, 41)])
@pytest.mark.parametrize("kind", KINDS)
def test_fp64_components_against_their_own_magnitudes(ctx, n, r, kind):
    rng = np.random.default_rng(100 * n + r + len(kind))
    z, x = _operands(rng, n, r, kind)
    y = _run(ctx, z, x)
    bound = Fraction(2 * ((n + 31) // 32) + 5) / 2 ** 52
    for f, s in [(0, 0), (5, 1), (7, r - 1), (7, 3), (n - 1, 2), (n // 2, 3), (n - 1, r - 1), (256, 0), (255, 4), (n // 3, r // 2)]:
        re = im = sr = si = Fraction(0)
        for a, b in zip(z[f], x[s]):
            p = [Fraction(v) for v in (a.real, a.imag, b.real, b.imag)]
            re += p[0] * p[2] - p[1] * p[3]
            im += p[0] * p[3] + p[1] * p[2]
            sr += abs(p[0] * p[2]) + abs(p[1] * p[3])
            si += abs(p[0] * p[3]) + abs(p[1] * p[2])
        assert abs(Fraction(y[s, f].real) - re) <= bound * sr, (f, s, float(abs(Fraction(y[s, f].real) - re) / sr))
        assert abs(Fraction(y[s, f].imag) - im) <= bound * si, (f, s, float(abs(Fraction(y[s, f].imag) - im) / si))


@pytest.mark.parametrize("n,r", [(1201, 520), (2111, 299), (1030, 600)])
@pytest.mark.parametrize("kind", KINDS)
def test_fp32_components_against_their_own_magnitudes(ctx, n, r, kind):
    rng = np.random.default_rng(100 * n + r + len(kind))
    z, x = (a.astype(np.complex64) for a in _operands(rng, n, r, kind))
    y = _run(ctx, z, x)
    zd, xd = z.astype(np.complex128), x.astype(np.complex128)
    want = xd @ zd.T
    zr, zi, xr, xi = abs(zd.real).T, abs(zd.imag).T, abs(xd.real), abs(xd.imag)
    bound, tiny = (2 * n + 8) * 2.0 ** -23, 4 * n * 2.0 ** -149
    for part, s in ((np.real, xr @ zr + xi @ zi), (np.imag, xr @ zi + xi @ zr)):
        assert (abs(part(y) - part(want)) <= bound * s + tiny).all()
    # and as a whole no worse than the explicit FP32 product by more than the noise of its sums
    if kind not in ("empty", "components"):
        other = _run(ctx, z, x, "f32")
        s = xr @ zr + xi @ zi + xr @ zi + xi @ zr
        assert np.linalg.norm((y - want) / s) <= 1.2 * np.linalg.norm((other - want) / s)


def test_a_small_entry_beside_a_large_one_counts(ctx):
    """(1, 1e-10) times (1e-10, 1), in blocks on both sides of the width from which the planes are taken."""
    for r in (64, 96, 1000):
        z = np.zeros((640, 640), np.complex64)
        z[:, 0], z[:, 1] = 1, 1e-10
        x = np.zeros((r, 640), np.complex64)
        x[:, 0], x[:, 1] = 1e-10, 1
        y = _run(ctx, z, x)
        assert abs(y - 2e-10).max() <= 1e-16

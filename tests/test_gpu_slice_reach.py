"""The digit planes at shapes that take them: the kernels that ran are told by the launches (five a block of up to 512
right-hand sides and rows in FP64: split, right-hand sides, product, magnitudes, combination; the masked tiles too in FP32),
so that a change of the dispatch cannot leave these tests to other kernels unnoticed."""
import numpy as np
import pytest

from emfa_gb300 import api
from test_gpu_slice import test_fp32_slice_product_against_exact_sums as fp32_check
from test_gpu_slice import test_slice_product_against_exact_sums as fp64_check

pytestmark = pytest.mark.gpu


def _launches(ctx, call):
    before = ctx.launches()
    out = call()
    return ctx.launches() - before, out


# rows: edges of the 128-row tiles; right-hand sides: the 16-column tile (up to 8), one and two 64-column tiles, two blocks
@pytest.mark.parametrize("n,r,blocks", [(257, 33, 1), (271, 65, 1), (383, 32, 1), (481, 17, 1), (641, 8, 1), (1023, 31, 1), (2049, 4, 1),
                                        (129, 513, 2)])
def test_fp64_shapes(ctx, n, r, blocks):
    for kind in ("normal", "extreme"):
        launches, _ = _launches(ctx, lambda: fp64_check(ctx, n, r, kind))
        assert launches == 1 + 4 * blocks


# the 32-column tile is left for the last 1 to 16 of a block; 128-column tiles, their edges, and K split over CTAs
@pytest.mark.parametrize("n,r,blocks", [(1201, 520, 2), (1291, 513, 2), (2111, 299, 1), (4099, 161, 1)])
def test_fp32_shapes(ctx, n, r, blocks):
    for kind in ("normal", "extreme"):
        launches, _ = _launches(ctx, lambda: fp32_check(ctx, n, r, kind))
        assert launches == 1 + 5 * blocks


@pytest.mark.parametrize("precision,n,r", [("f32", 1201, 520), ("f32", 2111, 299), ("f64", 513, 130), ("f64", 700, 8)])
def test_infinities_and_nans(ctx, precision, n, r):
    import torch
    c = torch.complex64 if precision == "f32" else torch.complex128
    g = torch.Generator(device="cuda").manual_seed(n)
    z = torch.randn(n, n, dtype=c, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=c, device="cuda", generator=g)
    z[7, 11] = float("inf")
    z[130, 0] = complex(0, float("nan"))
    z[n - 1, n - 1] = complex(0, -float("inf"))
    x[3, 5] = complex(-float("inf"), 0)
    x[r - 1, n - 1] = float("nan")
    launches, y = _launches(ctx, lambda: api.matvec(ctx, z, x))
    assert launches >= 5
    want = api.matvec(ctx, z, x, precision)
    y, want = torch.view_as_real(y).cpu().numpy(), torch.view_as_real(want).cpu().numpy()
    assert np.array_equal(np.isnan(y), np.isnan(want))
    assert np.array_equal(np.isposinf(y), np.isposinf(want)) and np.array_equal(np.isneginf(y), np.isneginf(want))
    ok = np.isfinite(want)
    assert ok.sum() > 2 * (n - 3) * (r - 2) - 1
    # both within (2 n + 8) eps of sum |z||x|, here at most n times about 16
    assert abs(y[ok] - want[ok]).max() <= 2 * (2 * n + 8) * np.finfo(y.dtype).eps * 16 * n

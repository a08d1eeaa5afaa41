"""The FP32 and FP64 GEMV and the FP32 tiles over blocks of right-hand sides: every block size, row remainders of a warp's 1, 2 or 4 rows,
k remainders of its unrolled steps, and the widths on both sides of its limits.

A lane adds every 32nd term in order and the lanes are summed by a fixed tree, whatever the block and the rows a warp
takes, so a column of a block is the product of that column alone, bit for bit.  Accuracy: a sum of m = ceil(n / 32)
complex terms a lane (2 m roundings of FMAs a component) and 5 more in the tree is off by at most
(2 m + 5) eps of the sum of |z||x| (first order; twice that covers the rest)."""
import numpy as np
import pytest

from emfa_gb300 import api
from test_gpu_slice import test_fp32_slice_product_against_exact_sums as slice_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 31, 33, 127, 129, 480, 1301, 3007])
@pytest.mark.parametrize("r", [1, 2, 3, 5, 7, 8, 9, 11, 16, 17, 32])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_gemv_block_equals_its_columns(ctx, n, r, precision):
    import torch
    if precision == "f64" and n > 480:
        pytest.skip("one row a warp at every size")
    ct = torch.complex64 if precision == "f32" else torch.complex128
    mode = "auto" if precision == "f32" else "f64"
    g = torch.Generator(device="cuda").manual_seed(n * 100 + r)
    z = torch.randn(n, n, dtype=ct, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=ct, device="cuda", generator=g)
    y = api.matvec(ctx, z, x, mode)
    for c in () if precision == "f32" and (r > 16 or r > 8 and n >= 2500) else sorted({0, 1, r // 2, r - 2, r - 1} & set(range(r))):
        assert torch.equal(y[c], api.matvec(ctx, z, x[c:c + 1].contiguous(), mode)[0])
    zd, xd = z.to(torch.complex128), x.to(torch.complex128)
    eps = np.finfo(np.float32 if precision == "f32" else np.float64).eps
    # FP64 references of an FP64 product carry an error of the same form
    bound = 2 * (2 * ((n + 31) // 32) + 5) * eps * (xd.abs() @ zd.abs().T) + (0 if precision == "f32" else 4 * n * eps * (xd.abs() @ zd.abs().T))
    assert bool(((y - xd @ zd.T).abs() <= 2 * bound).all())


def test_gemv_keeps_infinities_and_nans(ctx):
    """A short last block repeats its last column and a short last warp its last row: neither may leak."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    z = torch.randn(1301, 1301, dtype=torch.complex64, device="cuda", generator=g)
    x = torch.randn(15, 1301, dtype=torch.complex64, device="cuda", generator=g)
    clean = api.matvec(ctx, z, x)
    z[1300, 7] = float("inf")
    x[14, 1300] = float("nan")
    y = api.matvec(ctx, z, x)
    assert torch.equal(y[:14, :1300], clean[:14, :1300])
    assert not bool(torch.isfinite(torch.view_as_real(y[14])).any())
    assert not bool(torch.isfinite(torch.view_as_real(y[:, 1300])).all(-1).any())


@pytest.mark.parametrize("n,r", [(128, 33), (257, 34), (271, 33), (384, 40), (640, 330), (701, 299), (1030, 200)])
@pytest.mark.parametrize("kind", ["normal", "graded", "extreme"])
def test_blocks_above_the_gemv(ctx, n, r, kind):
    slice_check(ctx, n, r, kind)


@pytest.mark.parametrize("n", [17, 63, 65, 129, 500, 1111, 2501, 4003])
@pytest.mark.parametrize("r", [5, 8, 9, 16, 17, 24, 25, 33, 40, 41, 63, 80, 81, 97])
def test_tiles(ctx, n, r):
    """Clustered tiles: every count of right-hand sides a thread, one to eight parts of k, ragged rows, k and columns.
    A part is one chain of at most 2 n roundings a component in its longest form, and eight parts are added."""
    import torch
    if r <= 8 and n < 4000 or r <= 16 and n < 2500:
        pytest.skip("the GEMV's")
    g = torch.Generator(device="cuda").manual_seed(n * 100 + r)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=torch.complex64, device="cuda", generator=g)
    y = api.matvec(ctx, z, x)
    zd, xd = z.to(torch.complex128), x.to(torch.complex128)
    err = (y - xd @ zd.T).abs()
    bound = (2 * n + 8) * np.finfo(np.float32).eps * (xd.abs() @ zd.abs().T)
    assert bool((err <= bound).all())
    # and no worse than the 64 x 64 tiles of an explicit FP32 product by more than their noise
    other = (api.matvec(ctx, z, x, "f32") - xd @ zd.T).abs()
    assert float(err.norm()) <= 1.2 * float(other.norm()) or r <= 16


def test_tiles_keep_infinities_and_nans(ctx):
    import torch
    g = torch.Generator(device="cuda").manual_seed(4)
    z = torch.randn(1301, 1301, dtype=torch.complex64, device="cuda", generator=g)
    x = torch.randn(37, 1301, dtype=torch.complex64, device="cuda", generator=g)
    clean = api.matvec(ctx, z, x)
    z[1300, 7] = float("inf")
    x[36, 1300] = float("nan")
    y = api.matvec(ctx, z, x)
    assert torch.equal(y[:36, :1300], clean[:36, :1300])
    assert not bool(torch.isfinite(torch.view_as_real(y[36])).any())
    assert not bool(torch.isfinite(torch.view_as_real(y[:, 1300])).all(-1).any())

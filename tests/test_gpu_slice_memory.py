"""What digit planes hold between calls, and the blocks of rows that keep it bounded: sizes whose planes take more than
the 1 GiB that stays (FP64 from n = 5462 on, in blocks of 4864 rows at 6000; FP32 from 7328 on, 7040 rows at 7600).

Against the explicit mode's sums: a difference is at most the two bounds of sum |z||x|, of (2 ceil(n / 32) + 5) 2^-52
each in FP64 and (2 n + 8) 2^-23 each in FP32, and the operands' spread sends part of the results to their own sums."""
import pytest

from emfa_gb300 import api

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def _operands(n, r, dtype, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn(n, n, dtype=dtype, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=dtype, device="cuda", generator=g)
    d = 10 ** (torch.rand(n, device="cuda", generator=g) - 0.5)
    z *= d  # columns against x: some results below the digits' floor
    x /= d
    z[::97] *= 1e-3
    z[::89, 5] *= 1e6
    return z, x


@pytest.mark.parametrize("precision,n,r", [("f64", 6000, 9), ("f32", 7600, 104)])
def test_blocks_of_rows(emfa_lib, precision, n, r):
    import torch
    c = api.Context(0)
    dt = torch.complex128 if precision == "f64" else torch.complex64
    z, x = _operands(n, r, dt, n)
    before, launches = c.memory()[0], c.launches()
    y = api.matvec(c, z, x)
    assert c.launches() - launches >= 10  # two blocks of split, digits, product, magnitudes, combination
    assert c.memory()[0] - before <= GIB + GIB // 4
    other = api.matvec(c, z, x, precision)
    s = x.abs().to(torch.float64) @ z.abs().to(torch.float64).T
    bound = 2 * (2 * ((n + 31) // 32) + 5) * 2.0 ** -52 if precision == "f64" else 2 * (2 * n + 8) * 2.0 ** -23
    assert bool(((y - other).abs() <= 2 * bound * s).all())
    assert torch.equal(api.matvec(c, z, x), y)
    c.close()


def test_a_solve_gives_large_planes_back(emfa_lib):
    import torch
    c = api.Context(0)
    n, r = 6000, 4
    g = torch.Generator(device="cuda").manual_seed(3)
    z = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)
    z.diagonal().add_(400.0)
    b = torch.randn(r, n, dtype=torch.complex128, device="cuda", generator=g)
    before = c.memory()[0]
    x, info = api.solve(c, z, b, api.solver_params("gmres", tol=1e-9))
    assert info.converged == r
    assert float((x @ z.T - b).norm() / b.norm()) < 2e-9
    # the basis of 30 vectors, and less than a quarter of a GiB of scratch
    assert c.memory()[0] - before <= 31 * 16 * n * r + GIB // 4
    y, _ = api.solve(c, z, b, api.solver_params("gmres", tol=1e-9))
    assert torch.equal(x, y)
    c.close()

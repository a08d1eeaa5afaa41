"""Steps and tiles of the Krylov solves.  The split-FP16 product at the widths where its column tile changes (16, 64 and 144 real columns), the rows where a tile
ends, and K shorter and longer than the stages loaded ahead; and GMRES steps whose basis fits the shared memory of a CTA
that has an SM to itself, or of one of two.

Each right-hand side is scaled by itself and its sums run over k in one order, so a column of a block is the product of that
column alone, bit for bit.  Refined GMRES has to reach its tolerance on the true residual whatever the layout of a step."""
import numpy as np
import pytest

from emfa_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 128, 129, 257, 385, 900])
@pytest.mark.parametrize("r", [1, 7, 8, 9, 31, 32, 33, 73])
def test_block_equals_its_columns(ctx, n, r):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + 1000 * r)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=torch.complex64, device="cuda", generator=g)
    y = api.matvec(ctx, z, x, "f16x")
    for c in sorted({0, r // 2, r - 1}):
        assert torch.equal(y[c], api.matvec(ctx, z, x[c:c + 1].contiguous(), "f16x")[0])


@pytest.mark.parametrize("n", [33, 129, 300, 1000])
@pytest.mark.parametrize("r", [1, 8, 9, 32, 33, 56, 57, 72, 73, 150])
def test_residual_block_equals_its_columns(ctx, n, r):
    """The refinement residual at the widths of its column tiles (16, 64, 112 and 144)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + 1000 * r)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    b = torch.randn(r, n, dtype=torch.complex64, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=torch.complex128, device="cuda", generator=g)
    y = api.residual(ctx, z, x, b, "f16x")
    for c in sorted({0, r // 2, r - 1}):
        assert torch.equal(y[c], api.residual(ctx, z, x[c:c + 1].contiguous(), b[c:c + 1].contiguous(), "f16x")[0])
    # two 11-bit halves a factor: 2^-21 of |z||x| summed, the FP32 rounding of B - Z X, the dropped low-low products
    bound = 2.0 ** -19 * (x.abs() @ z.abs().to(torch.float64).T) + 2.0 ** -22 * b.abs()
    assert bool(((y - (b - x @ z.to(torch.complex128).T)).abs() <= bound).all())


@pytest.mark.parametrize("n,r", [(31, 1), (512, 1), (513, 2), (1024, 160), (1025, 1), (2500, 40), (4100, 30), (8200, 2)])
@pytest.mark.parametrize("restart", [2, 32])
def test_gmres_step_layouts(ctx, n, r, restart):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + r)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    z.diagonal().add_(2.5 * n ** 0.5)
    b = torch.randn(r, n, dtype=torch.complex64, device="cuda", generator=g)
    x, info = api.solve(ctx, z, b, api.solver_params("gmres", restart=restart, tol=1e-6, orth="cgs1_fused"))
    assert info.converged == r
    res = b.to(torch.complex128) - x @ z.to(torch.complex128).T
    # two roundings of the FP64 residual apart from the solver's own
    assert float((res.norm(dim=1) / b.norm(dim=1)).max()) <= 1e-6 * (1 + 1e-6)


@pytest.mark.parametrize("n,r", [(300, 700), (1024, 640), (1500, 320), (1501, 320), (4097, 130), (7680, 80), (8192, 77),
                                 (8193, 70)])
def test_one_launch_step_equals_the_passes(ctx, n, r):
    """A step on the FP16 basis by one cluster a right-hand side (up to eight chunks of 1024) and by the three passes: the
    same sums in the same order, so the same bits; a zero right-hand side among them is done at once.  Where the blocks are
    few (at most four CTAs an SM) the automatic choice is the FP32-basis step: the same solution to the tolerance."""
    import torch
    few = r * min(8, -(-n // 1024)) <= 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(n + r)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    z.diagonal().add_(2.5 * n ** 0.5)
    b = torch.randn(r, n, dtype=torch.complex64, device="cuda", generator=g)
    b[r // 2] = 0
    for restart in (3, 30):
        x, info = api.solve(ctx, z, b, api.solver_params("gmres", restart=restart, tol=1e-6))
        y, other = api.solve(ctx, z, b, api.solver_params("gmres", restart=restart, tol=1e-6, orth="cgs1_split"))
        assert info.converged == r and other.converged == r
        if few:
            assert float((x - y).norm() / y.norm()) < 1e-5
            continue
        assert (info.iterations, info.cycles) == (other.iterations, other.cycles)
        assert torch.equal(x, y)


@pytest.mark.parametrize("n,r", [(1, 1), (31, 1), (33, 3), (257, 2), (480, 1), (480, 91), (1025, 7), (2049, 48), (4097, 3),
                                 (8192, 1), (8193, 1)])
@pytest.mark.parametrize("restart", [1, 7, 31, 32])
def test_fp64_step_agrees_with_the_passes(ctx, n, r, restart):
    """The FP64 step in one launch (restarts up to 31, N up to 8192) against the separate passes: FP64 sums in another
    order, so both meet the target and agree to its rounding (condition below 10)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + r + restart)
    z = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)
    z.diagonal().add_(4 * n ** 0.5)
    b = torch.randn(r, n, dtype=torch.complex128, device="cuda", generator=g)
    if r > 2:
        b[1] = 0
    sols = []
    for orth in ("auto", "cgs2"):
        x, info = api.solve(ctx, z, b, api.solver_params("gmres", restart=restart, tol=1e-11, orth=orth, max_iter=3000))
        assert info.converged == r
        res = (b - x @ z.T).norm(dim=1) / b.norm(dim=1).clamp_min(1e-300)
        assert float(res.max()) <= 2e-11
        sols.append((x, info.iterations, info.cycles))
    # a step at the target's very edge may fall either way
    assert abs(sols[0][1] - sols[1][1]) <= max(1, restart) and abs(sols[0][2] - sols[1][2]) <= 1
    assert float((sols[0][0] - sols[1][0]).norm() / sols[1][0].norm()) <= 20 * 2e-11

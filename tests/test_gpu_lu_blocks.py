"""LU factor at the edges of its block schedule: one to six diagonal blocks (a pair of blocks, a pair and a single one, a
ragged last block of 1 to 63 rows), the sizes where the trailing update changes from 64- to 256-row tiles and where the
tiles of a block's columns and rows are more than the SMs, and pivots that tie.

The refined solution has to meet the tolerance in as few passes as a sound FP32 factor needs: a pass gains the factor's
relative accuracy, about cond(Z) n eps < 10 x 5000 x 6e-8 = 3e-3 at the worst, so 1e-6 takes at most three."""
import numpy as np
import pytest

from test_lu import _check, _random, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 16, 17, 31, 33, 79, 80, 127, 128, 129, 191, 192, 193, 255, 257, 319, 321, 384])
def test_lu_block_edges(ctx, n):
    Z, B = _random(n, 3, n + 17)
    X, info = _solve(ctx, Z, B)
    assert info.converged == 3 and info.iterations <= 3
    _check(Z, B, X)


@pytest.mark.parametrize("n", [900, 967, 1031, 4931])
def test_lu_tile_rules(ctx, n):
    import torch
    from emfa_gb300 import api
    g = torch.Generator(device="cuda").manual_seed(n)
    z = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=g)
    z.diagonal().add_(3 * n ** 0.5)
    b = torch.randn(9, n, dtype=torch.complex64, device="cuda", generator=g)
    x, info = api.solve(ctx, z, b, api.solver_params("lu", tol=1e-6))
    assert info.converged == 9 and info.iterations <= 3
    r = b.to(torch.complex128) - x @ z.to(torch.complex128).T
    assert float((r.norm(dim=1) / b.norm(dim=1)).max()) < 2e-6


def test_lu_tied_pivots_take_the_lowest_row(ctx):
    """Entries 0 and 1 or powers of i make exact ties in every column; a shuffle of the rows within a block that keeps the
    lowest row on ties solves all the same."""
    n = 64
    rng = np.random.default_rng(5)
    Z = np.eye(n)[rng.permutation(n)] * (1j ** rng.integers(0, 4, n))[:, None] + 0.0
    Z[:, 1:] += Z[:, :1]  # ties of the first column's entry with every other
    B = rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))
    X, info = _solve(ctx, Z, B)
    assert info.converged == 2 and info.iterations <= 1
    res = np.abs(B.astype(np.complex64).astype(np.complex128) - X @ Z.T).max()
    assert res < 64 * 6e-8 * np.abs(X).sum(axis=1).max()

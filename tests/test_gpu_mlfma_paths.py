"""The MLFMA mat-vec where its kernels change: the finest level in one kernel or, for boxes too large for its shared memory,
in two; one or several pattern levels; right-hand sides a pass of one, of up to eight, and a chunk and a rest.

The far and near parts are sums of the same FP32 products whatever the pass, so a column of a block is the column alone to
FP32 rounding of its own sums (a few hundred terms: 1e-5 of the column's norm is far above it), and near + far is the whole.
Against the CFIE entries themselves the multilevel approximation is held in test_gpu_mlfma_extent.py."""
import pytest

from emfa_gb300 import api
from emfa_gb300 import mesh as M

pytestmark = pytest.mark.gpu
FREQ = 3e8


@pytest.fixture(scope="module")
def target(ctx):
    return api.Geometry(ctx, M.icosphere(4, 1.6))


@pytest.mark.parametrize("threshold", [0.15, 0.25, 0.5, 0.9])
def test_parts_and_blocks(ctx, target, threshold):
    import torch
    geo, n = target, target.n
    op = api.Mlfma(geo, api.mlfma_params(FREQ, 0.5, threshold))
    g = torch.Generator(device="cuda").manual_seed(int(100 * threshold))
    x = torch.randn(9, n, dtype=torch.complex64, device="cuda", generator=g)
    single = [op.apply(x[r:r + 1].contiguous())[0] for r in range(9)]
    for r in (1, 2, 3, 5, 8, 9):
        y = op.apply(x[:r].contiguous())
        for c in range(r):
            assert float((y[c] - single[c]).norm() / single[c].norm()) < 1e-5
    near, far = op.apply_part(x[0], 1), op.apply_part(x[0], 2)
    assert float((near + far - single[0]).norm() / single[0].norm()) < 1e-5
    op.close()


def test_operators_of_one_context_in_turn(ctx, target):
    """Sets of tables and pattern buffers of two operators, grown by a larger block, released in the other order."""
    import torch
    geo = target
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(8, geo.n, dtype=torch.complex64, device="cuda", generator=g)
    a = api.Mlfma(geo, api.mlfma_params(FREQ, 0.5, 0.25))
    first = a.apply(x[:1].contiguous())
    b = api.Mlfma(geo, api.mlfma_params(FREQ, 0.5, 0.5))
    other = b.apply(x)
    assert torch.equal(a.apply(x)[:1], a.apply(x)[:1])
    a.close()
    assert torch.equal(b.apply(x), other)
    c = api.Mlfma(geo, api.mlfma_params(FREQ, 0.5, 0.25))
    assert torch.equal(c.apply(x[:1].contiguous()), first)
    b.close()
    c.close()

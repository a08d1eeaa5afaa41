"""A digit-plane product whose pipeline gives up: its result is NaN, the next call that looks says EMFA_ERR_TIMEOUT once,
and the products after it are right.  The wait is the pipelines' own, on a barrier that nothing arrives on, cut at 1 ms."""
import numpy as np
import pytest

from emfa_gb300 import _lib as L
from emfa_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture()
def product():
    import torch
    c = api.Context(0)
    g = torch.Generator(device="cuda").manual_seed(1)
    z = torch.randn(640, 640, dtype=torch.complex128, device="cuda", generator=g)
    x = torch.randn(40, 640, dtype=torch.complex128, device="cuda", generator=g)
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    want = api.matvec(c, z, x)

    def run():
        return L.lib().emfa_matvec(c.h, L.EMFA_F64, 0, api._ptr(z), 640, api._ptr(x), 40, api._ptr(y), None)

    yield c, run, y, want
    c.close()


def test_synchronize_reports_it(product):
    import torch
    c, run, y, want = product
    assert L.lib().emfa_diag_product_timeout(c.h) == 0
    assert run() == 0
    assert L.lib().emfa_ctx_synchronize(c.h) == 7
    assert b"digit-plane" in L.lib().emfa_last_error(c.h) and b"42" in L.lib().emfa_last_error(c.h)
    assert bool(torch.isnan(torch.view_as_real(y)).all())
    assert run() == 0 and L.lib().emfa_ctx_synchronize(c.h) == 0
    assert torch.equal(y, want)


def test_the_next_product_reports_it(product):
    import torch
    c, run, y, want = product
    assert L.lib().emfa_diag_product_timeout(c.h) == 0
    assert run() == 0
    torch.cuda.synchronize()
    assert run() == 7
    assert run() == 0 and L.lib().emfa_ctx_synchronize(c.h) == 0
    assert torch.equal(y, want)


def test_a_solve_has_its_own_word(product):
    import torch
    c, run, y, want = product
    assert L.lib().emfa_diag_product_timeout(c.h) == 0
    g = torch.Generator(device="cuda").manual_seed(2)
    z = torch.randn(640, 640, dtype=torch.complex128, device="cuda", generator=g) + 60 * torch.eye(640, device="cuda")
    b = torch.randn(40, 640, dtype=torch.complex128, device="cuda", generator=g)
    x, info = api.solve(c, z, b, api.solver_params("gmres", tol=1e-8))
    assert info.converged == 40
    assert float(((x @ z.T - b).norm() / b.norm())) < 1e-7
    assert run() == 0 and L.lib().emfa_ctx_synchronize(c.h) == 7
    assert np.isnan(y.cpu().numpy()).all()

"""FP64 residuals of blocks take the planes of single products: a residual after a product of its size holds no more device
memory, it leaves a solve's planes alone, and two threads' residuals on one context do not share one another's."""
import threading

import pytest

from emfa_gb300 import api

pytestmark = pytest.mark.gpu


def _data(seed, n=700, r=24):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    z, x, b = (torch.randn(*s, dtype=torch.complex128, device="cuda", generator=g) for s in ((n, n), (r, n), (r, n)))
    return z, x, b


def test_a_residual_reuses_a_products_memory(emfa_lib):
    import torch
    c = api.Context(0)
    z, x, b = _data(1)
    y = api.matvec(c, z, x)
    held = c.memory()[0]
    r = api.residual(c, z, x, b)
    assert torch.equal(r, b - y)
    assert c.memory()[0] == held
    c.close()


def test_residuals_of_two_threads(emfa_lib):
    """After one call each, so that no workspace grows while the other thread's product runs."""
    import torch
    c = api.Context(0)
    data = [_data(s) for s in (2, 3)]
    want = [api.residual(c, *d) for d in data]
    bad = []

    def work(i):
        for _ in range(40):
            if not torch.equal(api.residual(c, *data[i]), want[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
    c.close()

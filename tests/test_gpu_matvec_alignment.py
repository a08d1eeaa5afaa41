"""emfa_matvec on operands at the alignment of their scalars: complex64 at an odd float, complex128 at an odd double, at
widths that take the GEMV, the tiles and the digit planes when aligned.  The results are the explicit mode's of the aligned
operands, to the two sums' bounds ((2 n + 8) eps of sum |z||x| each)."""
import pytest

from emfa_gb300 import _lib as L
from emfa_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["z", "x", "y", "all"])
@pytest.mark.parametrize("precision,n,r", [("f32", 640, 3), ("f32", 300, 20), ("f32", 641, 40), ("f32", 1201, 520), ("f64", 640, 3),
                                           ("f64", 513, 41)])
def test_operands_at_odd_scalars(ctx, precision, n, r, which):
    import torch
    f, c = (torch.float32, torch.complex64) if precision == "f32" else (torch.float64, torch.complex128)
    g = torch.Generator(device="cuda").manual_seed(n + r)
    z = torch.randn(n, n, dtype=c, device="cuda", generator=g)
    x = torch.randn(r, n, dtype=c, device="cuda", generator=g)

    def place(a, odd):
        buf = torch.full((2 * a.numel() + 2,), float("nan"), dtype=f, device="cuda")
        at = buf[1:1 + 2 * a.numel()] if odd else buf[:2 * a.numel()]
        at.copy_(torch.view_as_real(a).reshape(-1))
        return buf, at

    bufs = [place(a, which in (k, "all")) for k, a in (("z", z), ("x", x), ("y", torch.zeros_like(x)))]
    torch.cuda.synchronize()
    prec = L.EMFA_F32 if precision == "f32" else L.EMFA_F64
    ctx.check(L.lib().emfa_matvec(ctx.h, prec, 0, bufs[0][1].data_ptr(), n, bufs[1][1].data_ptr(), r, bufs[2][1].data_ptr(),
                                  None))
    ctx.synchronize()
    y = torch.view_as_complex(bufs[2][1].reshape(r, n, 2).clone())
    want = api.matvec(ctx, z, x, precision)
    s = x.abs().to(torch.float64) @ z.abs().to(torch.float64).T
    eps = torch.finfo(f).eps
    assert bool(((y - want).abs() <= 2 * 2 * (2 * n + 8) * eps * s).all())
    assert torch.isnan(bufs[2][0][0 if which in ("y", "all") else -1]) and torch.isnan(bufs[2][0][-1])

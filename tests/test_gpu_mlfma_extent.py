"""MLFMA of long targets: strips whose top levels have more than 512 multipoles (a phi row of the interpolation is then a
CTA of its own) and, from about 180 wavelengths, rows too long for the shifted samples beside the theta pass.

The far block of the functions at one end and of those at three places along the strip, translated at the two top levels,
against the CFIE entries themselves.  The truncation and the three-point interpolation leave strips of 20 to 170
wavelengths, all of shorter levels, with a correlation of 0.989 and more and 0.79 to 1.01 of the size there (twelve
extents); 0.9 and 0.5 to 1.5 leave that some room.  A level that is missing gives zero, a wrong row, shift or list a
correlation of a few percent (some 7,000 entries)."""
import numpy as np
import pytest

from emfa_gb300 import api
from emfa_gb300 import mesh as M

pytestmark = pytest.mark.gpu
FREQ = 3e8
LAM = 299792458.0 / FREQ


def _strip(nx, ny, cell):
    xs, ys = np.arange(nx + 1) * cell, np.arange(ny + 1) * cell
    v = np.stack([np.repeat(xs, ny + 1), np.tile(ys, nx + 1), np.zeros((nx + 1) * (ny + 1))], 1)
    i = (np.arange(nx)[:, None] * (ny + 1) + np.arange(ny)[None]).reshape(-1)
    t = np.concatenate([np.stack([i, i + ny + 1, i + ny + 2], 1), np.stack([i, i + ny + 2, i + 1], 1)])
    return M.TriMesh(v, np.ascontiguousarray(t, dtype=np.int32), name="strip")


@pytest.mark.parametrize("extent", [120, 175, 200])
def test_far_blocks_along_a_strip(emfa_lib, extent):
    import torch
    c = api.Context(0)
    m = _strip(10 * extent, 5, 0.1 * LAM)
    geo = api.Geometry(c, m)
    mp = api.mlfma_params(FREQ, 0.5, 0.25)
    op = api.Mlfma(geo, mp)
    place = np.argsort(api.mlfma_plan(m, geo.rwg, mp)[3])  # in box order
    at = (m.verts[geo.rwg[:, 0], 0] + m.verts[geo.rwg[:, 1], 0]) / 2 / LAM
    src = np.nonzero(at < 0.45)[0]
    x = torch.zeros(len(src), geo.n, dtype=torch.complex64, device="cuda")
    x[torch.arange(len(src)), torch.from_numpy(place[src]).cuda()] = 1
    y = op.apply(x).cpu().numpy()[:, place]
    for part in (0.45, 0.8, 0.9):
        rec = np.nonzero(abs(at - (part * extent - 0.6)) < 0.5)[0]
        both = api.Geometry(c, m, np.ascontiguousarray(geo.rwg[np.concatenate([src, rec])]))
        z = api.fill_z(both, api.fill_params("cfie", "f64", FREQ, 0.5)).cpu().numpy()[len(src):, :len(src)]
        got = y[:, rec].T
        size = np.linalg.norm(got) / np.linalg.norm(z)
        assert 0.5 < size < 1.5, (part, size)
        assert abs(np.vdot(got, z)) > 0.9 * np.linalg.norm(got) * np.linalg.norm(z), part
        both.close()
    op.close()
    geo.close()
    c.close()

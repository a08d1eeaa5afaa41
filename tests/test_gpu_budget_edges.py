"""Calls at the edge of an HBM budget: what fitted without the patch fill's plan, or without the MLFMA set-up's tables
beside one another, still fits."""
import numpy as np
import pytest

from emfa_gb300 import api
from emfa_gb300 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision,disc", [("efie", "f64", "reference"), ("cfie", "f64", "reference"), ("efie", "f32", "config")])
def test_fill_without_room_for_its_plan(emfa_lib, kind, precision, disc):
    m = M.icosphere(2, 0.5)
    fp = api.fill_params(kind, precision, 3e8, 0.5, edm_mode=2, discretisation=disc)
    free = api.Context(0)
    geo = api.Geometry(free, m)
    want = api.fill_z(geo, fp).cpu().numpy()
    held = free.memory()[0]
    geo.close()
    free.close()
    tight = api.Context(0, held - 256)
    geo = api.Geometry(tight, m)
    z = api.fill_z(geo, fp).cpu().numpy()  # the last allocation is the plan's
    # the two kernels' bars against one another (test_gpu_fill_patch_tables.py)
    if precision == "f64":
        assert (abs(z - want) / np.maximum(abs(want), 1e-3 * abs(want).max())).max() < 1e-11
    else:
        assert np.linalg.norm(z - want) / np.linalg.norm(want) < 2e-5
    geo.close()
    tight.close()


def test_mlfma_setup_peak(emfa_lib):
    """Under a budget the set-up needs the operator and, beside it, at most the singular table of 9 FP64 pairs a triangle."""
    m = M.icosphere(4, 1.6)
    c = api.Context(0, 1 << 40)
    geo = api.Geometry(c, m)
    op = api.Mlfma(geo, api.mlfma_params(3e8, 0.5, 0.25))
    used, peak, _ = c.memory()
    assert peak - used <= 9 * 16 * len(m.tris)
    need = peak
    op.close()
    geo.close()
    c.close()
    tight = api.Context(0, need)
    geo = api.Geometry(tight, m)
    api.Mlfma(geo, api.mlfma_params(3e8, 0.5, 0.25)).close()
    geo.close()
    tight.close()

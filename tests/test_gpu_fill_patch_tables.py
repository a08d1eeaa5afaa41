"""The 7 x 7-point patch fill where its tables differ from a thread per entry: meshes whose edges join more than two
triangles, and entries that the tables give alone.

The fill of a thread per entry is taken by any RWG table with a function whose free vertex is no corner of its triangle: one
such row at the end, and the other rows and columns are the same matrix from the other kernel.  Both are pinned to the oracle
on closed surfaces (test_gpu_dense.py); here they are held against each other."""
import numpy as np
import pytest

from emfa_gb300 import api
from emfa_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _finned_sphere():
    """A sphere with a fin on every edge: three triangles an edge, six neighbours a triangle; the RWGs are the three pairs."""
    s = M.icosphere(1, 0.5)
    verts, tris = [v for v in s.verts], [list(t) for t in s.tris]
    edges = {}
    for t, tri in enumerate(s.tris.tolist()):
        for j in range(3):
            edges.setdefault(tuple(sorted((tri[j], tri[(j + 1) % 3]))), []).append((t, tri[(j + 2) % 3]))
    rows = []
    for (a, b), ((t0, v0), (t1, v1)) in edges.items():
        tip = len(verts)
        verts.append(1.35 * (s.verts[a] + s.verts[b]) / 2)
        fin = len(tris)
        tris.append([a, b, tip])
        rows += [[a, b, v0, v1, t0, t1], [a, b, v0, tip, t0, fin], [a, b, tip, v1, fin, t1]]
    return M.TriMesh(np.array(verts), np.array(tris, dtype=np.int32), name="fins"), np.array(rows, dtype=np.int32)


def _both(ctx, m, rows, precision):
    """The matrix by patches and by a thread per entry."""
    free = next(v for v in range(len(m.verts)) if v not in m.tris[rows[0][4]])
    odd = np.concatenate([rows, [[*rows[0][:2], free, *rows[0][3:]]]]).astype(np.int32)
    fp = api.fill_params("efie", precision, 3e8, 1.0, edm_mode=2, discretisation="config")
    out = []
    for table in (rows, odd):
        geo = api.Geometry(ctx, m, np.ascontiguousarray(table))
        out.append(api.fill_z(geo, fp).cpu().numpy()[:len(rows), :len(rows)])
        geo.close()
    return out


@pytest.mark.parametrize("precision,tol", [("f64", 1e-11), ("f32", 2e-5)])
def test_edges_of_three_triangles(ctx, precision, tol):
    """The oracle's bars for the two kernels: entries of 1e-3 of the largest and more, FP64; the whole matrix, FP32."""
    m, rows = _finned_sphere()
    assert rows.shape[0] > 48  # several patches, so that entries are mirrored
    a, b = _both(ctx, m, rows, precision)
    if precision == "f64":
        assert (abs(a - b) / np.maximum(abs(b), 1e-3 * abs(b).max())).max() < tol
    else:
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < tol


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("surface", ["sphere", "fins"])
def test_entries_of_tables_alone(ctx, precision, surface):
    """A diagonal entry has no regular pair: its FP64 table values are summed in FP64 and rounded once, bit for bit the
    other kernel's sum (same values, same order, one product after)."""
    if surface == "fins":
        m, rows = _finned_sphere()
        listed = {}  # the neighbours a triangle lists: its first three
        for r in rows:
            for t, o in ((r[4], r[5]), (r[5], r[4])):
                if len(listed.setdefault(t, [])) < 3 and o not in listed[t]:
                    listed[t].append(o)
        alone = [u for u, r in enumerate(rows) if r[5] in listed[r[4]] and r[4] in listed[r[5]]]
    else:
        m = M.icosphere(2, 0.5)
        rows = api.build_rwg(m.tris)
        alone = range(len(rows))
    a, b = _both(ctx, m, rows, precision)
    assert len(alone) > 100 and np.array_equal(np.diag(a)[alone], np.diag(b)[alone])

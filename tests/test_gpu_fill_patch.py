"""The patch fills (FP64 EFIE/CFIE and the 7 x 7-point EFIE) at the sizes where patches can go wrong: fewer RWGs than
a patch, one more than a patch, ragged and open meshes, far pairs under each mode, and RWG tables in any order."""
import numpy as np
import pytest

from emfa_gb300 import api, mesh

pytestmark = pytest.mark.gpu


def _mesh(name):
    if name == "tetra":  # 6 RWGs: less than a patch
        v = np.array([[0, 0, 0], [0.1, 0, 0], [0, 0.1, 0], [0, 0, 0.1]], dtype=np.float64)
        return mesh.TriMesh(v, np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], dtype=np.int32))
    if name == "strip25":  # an open strip with 25 interior edges: a patch and one RWG
        v = np.array([(0.05 * i, 0.06 * j, 0.01 * (i % 3)) for j in range(2) for i in range(14)])
        t = [tri for i in range(13) for tri in ([i, i + 1, i + 15], [i, i + 15, i + 14])]
        return mesh.TriMesh(v, np.array(t, dtype=np.int32))
    if name == "cube":
        return mesh.cube(3, 0.3)
    if name == "open":
        m = mesh.ellipsoid(3, (0.3, 0.25, 0.2))
        return mesh.TriMesh(m.verts, np.ascontiguousarray(m.tris[5:], dtype=np.int32))
    raise ValueError(name)


def _oracle(O, m, rwg, kind, disc, freq, edm, alpha=0.5):
    g = O.Geometry(m.verts, m.tris, rwg, 64)
    k = O.wavenumber(freq, 64)
    if kind == "cfie":
        return O.fill_z_cfie(g, k, alpha)
    if disc == "config":
        return O.fill_z_efie_cfg(g, k)
    return O.fill_z_efie(g, k, 3 * 299792458.0 / freq, edm_mode=edm)


# FP64: both sides sum the same few hundred terms with 2^-53 roundings, off the oracle's libm phases by a few ulp of
# kR < 100: 1e-12 of the largest entry.  FP32 7 x 7: the bar of the configuration fill, 2e-5 normwise.
@pytest.mark.parametrize("name", ["tetra", "strip25", "cube", "open"])
@pytest.mark.parametrize("kind,disc,precision", [("efie", "reference", "f64"), ("cfie", "reference", "f64"),
                                                 ("efie", "config", "f64"), ("efie", "config", "f32")])
def test_patch_fill_matches_oracle(ctx, oracle_mod, name, kind, disc, precision):
    m = _mesh(name)
    rwg = api.build_rwg(m.tris)
    geom = api.Geometry(ctx, m, rwg)
    fp = api.fill_params(kind, precision, 3e8, 0.5, edm_mode=2, discretisation=disc)
    z = api.fill_z(geom, fp).cpu().numpy()
    ref = _oracle(oracle_mod, m, rwg, kind, disc, 3e8, 2)
    if precision == "f64":
        assert np.abs(z - ref).max() <= 1e-12 * np.abs(ref).max()
    else:
        assert np.linalg.norm(z - ref) <= 2e-5 * np.linalg.norm(ref)


# cube of side 1 m at 1.5 GHz: most pairs are beyond 3 wavelengths (0.6 m), some patch pairs wholly
@pytest.mark.parametrize("edm", [0, 1, 2])
def test_patch_fill_far_modes(ctx, oracle_mod, edm):
    m = mesh.cube(4, 1.0)
    rwg = api.build_rwg(m.tris)
    geom = api.Geometry(ctx, m, rwg)
    z = api.fill_z(geom, api.fill_params("efie", "f64", 1.5e9, edm_mode=edm)).cpu().numpy()
    ref = _oracle(oracle_mod, m, rwg, "efie", "reference", 1.5e9, edm)
    if edm == 0:
        assert ((z == 0) == (ref == 0)).all() and (ref == 0).any()
    assert np.abs(z - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("kind,disc,precision", [("efie", "reference", "f64"), ("cfie", "reference", "f64"),
                                                 ("efie", "config", "f32")])
def test_patch_fill_of_a_permuted_table(ctx, kind, disc, precision):
    """The patches are chosen by place: a shuffled RWG table gives the shuffled matrix."""
    m = mesh.ellipsoid(3, (0.3, 0.25, 0.2))
    rwg = api.build_rwg(m.tris)
    perm = np.random.default_rng(3).permutation(rwg.shape[0])
    fp = api.fill_params(kind, precision, 3e8, 0.5, edm_mode=2, discretisation=disc)
    a = api.fill_z(api.Geometry(ctx, m, rwg), fp).cpu().numpy()
    b = api.fill_z(api.Geometry(ctx, m, rwg[perm]), fp).cpu().numpy()
    # the same pair values, each entry's four added in its own order of sides: equal
    assert np.array_equal(a[np.ix_(perm, perm)], b) or np.abs(a[np.ix_(perm, perm)] - b).max() <= (
        1e-13 if precision == "f64" else 2e-6) * np.abs(a).max()


@pytest.mark.parametrize("kind,disc,precision", [("efie", "reference", "f64"), ("cfie", "reference", "f64"),
                                                 ("efie", "config", "f64")])
def test_table_with_foreign_free_vertex(ctx, kind, disc, precision):
    """A free vertex that is no corner of its triangle is filled entry by entry; the other rows keep their values."""
    m = mesh.cube(2, 0.3)
    rwg = api.build_rwg(m.tris)
    fp = api.fill_params(kind, precision, 3e8, 0.5, edm_mode=2, discretisation=disc)
    a = api.fill_z(api.Geometry(ctx, m, rwg), fp).cpu().numpy()
    odd = rwg.copy()
    other = [v for v in range(m.n_vert) if v not in m.tris[odd[0, 4]]][0]
    odd[0, 2] = other
    b = api.fill_z(api.Geometry(ctx, m, odd), fp).cpu().numpy()
    assert np.isfinite(b).all()
    assert np.abs(a[1:, 1:] - b[1:, 1:]).max() <= 1e-12 * np.abs(a).max()
    assert np.abs(a[0] - b[0]).max() > 1e-3 * np.abs(a).max()

"""The work this framework is timed on, through its public entry points (emfa_gb300.api).

Sizes are those of the repository's configurations and workloads: dense problems of 480 to 7,680 unknowns
(N = 30 f^2 on a geodesic grid of frequency f, meshed at about ten edges a wavelength; three fewer for a shell with
one triangle left out), sweeps of up to 360 incidences, batches of 8-incidence EFIE problems, and MLFMA operators
of 10,830 to 122,880 unknowns.

A case is a dict with "path", one of

  job          dense_rcs: host mesh in, RCS out (RWG table, upload, fill, excitation, solve, far field)
  batch        serve: independent EFIE problems of uneven sizes, factored and solved on the engine's lanes
  fill         fill_z: the impedance matrix alone
  product      matvec: Y = Z X for a matrix in device memory
  mlfma_apply  Mlfma.apply: the multilevel operator's product
  mlfma_setup  Mlfma(...) and its first product: what a new geometry or frequency costs
"""
import functools
import math

import numpy as np
import torch

from emfa_gb300 import api, mesh, workloads

C0 = 299792458.0
DEV = "cuda:0"


def listed():
    return [
        # one small target, one plane wave, bistatic pattern: the shortest call, where launches and latency count
        dict(name="job_cfie_480x1", path="job", kind="cfie", precision="f32", method="gmres", f=4, n_inc=1),
        # monostatic sweep of a 2-wavelength target over 360 incidences (the dense benchmark job)
        dict(name="job_cfie_7680x360", path="job", kind="cfie", precision="f32", method="gmres", f=16, n_inc=360),
        # the plain FP64 path: a sweep in 1-degree steps over an octant, every stage in FP64
        dict(name="job_cfie_f64_1080x91", path="job", kind="cfie", precision="f64", method="gmres", f=6, n_inc=91),
        # a batch of uneven EFIE problems of 8 incidences each, LU with refinement on the engine's lanes
        dict(name="batch_efie_6", path="batch", count=6, f_lo=5, f_hi=11, n_inc=8),
        # impedance matrix of a 5,070-unknown target in the mixed path's precision
        dict(name="fill_cfie_f32_5070", path="fill", kind="cfie", precision="f32", disc="reference", f=13, open=False),
        # the FP64 matrix of an open shell (odd N)
        dict(name="fill_efie_f64_2427", path="fill", kind="efie", precision="f64", disc="reference", f=9, open=True),
        # the 7-point rule with adjacent-pair extraction, the accurate discretisation, at its benchmark size
        dict(name="fill_efie_cfg_f32_1920", path="fill", kind="efie", precision="f32", disc="config", f=8, open=False),
        # FP64 product for a block of right-hand sides
        dict(name="product_f64_2430x181", path="product", precision="f64", n=2430, n_rhs=181),
        # mixed-precision product of a ragged size
        dict(name="product_f32_5067x37", path="product", precision="f32", n=5067, n_rhs=37),
        # the multilevel product of the 5-wavelength sphere benchmark, one right-hand side
        dict(name="mlfma_apply_122880x1", path="mlfma_apply", f=64, n_rhs=1),
        # a served request's product: the smallest size that goes to the multilevel operator, 4 incidences
        dict(name="mlfma_apply_10830x4", path="mlfma_apply", f=19, n_rhs=4),
        # a served request's set-up: octree plan, patterns, translation tables, near field, first product
        dict(name="mlfma_setup_43320", path="mlfma_setup", f=38, n_rhs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["job", "job", "batch", "fill", "fill", "fill", "product", "product", "mlfma_apply",
                       "mlfma_apply", "mlfma_setup"])
    if path == "job":
        if rng.random() < 0.4:
            return dict(path=path, kind=rng.choice(["cfie", "efie"]), precision="f64", method="gmres",
                        f=rng.randint(4, 6), n_inc=_log_int(rng, 1, 91))
        if rng.random() < 0.3:
            return dict(path=path, kind="efie", precision="f32", method="lu", f=rng.randint(4, 13),
                        n_inc=_log_int(rng, 1, 16))
        return dict(path=path, kind="cfie", precision="f32", method="gmres", f=rng.randint(4, 16),
                    n_inc=_log_int(rng, 1, 360))
    if path == "batch":
        lo = rng.randint(4, 7)
        return dict(path=path, count=rng.randint(2, 6), f_lo=lo, f_hi=rng.randint(lo + 1, 11), n_inc=8)
    if path == "fill":
        kind = rng.choice(["cfie", "efie"])
        disc = rng.choice(["reference", "config"]) if kind == "efie" else "reference"
        precision = rng.choice(["f32", "f64"])
        f_hi = 13 if precision == "f32" and disc == "reference" else 9 if disc == "reference" else 8 \
            if precision == "f32" else 5
        return dict(path=path, kind=kind, precision=precision, disc=disc, f=rng.randint(4, f_hi),
                    open=rng.random() < 0.5)
    if path == "product":
        precision = rng.choice(["f32", "f64"])
        return dict(path=path, precision=precision, n=_log_int(rng, 480, 5070 if precision == "f32" else 2430),
                    n_rhs=_log_int(rng, 1, 360 if precision == "f32" else 181))
    if path == "mlfma_apply":
        f = _log_int(rng, 19, 64)
        return dict(path=path, f=f, n_rhs=_log_int(rng, 1, 8 if f <= 38 else 2))
    return dict(path=path, f=_log_int(rng, 19, 38), n_rhs=rng.randint(1, 4))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    """A program's context lives as long as the program."""
    return api.Context(0)


@functools.lru_cache(maxsize=8)
def _unit_sphere(f):
    return workloads.geodesic_sphere_fast(f)


def _target(f, rng, open_shell=False):
    """(mesh, frequency): an ellipsoid of seeded semi-axes with about ten edges a wavelength."""
    v, t = _unit_sphere(f)
    semi = np.array([1.0, rng.uniform(0.85, 1.0), rng.uniform(0.7, 1.0)])
    if open_shell:
        t = np.delete(t, int(rng.integers(0, t.shape[0])), axis=0)
    m = mesh.TriMesh(mesh.round6(v * semi), np.ascontiguousarray(t, dtype=np.int32), name="target")
    edge = math.sqrt(4 * math.pi * 4 / (math.sqrt(3) * 20 * f * f)) * float(semi.mean())
    return m, C0 / (10 * edge)


def _incidences(n, rng):
    return np.stack([rng.uniform(0, 180, n), rng.uniform(0, 360, n), np.zeros(n)], 1)


def _job_inputs(case, seed):
    rng = np.random.default_rng(seed)
    m, freq = _target(case["f"], rng)
    ang = _incidences(case["n_inc"], rng)
    if case["n_inc"] == 1:
        return m, freq, ang, api.bistatic_dirs(), False
    return m, freq, ang, api.monostatic_dirs(ang), True


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        # sizes spread evenly over the range, largest last, as a batch of uneven targets is
        f = case["f_lo"] + (case["f_hi"] - case["f_lo"]) * i // max(1, case["count"] - 1)
        m, freq = _target(f, rng)
        ang = _incidences(case["n_inc"], rng)
        out.append((m, freq, ang, api.monostatic_dirs(ang)))
    return out


def _product_inputs(case, seed):
    """A matrix with an impedance matrix's make-up: a free-space kernel between points on a sphere weighted by
    the angle of seeded tangents, and a dominant diagonal; right-hand sides of unit variance."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n, r = case["n"], case["n_rhs"]
    dt = torch.complex128 if case["precision"] == "f64" else torch.complex64
    p = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64), dim=1)
    u = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64), dim=1)
    d = torch.cdist(p, p, compute_mode="donot_use_mm_for_euclid_dist") + 2.0 / math.sqrt(n)
    z = torch.polar((u @ u.T) / d, -math.pi * math.sqrt(n) / 10 * d)
    z.diagonal().add_(2.0 * math.sqrt(n) * (1 + 0.5j))
    x = torch.randn(r, n, generator=g, device=DEV, dtype=dt)
    return z.to(dt), x


def prepare(case, seed):
    path = case["path"]
    if path == "job":
        m, freq, ang, dirs, per_rhs = _job_inputs(case, seed)
        fp = api.fill_params(case["kind"], case["precision"], freq, 0.5, edm_mode=2)
        return dict(path=path, ctx=_context(), mesh=m, fp=fp, ang=ang, dirs=dirs, per_rhs=per_rhs,
                    sp=api.solver_params(case["method"], tol=1e-6 if case["method"] == "gmres" else 1e-5))
    if path == "batch":
        return dict(path=path, reqs=[api.RcsRequest(m, freq, ang, dirs, kind="efie", per_rhs=True)
                                     for m, freq, ang, dirs in _batch_inputs(case, seed)])
    if path == "product":
        z, x = _product_inputs(case, seed)
        return dict(path=path, ctx=_context(), z=z, x=x)
    rng = np.random.default_rng(seed)
    m, freq = _target(case["f"], rng, case.get("open", False))
    geom = api.Geometry(_context(), m)
    if path == "fill":
        fp = api.fill_params(case["kind"], case["precision"], freq, 0.5, edm_mode=2, discretisation=case["disc"])
        return dict(path=path, geom=geom, fp=fp)
    x = rng.standard_normal((case["n_rhs"], geom.n, 2)).astype(np.float32)
    x = torch.view_as_complex(torch.from_numpy(x).to(DEV))
    mp = api.mlfma_params(freq, 0.5, 0.25)
    if path == "mlfma_apply":
        return dict(path=path, op=api.Mlfma(geom, mp), x=x)
    return dict(path=path, geom=geom, mp=mp, x=x)


def run(state):
    path = state["path"]
    if path == "job":
        return api.dense_rcs(state["ctx"], state["mesh"], state["fp"], state["ang"], state["sp"], state["dirs"],
                             state["per_rhs"])[0]
    if path == "batch":
        api.serve(state["reqs"])
        return [r.rcs for r in state["reqs"]]
    if path == "fill":
        return api.fill_z(state["geom"], state["fp"])
    if path == "product":
        return api.matvec(state["ctx"], state["z"], state["x"])
    if path == "mlfma_apply":
        return state["op"].apply(state["x"])
    op = api.Mlfma(state["geom"], state["mp"])
    y = op.apply(state["x"])
    op.close()
    return y


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _fill_flops(n, kind, disc):
    # a kernel value and its part in the three edges' sums, for every point pair of every triangle pair
    t = 2 * n / 3
    return t * t * (49 if disc == "config" else 9) * (75 if kind == "cfie" else 40)


def _job_flops(n, n_inc, kind, method):
    # GMRES: at least ten products of the block; LU: factor and solve
    solve = 8 / 3 * n ** 3 + 8 * n * n * n_inc if method == "lu" else 10 * 8 * n * n * n_inc
    return _fill_flops(n, kind, "reference") + solve


def work(case):
    path = case["path"]
    if path == "product":
        b = 16 if case["precision"] == "f64" else 8
        n, r = case["n"], case["n_rhs"]
        return dict(bytes=b * (n * n + 2 * n * r), flops=8 * n * n * r)
    if path == "batch":
        fs = [case["f_lo"] + (case["f_hi"] - case["f_lo"]) * i // max(1, case["count"] - 1)
              for i in range(case["count"])]
        return dict(bytes=sum(16 * 30 * f * f * case["n_inc"] + 60 * 30 * f * f for f in fs),
                    flops=sum(_job_flops(30 * f * f, case["n_inc"], "efie", "lu") for f in fs))
    n = 30 * case["f"] ** 2 - (3 if case.get("open") else 0)
    if path == "job":
        return dict(bytes=60 * n + 8 * case["n_inc"], flops=_job_flops(n, case["n_inc"], case["kind"], case["method"]))
    if path == "fill":
        return dict(bytes=(16 if case["precision"] == "f64" else 8) * n * n,
                    flops=_fill_flops(n, case["kind"], case["disc"]))
    # per unknown: radiation and receive patterns (128 samples, 16 bytes each) and about 100 near entries;
    # per far interaction and right-hand side (about 720 sample products an unknown): 24 flops
    r = case["n_rhs"]
    one = dict(bytes=n * (2 * 128 * 16 + 100 * 8 + 16 * r), flops=n * r * (2 * 128 * 16 + 100 * 8 + 720 * 24))
    if path == "mlfma_setup":  # writes what the product reads; near entries of 4 x 9 point pairs over 9 edges
        one = dict(bytes=2 * one["bytes"], flops=one["flops"] + n * 100 * 4 * 75 + n * 2 * 128 * 150)
    return one


# ---------------------------------------------------------------------------
# the same values in plain FP64 torch
# ---------------------------------------------------------------------------
_Z0 = 120 * math.pi
_W7 = [2 * w for w in (0.112500000000000, 0.062969590272413, 0.062969590272413, 0.062969590272413,
                       0.066197076394253, 0.066197076394253, 0.066197076394253)]
_G7 = [(0.333333333333333, 0.333333333333333), (0.797426985353087, 0.101286507323456),
       (0.101286507323456, 0.797426985353087), (0.101286507323456, 0.101286507323456),
       (0.470142064105115, 0.470142064105115), (0.470142064105115, 0.059715871789770),
       (0.059715871789770, 0.470142064105115)]


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _Surface:
    """RWG functions of a mesh: edges in order of first appearance, + side the triangle that brings the edge."""

    def __init__(self, m):
        seen, rows = {}, []
        for t, tri in enumerate(m.tris.tolist()):
            for j in range(3):
                a, b, c = tri[j], tri[(j + 1) % 3], (j + 2) % 3
                if (b, a) in seen:
                    rows[seen.pop((b, a))][3:] = [t, c]
                else:
                    seen[(a, b)] = len(rows)
                    rows.append([(a, b), t, c, -1, -1])
        rows = [r for r in rows if r[3] >= 0]
        self.v = torch.tensor(m.verts, dtype=torch.float64, device=DEV)
        self.t = torch.tensor(m.tris, dtype=torch.long, device=DEV)
        e = torch.tensor([r[0] for r in rows], device=DEV)
        self.tri = [torch.tensor([r[1 + 2 * s] for r in rows], device=DEV) for s in (0, 1)]
        self.cor = [torch.tensor([r[2 + 2 * s] for r in rows], device=DEV) for s in (0, 1)]
        self.n = len(rows)
        self.c = self.v[self.t]  # corners (T, 3, 3)
        self.len = (self.v[e[:, 0]] - self.v[e[:, 1]]).norm(dim=1)
        self.free = [self.c[self.tri[s], self.cor[s]] for s in (0, 1)]
        cr = torch.linalg.cross(self.c[:, 1] - self.c[:, 0], self.c[:, 2] - self.c[:, 1])
        self.area, self.nrm = 0.5 * cr.norm(dim=1), _unit(cr)
        bary = torch.full((3, 3), 1 / 6, dtype=torch.float64, device=DEV) + 0.5 * torch.eye(3, device=DEV)
        self.q3 = torch.einsum("pj,tjx->tpx", bary, self.c)
        b7 = torch.tensor([(a, b, 1 - a - b) for a, b in _G7], dtype=torch.float64, device=DEV)
        self.q7 = torch.einsum("pj,tjx->tpx", b7, self.c)
        # RWG and sign of every triangle's corner, -1 where its opposite edge is a boundary
        self.of = torch.full((self.t.shape[0], 3), -1, dtype=torch.long, device=DEV)
        self.sgn = torch.zeros((self.t.shape[0], 3), dtype=torch.float64, device=DEV)
        for s in (0, 1):
            self.of[self.tri[s], self.cor[s]] = torch.arange(self.n, device=DEV)
            self.sgn[self.tri[s], self.cor[s]] = 1.0 - 2 * s

    def add_pairs(self, z, tf, ts, val):
        """Adds val[i, a, b], the value of triangle pair (tf[i], ts[i]) for corners (a, b), to the entries."""
        for a in range(3):
            for b in range(3):
                f, s = self.of[tf, a], self.of[ts, b]
                ok = (f >= 0) & (s >= 0)
                w = (self.sgn[tf, a] * self.sgn[ts, b])[ok] * self.len[f[ok]] * self.len[s[ok]]
                z.index_put_((f[ok], s[ok]), val[ok, a, b] * w, accumulate=True)


def _regular(S, k, q, w, skip, mfie):
    """Sums over the point pairs of all triangle pairs but those in `skip`, by entries: the EFIE and MFIE parts."""
    ze = torch.zeros(S.n, S.n, dtype=torch.complex128, device=DEV)
    zm = torch.zeros_like(ze) if mfie else None
    for i in range(len(w)):
        for j in range(len(w)):
            r = torch.cdist(q[:, i], q[:, j], compute_mode="donot_use_mm_for_euclid_dist")
            r[skip] = 1.0
            g = torch.polar(w[i] * w[j] / r, -k * r)
            g[skip] = 0
            h = g * torch.complex(torch.ones_like(r), k * r) / (r * r) if mfie else None
            for a in (0, 1):
                for b in (0, 1):
                    sg = 1.0 if a == b else -1.0
                    at = (S.tri[a][:, None], S.tri[b][None, :])
                    p, o = q[S.tri[a], i], q[S.tri[b], j]
                    rf, rs = p - S.free[a], o - S.free[b]
                    d = rf @ rs.T
                    ze += g[at] * (sg * (0.25 * d - 1 / k ** 2))
                    if mfie:
                        n = S.nrm[S.tri[a]]
                        m = (_dot(rf, p)[:, None] - rf @ o.T) * (n @ rs.T) - d * (_dot(n, p)[:, None] - n @ o.T)
                        zm += h[at] * (sg * m)
    return ze, zm


def _self_efie(S, k):
    """Self terms of the 3 x 3-point rule by (triangle, field corner, source corner): the expansion of the smooth
    part and the closed form of the 1/R part."""
    val = torch.zeros(S.t.shape[0], 3, 3, dtype=torch.complex128, device=DEV)
    for p in range(3):
        g = S.q3[:, p]
        rf = g[:, None] - S.c
        for q in range(3):
            r = (g - S.q3[:, q]).norm(dim=1)
            rs = S.q3[:, q][:, None] - S.c
            coff = torch.complex(-0.5 * k * k * r, k / 6 * (k * k * r * r - 6))
            val += coff[:, None, None] / 9 * (0.25 * torch.einsum("tax,tbx->tab", rf, rs) - 1 / k ** 2)
        i1 = torch.zeros_like(g)
        i2 = torch.zeros_like(g[:, 0])
        for e in range(3):
            a, b = S.c[:, (e + 1) % 3], S.c[:, e]
            l = _unit(a - b)
            u = torch.linalg.cross(l, S.nrm)
            p0 = _dot(b - g, u).abs()
            lp, lm, rp, rm = _dot(a - g, l), _dot(b - g, l), (a - g).norm(dim=1), (b - g).norm(dim=1)
            lg = torch.log((rp + lp) / (rm + lm))
            i1 += 0.5 * u * (p0 * p0 * lg + lp * rp - lm * rm)[:, None]
            i2 += p0 * lg
        src = i1[:, None] + (g[:, None] - S.c) * i2[:, None, None]
        val += ((0.25 * torch.einsum("tax,tbx->tab", rf, src) - i2[:, None, None] / k ** 2) / 3) / S.area[:, None, None]
    return val


def _self_cfie(S, k, alpha):
    """Self terms of the combined equation; its logarithmic part takes the last point's source vector."""
    ze = torch.zeros(S.t.shape[0], 3, 3, dtype=torch.complex128, device=DEV)
    zm = torch.zeros(S.t.shape[0], 3, 3, dtype=torch.float64, device=DEV)
    for p in range(3):
        g = S.q3[:, p]
        rf = g[:, None] - S.c
        for q in range(3):
            r = (g - S.q3[:, q]).norm(dim=1)
            rs = S.q3[:, q][:, None] - S.c
            e = 0.25 * torch.einsum("tax,tbx->tab", rf, rs) - 1 / k ** 2
            coff = torch.complex(-0.5 * k * k * r, k / 6 * (k * k * r * r - 6))
            ze += coff[:, None, None] / 9 * e
        for i in range(3):
            a, b = S.c[:, (i + 1) % 3], S.c[:, i]
            l = _unit(a - b)
            p0 = (b + l * _dot(g - b, l)[:, None] - g).norm(dim=1)
            lg = torch.log(((a - g).norm(dim=1) + _dot(a - g, l)) / ((b - g).norm(dim=1) + _dot(b - g, l)))
            ze += e / 3 * (p0 * lg / S.area)[:, None, None]
        zm += torch.einsum("tax,tbx->tab", rf, rf) / 3
    return alpha * 1j * k * _Z0 / (4 * math.pi) * ze + (1 - alpha) * _Z0 * zm / (8 * S.area[:, None, None])


def _singular_config(S, k):
    """Self and edge-adjacent pairs of the 7-point rule: (mask, field triangles, source triangles, values)."""
    t = S.t.shape[0]
    skip = torch.eye(t, dtype=torch.bool, device=DEV)
    skip[S.tri[0], S.tri[1]] = True
    skip[S.tri[1], S.tri[0]] = True
    tf, ts = torch.nonzero(skip, as_tuple=True)
    val = torch.zeros(tf.shape[0], 3, 3, dtype=torch.complex128, device=DEV)
    cf, cs, n = S.c[tf], S.c[ts], S.nrm[ts]
    for p in range(7):
        g = S.q7[tf, p]
        rf = g[:, None] - cf
        for q in range(7):
            o = S.q7[ts, q]
            r = (g - o).norm(dim=1)
            rr = torch.where(r > 0, r, torch.ones_like(r))
            gs = torch.complex(-2 * torch.sin(0.5 * k * rr) ** 2 / rr, -torch.sin(k * rr) / rr)
            gs = torch.where(r > 0, gs, torch.full_like(gs, -1j * k))
            val += (_W7[p] * _W7[q] * gs)[:, None, None] * (
                0.25 * torch.einsum("tax,tbx->tab", rf, o[:, None] - cs) - 1 / k ** 2)
        h = _dot(g - cs[:, 0], n)
        rho = g - n * h[:, None]
        i1 = torch.zeros_like(h)
        ir = torch.zeros_like(g)
        for e in range(3):
            a, b = cs[:, (e + 1) % 3], cs[:, e]
            l = _unit(a - b)
            u = torch.linalg.cross(l, n)
            lp, lm, sd = _dot(a - rho, l), _dot(b - rho, l), _dot(b - rho, u)
            r02 = sd * sd + h * h
            rp, rm = torch.sqrt(r02 + lp * lp), torch.sqrt(r02 + lm * lm)
            lg = torch.log(torch.where(lp >= 0, rp + lp, r02 / (rp - lp)) / torch.where(lm >= 0, rm + lm, r02 / (rm - lm)))
            ah = h.abs()
            ir += u * (0.5 * (r02 * lg + lp * rp - lm * rm))[:, None]
            i1 += sd * lg - torch.sign(sd) * ah * (torch.atan(sd.abs() * lp / (r02 + ah * rp))
                                                  - torch.atan(sd.abs() * lm / (r02 + ah * rm)))
        src = ir[:, None] + (rho[:, None] - cs) * i1[:, None, None]
        val += _W7[p] * (0.25 * torch.einsum("tax,tbx->tab", rf, src) - i1[:, None, None] / k ** 2) \
            / S.area[ts][:, None, None]
    return skip, tf, ts, val


def _impedance(S, freq, kind, disc="reference", alpha=0.5):
    k = 2 * math.pi * freq / C0
    ll = S.len[:, None] * S.len[None, :]
    if disc == "config":
        skip, tf, ts, val = _singular_config(S, k)
        z = _regular(S, k, S.q7, _W7, skip, False)[0].mul_(ll)
        S.add_pairs(z, tf, ts, val)
        return z.mul_(1j * k * _Z0 / (4 * math.pi))
    t = torch.arange(S.t.shape[0], device=DEV)
    skip = torch.eye(S.t.shape[0], dtype=torch.bool, device=DEV)
    ze, zm = _regular(S, k, S.q3, [1 / 3] * 3, skip, kind == "cfie")
    if kind == "cfie":
        z = ze.mul_(alpha * 1j * k * _Z0 / (4 * math.pi)).add_(zm, alpha=(1 - alpha) * _Z0 / (16 * math.pi)).mul_(ll)
        S.add_pairs(z, t, t, _self_cfie(S, k, alpha))
        return z
    z = ze.mul_(ll)
    S.add_pairs(z, t, t, _self_efie(S, k))
    return z.mul_(1j * k * _Z0 / (4 * math.pi))


def _rcs(m, freq, kind, ang, dirs, per_rhs, alpha=0.5):
    """RCS in dBsm of every incidence, by a direct solve."""
    S = _Surface(m)
    k = 2 * math.pi * freq / C0
    z = _impedance(S, freq, kind, alpha=alpha)
    th, ph, po = np.deg2rad(ang).T
    kk = np.stack([-np.sin(th) * np.cos(ph), -np.sin(th) * np.sin(ph), -np.cos(th)], 1)
    ee = np.stack([-np.cos(po) * np.cos(th) * np.cos(ph) - np.sin(po) * np.sin(ph),
                   -np.cos(po) * np.cos(th) * np.sin(ph) + np.sin(po) * np.cos(ph), np.cos(po) * np.sin(th)], 1)
    kk, ee, hh = (torch.tensor(a, device=DEV) for a in (kk, ee, np.cross(kk, ee)))
    v = torch.zeros(S.n, len(ang), dtype=torch.complex128, device=DEV)
    q, w = (S.q3, [1 / 3] * 3) if kind == "cfie" else (S.q7, _W7)
    for s in (0, 1):
        for i in range(len(w)):
            p = q[S.tri[s], i]
            rho = (p - S.free[s]) * (1 - 2 * s)
            amp = rho @ ee.T
            if kind == "cfie":
                amp = alpha * amp + (1 - alpha) * (torch.linalg.cross(rho, S.nrm[S.tri[s]]) @ hh.T)
            v += torch.polar(w[i] * amp, -k * (p @ kk.T))
    cur = torch.linalg.solve(z, v * (0.5 * S.len)[:, None])
    d = torch.tensor(np.asarray(dirs), dtype=torch.float64, device=DEV)
    out = []
    for a in range(len(ang)):
        da = d[a] if per_rhs else d
        far = torch.zeros(da.shape[0], 3, dtype=torch.complex128, device=DEV)
        il = cur[:, a] * S.len
        for s in (0, 1):
            for i in range(7):
                p = S.q7[S.tri[s], i]
                x = k * (da @ p.T)
                far += (torch.polar(torch.full_like(x, _W7[i] * (1 - 2 * s)), x) * il) @ (p - S.free[s]).to(far.dtype)
        dc = da.to(far.dtype)
        es = 0.5 * torch.linalg.cross(dc, torch.linalg.cross(dc, far))
        out.append(10 * torch.log10(_Z0 ** 2 * k * k * es.abs().square().sum(1) / (4 * math.pi)))
    return torch.stack(out).cpu().numpy()


def exact(case, seed):
    path = case["path"]
    if path == "job":
        m, freq, ang, dirs, per_rhs = _job_inputs(case, seed)
        return _rcs(m, freq, case["kind"], ang, dirs, per_rhs)
    if path == "batch":
        return [_rcs(m, freq, "efie", ang, dirs, True) for m, freq, ang, dirs in _batch_inputs(case, seed)]
    if path == "fill":
        m, freq = _target(case["f"], np.random.default_rng(seed), case["open"])
        return _impedance(_Surface(m), freq, case["kind"], case["disc"])
    if path == "product":
        z, x = _product_inputs(case, seed)
        return x.to(torch.complex128) @ z.to(torch.complex128).T
    # the multilevel product has its own truncation and interpolation error, far above rounding: its value in 64
    # bits is a whole multilevel code on the CPU, minutes at these sizes
    return None

"""Corner forces of compressible neo-Hookean elements in the plain FP64 mode
(64-bit fixed point, FP64 for the elements it leaves out) against the same
formulas in extended precision, over element shapes, sizes, rigid motions,
stretches, volume changes and materials at and beyond the ends of its range."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu

N = 600   # tets a case: two CTAs' worth and a remainder
EPS = 2.0 ** -53


def tets(rng, scale, flat):
    """N disjoint jittered corner tets, z scaled by `flat`; X (3, 4N), conn."""
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    x = (ref[None] + rng.uniform(-0.15, 0.15, (N, 4, 3))) * [1, 1, flat] + rng.uniform(-3, 3, (N, 1, 3))
    return np.ascontiguousarray((scale * x).reshape(4 * N, 3).T), np.arange(4 * N, dtype=np.int32).reshape(N, 4)


def rotation(axis, angle):
    k = np.asarray(axis, float) / np.linalg.norm(axis)
    K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
    return np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K


def reference(X, u, conn, lam, mu):
    """Forces (N, 4, 3) in extended precision and their error scale (N, 4)."""
    L = np.longdouble
    x, w = X.T.astype(L)[conn], u.T.astype(L)[conn]
    E = x[:, 1:] - x[:, :1]
    e = E + (w[:, 1:] - w[:, :1])
    nxt, prv = [1, 2, 0], [2, 0, 1]
    G, C = np.cross(E[:, nxt], E[:, prv]), np.cross(e[:, nxt], e[:, prv])
    D0, D = (E[:, 0] * G[:, 0]).sum(-1), (e[:, 0] * C[:, 0]).sum(-1)
    G = G / D0[:, None, None]
    M = np.einsum("nai,nbi->nab", G, G)
    wJ, J = L(0.166666666667) * abs(D0), D / D0
    lam, mu = L(lam), L(mu)
    c2 = wJ * (lam * np.log(J) - mu) / D
    f = (wJ * mu)[:, None, None] * np.einsum("nab,nbi->nai", M, e) + c2[:, None, None] * C
    f = np.concatenate([-f.sum(1, keepdims=True), f], 1)
    # every rounding of either form is relative to these sums of magnitudes; J's
    # error is that of a product of three edges over the volume
    ne, nE = np.linalg.norm(e.astype(float), axis=-1), np.linalg.norm(E.astype(float), axis=-1)
    kap = ne.prod(1) / abs(D.astype(float)) + nE.prod(1) / abs(D0.astype(float))
    wJ, J, lam, mu = wJ.astype(float), J.astype(float), float(lam), float(mu)
    cross = np.stack([ne[:, 1] * ne[:, 2], ne[:, 2] * ne[:, 0], ne[:, 0] * ne[:, 1]], 1)
    s = (wJ * mu)[:, None] * np.einsum("nab,nb->na", abs(M.astype(float)), np.maximum(ne, nE))
    s += (wJ * (abs(mu - lam * np.log(J)) + (abs(lam) + mu) * kap) / abs(D.astype(float)))[:, None] * cross
    s = kap[:, None] * s
    return f, np.concatenate([s.sum(1, keepdims=True), s], 1)


CASES = {
    "rest": dict(),
    "small strain": dict(strain=1e-7),
    "strain": dict(strain=1e-3),
    "volume near the short series' end": dict(strain=4e-3),
    "volume near the long series' end": dict(strain=3e-2),
    "volume beyond the series": dict(strain=0.15),
    "compressed": dict(stretch=0.55),
    "stretched inside the range": dict(stretch=1.9),
    "stretched past the range": dict(stretch=4.5),
    "rotated": dict(rot=2.8, strain=1e-3),
    "moved far": dict(shift=1e3, strain=1e-3),
    "flat": dict(flat=0.05, strain=1e-3),
    "flat past the range": dict(flat=0.004, strain=1e-3),
    "tall": dict(flat=30.0, strain=1e-3),
    "small body": dict(scale=1e-9, strain=1e-3),
    "large body": dict(scale=1e7, strain=1e-3),
    "no Poisson effect": dict(nu=0.0, strain=1e-2),
    "auxetic": dict(nu=-0.6, strain=1e-2),
    "nearly incompressible": dict(nu=0.49, strain=1e-3),
    "incompressible but for a little": dict(nu=0.4999, strain=1e-3),
    "soft": dict(young=1e-4, strain=1e-2),
    "hard": dict(young=1e13, strain=1e-2),
}


@pytest.mark.parametrize("name", list(CASES))
def test_corner_forces(name):
    o = dict(strain=0.0, stretch=1.0, rot=0.0, shift=0.0, flat=1.0, scale=1.0, nu=0.3, young=1e6)
    o.update(CASES[name])
    rng = np.random.default_rng(len(name))
    X, conn = tets(rng, o["scale"], o["flat"])
    x = X.T[conn]
    F = rotation([1, 2, -1], o["rot"]) @ (o["stretch"] * np.eye(3)) + o["strain"] * rng.uniform(-1, 1, (N, 3, 3))
    y = np.einsum("nij,naj->nai", F, x - x[:, :1]) + x[:, :1] + o["shift"] * o["scale"] * np.array([1.0, -0.7, 0.3])
    u = np.ascontiguousarray((y - x).reshape(4 * N, 3).T)
    S = msx.Solver(X, conn, [(msx.COMPRESSIBLE_NH, o["young"], o["nu"], 1000.0)], [], 0.0, 1e30, 0.5)
    S.set_state(u.ravel())
    S.run(1)   # from rest: the forces are those of u
    f = np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, np.arange(4 * N)) for c in range(3)], 1).reshape(N, 4, 3)
    assert np.array_equal(S.state()[0], u.ravel())
    S.close()
    lam = o["young"] * o["nu"] / ((1 + o["nu"]) * (1 - 2 * o["nu"]))
    want, scale = reference(X, u, conn, lam, 0.5 * o["young"] / (1 + o["nu"]))
    # the moved body's u holds positions to EPS |u|: the forces' inputs are exact, their edges round at that size
    edge = 1.0 + o["shift"] * 1e-3
    assert np.isfinite(f).all()
    err = np.abs((f - want).astype(float)).max(-1) / (64 * EPS * edge * scale)
    assert err.max() <= 1.0, err.max()


def test_non_finite_displacement_is_reported():
    X, conn = tets(np.random.default_rng(3), 1.0, 1.0)
    S = msx.Solver(X, conn, [(msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
    u = np.zeros(3 * X.shape[1])
    u[1] = np.nan
    S.set_state(u)
    with pytest.raises(msx.MsxError) as err:
        S.run(3)
    assert err.value.status == 4
    S.close()


def test_materials_of_two_laws():
    """A part whose second material is not compressible neo-Hookean: each element takes its own law's form."""
    import oracle as O
    X, conn = msx.mesh_cube(6, 3, 0.1)
    mesh = O.Mesh(X, conn)
    ids = (np.arange(conn.shape[0]) % 3 == 1).astype(np.int32)
    bcs = msx.cube_bcs(6, 0.002)
    mesh.elem_mat = ids
    mats = [O.Material(O.COMPRESSIBLE_NH), O.Material(O.STVK)]
    ref = O.run(mesh, mats, [O.Solver(0.0, 0.01, 0.5, bcs)])
    S = msx.Solver(X, conn, [(msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0), (msx.STVK, 1e6, 0.3, 1000.0)], bcs, 0.0, 0.01, 0.5,
                   elem_material=ids)
    rep = S.run()
    u = S.state()[0]
    S.close()
    assert rep.steps == ref.steps and np.linalg.norm(u - ref.u) <= 1e-10 * np.linalg.norm(ref.u)

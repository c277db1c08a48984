"""Corner forces of St-Venant-Kirchhoff and linear elastic elements in the plain
FP64 mode (64-bit fixed point, FP64 for the elements it leaves out) against the
same formulas in extended precision, over element shapes, sizes, rigid motions,
stretches and materials at and beyond the ends of its range."""
import numpy as np
import pytest

import msx
from test_gpu_fixed_point import EPS, N, rotation, tets

pytestmark = pytest.mark.gpu


def reference(X, u, conn, linear, lam, mu2):
    """Forces (N, 4, 3) in extended precision and their error scale (N, 4)."""
    L = np.longdouble
    x, w = X.T.astype(L)[conn], u.T.astype(L)[conn]
    E, du = x[:, 1:] - x[:, :1], w[:, 1:] - w[:, :1]
    G = np.cross(E[:, [1, 2, 0]], E[:, [2, 0, 1]])
    D = (E[:, 0] * G[:, 0]).sum(-1)
    G = G / D[:, None, None]
    H = np.einsum("nbi,nbj->nij", du, G)
    S = H + H.transpose(0, 2, 1)
    if not linear:
        S = S + np.einsum("nki,nkj->nij", H, H)
    I = np.eye(3, dtype=L)
    S = (L(mu2) * S + L(lam) * np.einsum("nii->n", S)[:, None, None] * I) / 2
    P = S if linear else np.einsum("nij,njk->nik", I + H, S)
    wJ = L(0.166666666667) * abs(D)
    f = wJ[:, None, None] * np.einsum("nij,naj->nai", P, G)
    f = np.concatenate([-f.sum(1, keepdims=True), f], 1)
    # roundings of H, S and P: relative to 1 and to the sums of magnitudes that
    # make H, whose gradients carry a relative error of the edges over the heights
    dn, gn, En = (np.linalg.norm(a.astype(float), axis=-1) for a in (du, G, E))
    h = (dn * gn).sum(-1)
    kap = En.prod(1) / abs(D.astype(float))
    s = wJ.astype(float) * (mu2 + 3 * abs(lam)) * kap * (1 + h) ** (1 if linear else 3)
    s = s[:, None] * gn
    return f, np.concatenate([s.sum(1, keepdims=True), s], 1)


CASES = {
    "rest": dict(),
    "small strain": dict(strain=1e-7),
    "strain": dict(strain=1e-3),
    "large strain": dict(strain=0.2),
    "compressed": dict(stretch=0.4),
    "stretched inside the range": dict(stretch=1.5),
    "stretched past the range": dict(stretch=4.5),
    "rotated": dict(rot=2.8, strain=1e-3),
    "moved far": dict(shift=1e3, strain=1e-3),
    "flat": dict(flat=0.3, strain=1e-3),
    "flat past the range": dict(flat=0.02, strain=1e-3),
    "tall": dict(flat=5.0, strain=1e-3),
    "small body": dict(scale=1e-9, strain=1e-3),
    "large body": dict(scale=1e7, strain=1e-3),
    "no Poisson effect": dict(nu=0.0, strain=1e-2),
    "auxetic": dict(nu=-0.6, strain=1e-2),
    "nearly incompressible": dict(nu=0.4999, strain=1e-3),
    "incompressible past the range": dict(nu=0.4999999, strain=1e-3),
    "soft": dict(young=1e-4, strain=1e-2),
    "hard": dict(young=1e13, strain=1e-2),
}


@pytest.mark.parametrize("law", [msx.STVK, msx.LINEAR_ELASTIC])
@pytest.mark.parametrize("name", list(CASES))
def test_corner_forces(name, law):
    o = dict(strain=0.0, stretch=1.0, rot=0.0, shift=0.0, flat=1.0, scale=1.0, nu=0.3, young=1e6)
    o.update(CASES[name])
    rng = np.random.default_rng(len(name))
    X, conn = tets(rng, o["scale"], o["flat"])
    x = X.T[conn]
    F = rotation([1, 2, -1], o["rot"]) @ (o["stretch"] * np.eye(3)) + o["strain"] * rng.uniform(-1, 1, (N, 3, 3))
    y = np.einsum("nij,naj->nai", F, x - x[:, :1]) + x[:, :1] + o["shift"] * o["scale"] * np.array([1.0, -0.7, 0.3])
    u = np.ascontiguousarray((y - x).reshape(4 * N, 3).T)
    S = msx.Solver(X, conn, [(law, o["young"], o["nu"], 1000.0)], [], 0.0, 1e30, 0.5)
    S.set_state(u.ravel())
    S.run(1)   # from rest: the forces are those of u
    f = np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, np.arange(4 * N)) for c in range(3)], 1).reshape(N, 4, 3)
    assert np.array_equal(S.state()[0], u.ravel())
    S.close()
    lam = o["young"] * o["nu"] / ((1 + o["nu"]) * (1 - 2 * o["nu"]))
    want, scale = reference(X, u, conn, law == msx.LINEAR_ELASTIC, lam, o["young"] / (1 + o["nu"]))
    edge = 1.0 + o["shift"] * 1e-3   # positions are held to EPS |u|
    assert np.isfinite(f).all()
    err = np.abs((f - want).astype(float)).max(-1) / (64 * EPS * edge * scale)
    assert err.max() <= 1.0, err.max()


@pytest.mark.parametrize("law", [msx.STVK, msx.LINEAR_ELASTIC])
def test_non_finite_displacement_is_reported(law):
    X, conn = tets(np.random.default_rng(3), 1.0, 1.0)
    S = msx.Solver(X, conn, [(law, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
    u = np.zeros(3 * X.shape[1])
    u[1] = np.nan
    S.set_state(u)
    with pytest.raises(msx.MsxError) as err:
        S.run(3)
    assert err.value.status == 4
    S.close()


@pytest.mark.parametrize("law", [msx.STVK, msx.LINEAR_ELASTIC])
def test_unborn_elements_have_no_force(law):
    X, conn = tets(np.random.default_rng(5), 1.0, 1.0)
    born = np.where(np.arange(N) % 3 == 0, 1e20, 0.0)
    u = 1e-3 * np.random.default_rng(6).uniform(-1, 1, 3 * X.shape[1])
    f = []
    for times in (None, born):
        S = msx.Solver(X, conn, [(law, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
        if times is not None:
            S.set_activation(times)
        S.set_state(u)
        S.run(1)
        f.append(np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, np.arange(4 * N)) for c in range(3)], 1)
                 .reshape(N, 4, 3))
        S.close()
    assert (f[1][::3] == 0).all() and (f[0][::3] != 0).any()
    keep = np.arange(N) % 3 != 0
    assert np.array_equal(f[0][keep], f[1][keep])

"""Meshes in which some, most or all elements are left out by the fixed-point
forms of the plain FP64 mode (flat tets, tets stretched past the range), which the element
kernels list and compute at the end of a tile: forces against extended
precision, the time step, and the same bits from the pool's tiles, around the
sizes of CTAs and tiles."""
import numpy as np
import pytest

import msx
import test_gpu_fixed_point as cnh
import test_gpu_fixed_stress as svk
from test_gpu_fixed_point import EPS
from test_gpu_sliver_dt import expected_dt

pytestmark = pytest.mark.gpu

LAWS = [msx.COMPRESSIBLE_NH, msx.STVK, msx.LINEAR_ELASTIC]
YOUNG, NU = 1e6, 0.3
LAM, MU2 = YOUNG * NU / ((1 + NU) * (1 - 2 * NU)), YOUNG / (1 + NU)


HEIGHT = 4e-4   # flatter than any of the forms takes


def mesh(n, flat, far, seed):
    """n disjoint jittered corner tets, a share `flat` of them of that height, and a displacement of strain 1e-3 that
    stretches a share `far` of them sixfold along x."""
    rng = np.random.default_rng(seed)
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    x = ref[None] + rng.uniform(-0.15, 0.15, (n, 4, 3))
    x[rng.random(n) < flat, :, 2] *= HEIGHT
    F = np.eye(3) + 1e-3 * rng.uniform(-1, 1, (n, 3, 3))
    F[rng.random(n) < far, 0] *= 6.0
    y = np.einsum("nij,naj->nai", F, x - x[:, :1]) + x[:, :1]
    X = np.ascontiguousarray(x.reshape(4 * n, 3).T)
    u = np.ascontiguousarray((y - x).reshape(4 * n, 3).T)
    return X, np.arange(4 * n, dtype=np.int32).reshape(n, 4), u


def check(f, X, u, conn, law):
    if law == msx.COMPRESSIBLE_NH:
        want, scale = cnh.reference(X, u, conn, LAM, 0.5 * MU2)
    else:
        want, scale = svk.reference(X, u, conn, law == msx.LINEAR_ELASTIC, LAM, MU2)
    err = np.abs((f.reshape(3, -1).T.reshape(-1, 4, 3) - want).astype(float)).max(-1) / (64 * EPS * scale)
    assert np.isfinite(f).all() and err.max() <= 1.0, err.max()


@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("flat,far", [(0.01, 0.0), (0.5, 0.0), (1.0, 0.0), (0.0, 0.02), (0.0, 1.0), (0.3, 0.3)])
@pytest.mark.parametrize("n", [1, 31, 129, 700, 19457, 90000])
def test_forces_and_time_step(n, flat, far, law):
    if n > 700 and law == msx.LINEAR_ELASTIC:
        pytest.skip("the same kernel as St-Venant-Kirchhoff's")
    X, conn, u = mesh(n, flat, far, n)
    nodes = np.arange(X.shape[1])
    S = msx.Solver(X, conn, [(law, YOUNG, NU, 1000.0)], [], 0.0, 1e30, 0.5)
    check(S.internal_force(u.ravel()), X, u, conn, law)
    S.set_state(u.ravel())
    first = S.run(1).dt
    check(np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, nodes) for c in range(3)]), X, u, conn, law)
    second = S.run(1).dt
    S.close()
    want = expected_dt(X, conn, u, law)
    tol = 64 * EPS * 2 / HEIGHT   # positions of size 2
    assert abs(first - want) <= tol * want and abs(second - want) <= tol * want


@pytest.mark.parametrize("law", [msx.COMPRESSIBLE_NH, msx.STVK])
@pytest.mark.parametrize("tile", [128, 256, 1024, 4096])
def test_pool_bits(law, tile):
    """Nodes driven in one step to where some tets are stretched past the range: the pool's tiles give the bits of the
    solve run alone."""
    X, conn, u = mesh(5000, 0.2, 0.2, 3)
    bcs = msx.bc_array([])
    bcs = np.zeros(3 * X.shape[1] // 2, bcs.dtype)
    bcs["dof"] = 2 * np.arange(len(bcs))
    bcs["mode"] = msx.BC_INST
    bcs["value"] = u.ravel()[bcs["dof"]]
    mat = (law, YOUNG, NU, 1000.0)
    S = msx.Solver(X, conn, [mat], bcs, 0.0, 1e30, 0.5, max_steps=5)
    S.run()
    alone = S.state()
    S.close()
    P = msx.Pool(max_slots=1, precision=msx.FP64, elems_per_block=tile)
    t = P.submit(X, conn, mat, bcs, 5)
    P.wait(t)
    pooled = P.fetch(t)
    P.close()
    for a, b in zip(alone, pooled):   # the flattest tets of St-Venant-Kirchhoff overturn: NaN in both
        assert np.array_equal(a, b, equal_nan=True)


def test_two_laws_in_a_tile():
    """Left-out elements of both laws share a tile: each takes its own law's FP64 form."""
    X, conn, u = mesh(3000, 0.4, 0.1, 11)
    ids = (np.arange(len(conn)) % 3 == 1).astype(np.int32)
    S = msx.Solver(X, conn, [(msx.COMPRESSIBLE_NH, YOUNG, NU, 1000.0), (msx.STVK, YOUNG, NU, 1000.0)], [], 0.0, 1e30, 0.5,
                   elem_material=ids)
    S.set_state(u.ravel())
    S.run(1)
    f = np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, np.arange(X.shape[1])) for c in range(3)])
    S.close()
    for k, law in enumerate((msx.COMPRESSIBLE_NH, msx.STVK)):
        mine = conn[ids == k]
        check(np.ascontiguousarray(f[:, mine.ravel()]), np.ascontiguousarray(X[:, mine.ravel()]),
              np.ascontiguousarray(u[:, mine.ravel()]), np.arange(mine.size).reshape(-1, 4), law)

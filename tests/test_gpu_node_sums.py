"""The FP64 node kernel's sums of corner forces where its integer form ends (a
component of zeros, forces near the bottom of the FP64 range) and over meshes of
several passes a block, which the single-solve kernel hands out in another way
than the pool's."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu


def forces(young, u, X, conn):
    S = msx.Solver(X, conn, [(msx.LINEAR_ELASTIC, young, 0.0, 1e-3 * young)], [], 0.0, 1e30, 0.5)
    S.set_state(u.ravel())
    S.run(1)   # from rest: the forces are those of u
    nn = X.shape[1]
    f = np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, np.arange(nn)) for c in range(3)])
    S.close()
    return f


@pytest.mark.parametrize("k", [-300, -700, -900, -930, -940, -950])
def test_forces_scale_with_the_modulus(k):
    """Linear elasticity: forces are proportional to a power-of-two modulus, through integer sums or FP64 ones
    (forces of 2^-948 and less)."""
    X, conn = msx.mesh_cube(4, 3, 0.1)
    u = 1e-2 * np.random.default_rng(1).uniform(-1, 1, X.shape)
    u[1] = 0.0
    f, g = forces(1.0, u, X, conn), forces(2.0 ** k, u, X, conn) * 2.0 ** -k
    # corner forces scale exactly; the 24 terms of a node add with at most 24 roundings of their sum of magnitudes
    assert np.abs(f - g).max() <= 24 * 24 * 2.0 ** -53 * np.abs(f).max()


def test_components_of_zeros():
    X, conn = msx.mesh_cube(4, 3, 0.0)
    assert (forces(1e6, np.zeros_like(X), X, conn) == 0).all()
    u = np.zeros_like(X)
    u[0] = 1e-3 * X[0]   # no Poisson effect: no force along y and z
    f = forces(1e6, u, X, conn)
    assert np.abs(f[0]).max() > 1 and (np.abs(f[1:]) <= 1e-12 * np.abs(f[0]).max()).all()


@pytest.mark.parametrize("precision", [msx.FP64, msx.MIXED, msx.DOUBLE_WORD])
@pytest.mark.parametrize("n", [28, 35, 43])
def test_single_equals_pool(n, precision):
    """24,389 to 85,184 nodes: a grid of one and of several passes a block."""
    X, conn = msx.mesh_cube(n, 2, 0.1)
    bcs = msx.cube_bcs(n, 0.05, msx.BC_VEL_RAMP, 4)
    mat = (msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0)
    S = msx.Solver(X, conn, [mat], bcs, 0.0, 1e30, 0.5, precision=precision)
    S.run(6)
    u, v = S.state()[:2]
    S.close()
    P = msx.Pool(max_slots=1, precision=precision)
    t = P.submit(X, conn, mat, bcs, 6)
    P.wait(t)
    w, x = P.fetch(t)[:2]
    P.close()
    assert np.array_equal(u, w) and np.array_equal(v, x)

"""The time step of meshes whose CFL minimum is a reference sliver (a tet flatter
than the FP32 screen resolves, which is always recomputed in FP64), under large
rotations and shears, in the four precision modes and the pool."""
import numpy as np
import pytest

import msx
from test_gpu_fixed_point import rotation

pytestmark = pytest.mark.gpu

PRECISIONS = [msx.FP64, msx.FP64_EXACT, msx.MIXED, msx.DOUBLE_WORD]
MOTIONS = {
    "rest": np.eye(3),
    "rotated by 91 degrees": rotation([1, 2, -1], np.radians(91)),
    "rotated by 120 degrees": rotation([1, 2, -1], np.radians(120)),
    "rotated by 180 degrees": rotation([0, 1, 1], np.pi),
    "sheared in the sliver's plane": np.eye(3) + 3.0 * np.outer([1, 0, 0], [0, 1, 0]),
    "sheared across the sliver": np.eye(3) + 2.5 * np.outer([1, 0, 0], [0, 0, 1]),
    "stretched": np.diag([4.0, 4.0, 4.0]),
}


def mesh(height):
    """A 4^3 cube and, apart from it, one flat tet of the given height over its base."""
    X, conn = msx.mesh_cube(4, 5, 0.1)
    flat = np.array([[2, 0, 0], [2.3, 0, 0], [2, 0.3, 0], [2.1, 0.1, height]]).T
    nn = X.shape[1]
    return (np.ascontiguousarray(np.concatenate([X, flat], 1)),
            np.ascontiguousarray(np.concatenate([conn, nn + np.arange(4, dtype=np.int32)[None]]).astype(np.int32)))


def inscribed(X, conn):
    x = X.T[conn]
    e = x[:, 1:] - x[:, :1]
    six_v = abs(np.linalg.det(e))
    faces = [np.cross(e[:, 0], e[:, 1]), np.cross(e[:, 0], e[:, 2]), np.cross(e[:, 1], e[:, 2]),
             np.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])]
    return 2 * six_v / sum(np.linalg.norm(f, axis=1) for f in faces)


def expected_dt(X, conn, u, law):
    E, nu, rho = 1e6, 0.3, 1000.0
    c = np.sqrt(E / rho) if law >= 2 else np.sqrt(E * (1 - nu) / ((1 + nu) * (1 - 2 * nu)) / rho)
    return 0.5 * min(inscribed(X, conn).min(), inscribed(X + u, conn).min()) / c


# 6V over the product of the edges: 0.063 marks a sliver
@pytest.mark.parametrize("height", [0.008, 1e-4])
@pytest.mark.parametrize("name", list(MOTIONS))
@pytest.mark.parametrize("precision", PRECISIONS)
def test_time_step(name, precision, height):
    X, conn = mesh(height)
    assert inscribed(X, conn).argmin() == len(conn) - 1
    u = MOTIONS[name] @ (X - 0.5) + 0.5 - X
    for law in (msx.COMPRESSIBLE_NH, msx.STVK):
        S = msx.Solver(X, conn, [(law, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5, precision=precision)
        S.set_state(u.ravel())
        first, second = S.run(1).dt, S.run(1).dt
        S.close()
        want = expected_dt(X, conn, u, law)
        # FP64 roundings of positions of size 8 over the sliver's height, and u's own 2^-48 in the pair-state modes
        tol = (2.0 ** -53 * 64 + (2.0 ** -46 if precision in (msx.MIXED, msx.DOUBLE_WORD) else 0)) * 8 / height
        assert abs(first - want) <= tol * want and abs(second - want) <= tol * want, (first, second, want)


@pytest.mark.parametrize("precision", [msx.FP64, msx.MIXED, msx.DOUBLE_WORD])
@pytest.mark.parametrize("name", ["rotated by 120 degrees", "rotated by 180 degrees"])
def test_pool(name, precision):
    """Every node driven to the rotated position in the first step: the same bits as the solve run alone, at the
    sliver's time step."""
    X, conn = mesh(0.008)
    u = MOTIONS[name] @ (X - 0.5) + 0.5 - X
    bcs = [(int(d), msx.BC_INST, float(v), 0) for d, v in enumerate(u.ravel())]
    mat = (msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0)
    S = msx.Solver(X, conn, [mat], bcs, 0.0, 1e30, 0.5, max_steps=4, precision=precision)
    rep = S.run()
    state = S.state()
    S.close()
    want = expected_dt(X, conn, u, msx.COMPRESSIBLE_NH)
    assert rep.steps == 4 and abs(rep.t - 4 * want) <= 1e-9 * want
    P = msx.Pool(max_slots=1, precision=precision, elems_per_block=256)
    t = P.submit(X, conn, mat, bcs, 4)
    res = P.wait(t)
    pooled = P.fetch(t)
    P.close()
    assert res["t"] == rep.t
    for a, b in zip(state, pooled):
        assert np.array_equal(a, b)

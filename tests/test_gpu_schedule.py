"""Single solves at the sizes where the step kernels' schedule changes (CTA
size, one tile a CTA or the tile queue, remainders of tiles and of node
passes), against the oracle, and whatever the schedule: the same solve split
into several calls, and the pool's kernels, give the same bits."""
import numpy as np
import pytest

import msx
import oracle as O

pytestmark = pytest.mark.gpu

# hexes a side -> tets: one warp's worth and less, a tile's edge, 152 x 128
# elements (128-thread CTAs up to there), one tile a CTA up to 304 x 256, above
SIDES = [1, 2, 3, 5, 14, 15, 23, 24]


@pytest.mark.parametrize("n", SIDES)
@pytest.mark.parametrize("precision,tol", [(msx.FP64, 1e-11), (msx.MIXED, 1e-5), (msx.DOUBLE_WORD, 1e-10)])
def test_sizes(n, precision, tol):
    mesh = O.cube_mesh(n)
    bcs = O.cube_bcs(n, 0.05, O.BC_VEL_RAMP, 4)
    ref = O.run(mesh, [O.Material(O.COMPRESSIBLE_NH)], [O.Solver(0.0, 1e30, 0.5, bcs, max_steps=6)])
    S = msx.Solver(mesh.X, mesh.conn, [(msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0)], bcs, 0.0, 1e30, 0.5, max_steps=6,
                   precision=precision)
    steps = S.run(2).steps + S.run(3).steps + S.run().steps
    u, v, a = S.state()
    S.close()
    assert steps == ref.steps == 6
    assert np.linalg.norm(u - ref.u) <= tol * np.linalg.norm(ref.u)
    assert np.linalg.norm(v - ref.v) <= 10 * tol * np.linalg.norm(ref.v)
    P = msx.Pool(max_slots=2, precision=precision, elems_per_block=256)
    t = P.submit(mesh.X, mesh.conn, (msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0), bcs, 6)
    P.wait(t)
    pu, pv, pa = P.fetch(t)
    P.close()
    assert np.array_equal(u, pu) and np.array_equal(v, pv) and np.array_equal(a, pa)


DEFORMATIONS = {
    "rest": lambda x, h: 0 * x,
    "small": lambda x, h: 1e-3 * np.sin(3 * x[[1, 2, 0]]) * x[2],
    "sheared": lambda x, h: np.stack([0.3 * x[2], 0 * x[0], 0 * x[0]]),
    "one node pushed into its elements": lambda x, h: np.where(
        np.arange(x.shape[1]) == np.argmin(((x - 0.5) ** 2).sum(0)), 0.45 * h, 0.0) * np.array([[1.0], [0.3], [-0.2]]),
    "rotated by 90 degrees": lambda x, h: np.stack([-x[1], x[0], x[2]]) - x,
    "moved": lambda x, h: 0 * x + np.array([[40.0], [-7.0], [3.0]]) * h,
    "shrunk": lambda x, h: -0.3 * x,
    "swollen": lambda x, h: 0.4 * x,
}


@pytest.mark.parametrize("jitter", [0.0, 0.1])
@pytest.mark.parametrize("name", list(DEFORMATIONS))
@pytest.mark.parametrize("precision", [msx.FP64, msx.FP64_EXACT, msx.MIXED, msx.DOUBLE_WORD])
def test_time_step_is_the_minimum(name, jitter, precision):
    """The step's dt, found by the gated screen in the element kernel, against the block's first dt, which an FP64
    pass over every element gives: from rest the displacement of both steps is the initial one."""
    n = 7
    X, conn = msx.mesh_cube(n, 9, jitter)
    u = DEFORMATIONS[name](X, 1.0 / n)
    for law in (msx.COMPRESSIBLE_NH, msx.STVK):
        S = msx.Solver(X, conn, [(law, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5, precision=precision)
        S.set_state(u.ravel())
        first, second = S.run(1).dt, S.run(1).dt
        S.close()
        # 60 roundings of FP64, and u's own 2^-48 in the pair-state modes
        tol = 60 * 2.0 ** -53 * 4 + (2.0 ** -46 * np.abs(u).max() * n if precision in (msx.MIXED, msx.DOUBLE_WORD) else 0)
        assert abs(second - first) <= tol * first

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

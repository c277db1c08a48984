"""What a resident solve of a pool counts against its memory budget: no more than
these bytes, whatever the law's element data are, so that a budget that once
held a solve still does; and the pooled solve, whose arrays are fewer than a
handle's, gives the bits of the solve run alone."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu


def bytes_held(nn, ne, nbc, precision, law):
    r = lambda b: (b + 255) & ~255
    pairs = precision != msx.FP64
    b = r(16 * ne) + r(72 * ne) + 2 * r(8 * ne) + r(36 * ne) + 2 * r(4 * ne)   # conn, gradients, weights, lengths
    b += 4 * r(24 * nn) + 2 * r(8 * nn) + r(24 * nn)                           # X, u, v, a, mass and its inverse
    if pairs:
        b += 2 * r(24 * nn) + r(8 * nn)
    if precision == msx.FP64:
        b += r(32 * nn)
        if law == msx.COMPRESSIBLE_NH:
            b += r(72 * ne) + r(48 * ne) + r(8 * ne)
    if precision == msx.DOUBLE_WORD:
        b += r(36 * ne) + r(4 * ne)
    b += r(64 * ne) if precision == msx.MIXED else r(96 * ne)                  # corner forces
    b += r(4 * (nn + 1)) + r(16 * ne) + r(4 * nn) + r(16 * ne)
    k = max(1, min(nn, nbc))
    return b + r(24 * k) + r(8 * k) + r(16 * max(1, nbc))


@pytest.mark.parametrize("precision", [msx.FP64, msx.MIXED, msx.DOUBLE_WORD])
@pytest.mark.parametrize("law", [msx.NEO_HOOKEAN, msx.COMPRESSIBLE_NH, msx.STVK, msx.LINEAR_ELASTIC])
@pytest.mark.parametrize("n", [1, 5, 12])
def test_budget(n, law, precision):
    X, conn = msx.mesh_cube(n, 4, 0.1)
    X = X * np.array([1.0, 1.0, 0.3])[:, None]
    bcs = msx.cube_bcs(n, 0.02, msx.BC_VEL_RAMP, 4)
    mat = (law, 1e6, 0.3, 1000.0)
    budget = bytes_held(X.shape[1], conn.shape[0], len(bcs), precision, law)
    P = msx.Pool(max_slots=4, precision=precision, hbm_budget_bytes=2 * budget, elems_per_block=256)
    tickets = [P.submit(X, conn, mat, bcs, 9) for _ in range(2)]
    assert None not in tickets
    for t in tickets:
        P.wait(t)
    pooled = [P.fetch(t) for t in tickets]
    P.close()
    S = msx.Solver(X, conn, [mat], bcs, 0.0, 1e30, 0.5, max_steps=9, precision=precision)
    S.run()
    alone = S.state()
    S.close()
    for got in pooled:
        for a, b in zip(got, alone):
            assert np.array_equal(a, b)

"""A solver block refused for its boundary conditions has already set its
options: a run after it follows the new end time, scale factor and precision
with the boundary conditions that were there, also when steps of the block
before have been captured."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu

PRECISIONS = [msx.FP64, msx.FP64_EXACT, msx.MIXED, msx.DOUBLE_WORD]


@pytest.mark.parametrize("before", PRECISIONS)
@pytest.mark.parametrize("after", PRECISIONS)
def test_options_of_a_refused_block_hold(before, after):
    n = 6
    X, conn = msx.mesh_cube(n, 3, 0.1)
    bcs = msx.cube_bcs(n, 0.0, msx.BC_INST)   # held: their tables don't depend on a block's times
    u = 1e-3 * np.random.default_rng(1).uniform(-1, 1, X.shape) * X[2]
    mat = [(msx.COMPRESSIBLE_NH, 1e6, 0.3, 1000.0)]

    def start():
        S = msx.Solver(X, conn, mat, bcs, 0.0, 1e30, 0.5, max_steps=12, precision=before, steps_per_graph=4)
        S.set_state(u.ravel())
        S.run(6)
        S.run()   # replays captured chunks
        return S

    S = start()
    dt = S.run().dt
    tf = 7.3 * dt * 0.6
    with pytest.raises(msx.MsxError):
        S.next_solver([(3 * X.shape[1] + 5, msx.BC_INST, 0.0, 0)], 0.0, tf, 0.3, 40, precision=after, steps_per_graph=4)
    got = S.run()
    state = S.state()
    S.close()
    S = start()
    S.next_solver(bcs, 0.0, tf, 0.3, 40, precision=after, steps_per_graph=4)
    want = S.run()
    expected = S.state()
    S.close()
    assert 7 <= want.steps < 40
    assert (got.steps, got.t, got.dt) == (want.steps, want.t, want.dt)
    for a, b in zip(state, expected):
        assert np.array_equal(a, b)

"""The FP64 CFL value of a candidate is the same bits whether four lanes compute
it (few candidates in a tile) or one does (tiles full of them): the time step of
tets that occur once and of the same tets many times over."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [msx.FP64, msx.DOUBLE_WORD])
@pytest.mark.parametrize("copies", [2, 20, 60, 70, 130, 1000])
def test_time_step_bits(precision, copies):
    rng = np.random.default_rng(copies)
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    for _ in range(4):
        tet = ref + rng.uniform(-0.15, 0.15, (4, 3)) + rng.uniform(-2, 2, (1, 3))
        du = 0.05 * rng.uniform(-1, 1, (4, 3))
        dts = []
        for n in (1, copies):
            X = np.ascontiguousarray(np.tile(tet, (n, 1)).T)
            S = msx.Solver(X, np.arange(4 * n, dtype=np.int32).reshape(n, 4), [(msx.STVK, 1e6, 0.3, 1000.0)], [], 0.0, 1e30,
                           0.5, precision=precision)
            S.set_state(np.ascontiguousarray(np.tile(du, (n, 1)).T).ravel())
            S.run(1)
            dts.append(S.run(1).dt)
            S.close()
        assert dts[0] == dts[1] > 0

"""Corner forces of compressible neo-Hookean elements in flat and tall hexes in
the plain FP64 mode, inside the fixed-point form's range and left out of it: the
error is that of rounding F once, some EPS / strain of the forces, whatever the
flatness (the form from the deformed edges loses ten times that in FP64)."""
import numpy as np
import pytest

import msx
import test_gpu_fixed_point as cnh
from test_fixed_point_host import EPS, YOUNG, grid, lame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aspect", [(1, 1, 1), (1, 1, 0.2), (1.05, 2.1, 0.12), (0.08, 0.2, 1.83), (0.3, 2.7, 0.1), (1, 1, 5)])
@pytest.mark.parametrize("jitter", [0.0, 0.1])
def test_error_does_not_grow_with_flatness(aspect, jitter):
    X, conn = grid(4, tuple(0.25 * a for a in aspect), jitter)
    X = np.ascontiguousarray(X[:, conn.ravel()])   # tets apart: nodal forces are corner forces
    conn = np.arange(conn.size, dtype=np.int32).reshape(-1, 4)
    lam, mu2 = lame(0.3)
    S = msx.Solver(X, conn, [(msx.COMPRESSIBLE_NH, YOUNG, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
    rng = np.random.default_rng(3)
    for strain in (1e-2, 1e-4, 1e-6):
        u = strain * 0.3 * 0.25 * min(aspect) * rng.uniform(-1, 1, X.shape)
        f = S.internal_force(u.ravel()).reshape(3, -1).T.reshape(-1, 4, 3)
        want = cnh.reference(X, u, conn, lam, 0.5 * mu2)[0]
        assert float(np.sqrt(((f - want) ** 2).sum() / (want ** 2).sum())) <= 16 * EPS / strain, strain
    S.close()

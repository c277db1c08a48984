"""Corner forces of linear elastic and St-Venant-Kirchhoff elements in the plain
FP64 mode at small strains on unjittered grids, whose precision is relative to
the strain and not to the element."""
import numpy as np
import pytest

import msx
import test_gpu_fixed_stress as svk
from test_fixed_point_host import EPS, MOTIONS, YOUNG, grid, lame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law", [msx.LINEAR_ELASTIC, msx.STVK])
@pytest.mark.parametrize("motion", list(MOTIONS))
def test_error_is_relative_to_the_strain(law, motion):
    X, conn = grid(4, (0.1, 0.1, 0.1), 0.0)
    X = np.ascontiguousarray(X[:, conn.ravel()])   # tets apart: nodal forces are corner forces
    conn = np.arange(conn.size, dtype=np.int32).reshape(-1, 4)
    lam, mu2 = lame(0.3)
    S = msx.Solver(X, conn, [(law, YOUNG, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
    for strain in (1e-3, 1e-5, 1e-7, 1e-9, 1e-12):
        u = strain * (MOTIONS[motion] @ X)
        f = S.internal_force(u).reshape(3, -1).T.reshape(-1, 4, 3)
        want = svk.reference(X, u, conn, law == msx.LINEAR_ELASTIC, lam, mu2)[0]
        # an error of one unit of 2^-55 in each of some ten roundings, and the result's own
        assert float(np.sqrt(((f - want) ** 2).sum() / (want ** 2).sum())) <= 4 * EPS, strain
    S.close()

"""The exact mode against the oracle bit for bit, signs of zeros included, where
sums are made of zeros: a body at rest, motions along one axis, mirrored ones."""
import numpy as np
import pytest

import msx
import oracle as O

pytestmark = pytest.mark.gpu

LAWS = [(msx.NEO_HOOKEAN, O.NEO_HOOKEAN), (msx.COMPRESSIBLE_NH, O.COMPRESSIBLE_NH), (msx.STVK, O.STVK),
        (msx.LINEAR_ELASTIC, O.LINEAR_ELASTIC)]
MOTIONS = {
    "pulled along z": (0.02, msx.BC_VEL_RAMP),
    "pushed along z": (-0.02, msx.BC_VEL_RAMP),
    "held": (0.0, msx.BC_VEL_RAMP),
}


@pytest.mark.parametrize("law", range(4))
@pytest.mark.parametrize("name", list(MOTIONS))
def test_bits(name, law):
    mesh = O.cube_mesh(3)
    top, kind = MOTIONS[name]
    bcs = O.cube_bcs(3, top, kind, 4)
    ref = O.run(mesh, [O.Material(LAWS[law][1])], [O.Solver(0.0, 1e30, 0.5, bcs, max_steps=8)])
    S = msx.Solver(mesh.X, mesh.conn, [(LAWS[law][0], 1e6, 0.3, 1000.0)], bcs, 0.0, 1e30, 0.5, max_steps=8,
                   precision=msx.FP64_EXACT)
    S.run()
    for got, want in zip(S.state(), (ref.u, ref.v, ref.a)):
        if LAWS[law][0] in (msx.STVK, msx.LINEAR_ELASTIC):   # no log or pow of the host's library in them
            assert np.array_equal(got.view(np.int64), np.ascontiguousarray(want).view(np.int64))
        else:
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
    S.close()

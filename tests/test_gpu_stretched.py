"""Corner forces in the plain FP64 mode of elements stretched far beyond the
fixed-point forms' range (they go the FP64 way), through every entry point that
evaluates them: internal_force, run and the pool."""
import numpy as np
import pytest

import msx
import test_gpu_fixed_point as cnh
import test_gpu_fixed_stress as svk
from test_gpu_fixed_point import EPS

pytestmark = pytest.mark.gpu

# displacements of one node in edge lengths, both sides of the range and of multiples of 2^61 of its unit
MOVES = np.array([0.5, 1.9, 3, 8, 15, 16, 17, 31, 32, 33, 48, 63.5, 64, 100, 128, 1000])
LAWS = [msx.COMPRESSIBLE_NH, msx.STVK, msx.LINEAR_ELASTIC]
YOUNG, NU = 1e6, 0.3
LAM, MU2 = YOUNG * NU / ((1 + NU) * (1 - 2 * NU)), YOUNG / (1 + NU)


def mesh():
    """Disjoint unit corner tets; node k % 4 of tet k moves by MOVES along axis (k / 4) % 3, outwards."""
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    n = 12 * len(MOVES)
    X = np.ascontiguousarray(np.tile(ref, (n, 1)).T)
    conn = np.arange(4 * n, dtype=np.int32).reshape(n, 4)
    k = np.arange(n)
    node, axis = 4 * k + k % 4, (k // 4) % 3
    way = np.where(k % 4 == 0, -1.0, 1.0)
    return X, conn, node + axis * X.shape[1], way * MOVES[k // 12]


def check(f, X, u, conn, law):
    u = u.reshape(3, -1)
    f = f.reshape(3, -1).T.reshape(-1, 4, 3)
    if law == msx.COMPRESSIBLE_NH:
        want, scale = cnh.reference(X, u, conn, LAM, 0.5 * MU2)
    else:
        want, scale = svk.reference(X, u, conn, law == msx.LINEAR_ELASTIC, LAM, MU2)
    err = np.abs((f - want).astype(float)).max(-1) / (64 * EPS * scale)
    assert np.isfinite(f).all() and err.max() <= 1.0, err.max()


@pytest.mark.parametrize("law", LAWS)
def test_internal_force(law):
    X, conn, dof, by = mesh()
    u = np.zeros(3 * X.shape[1])
    u[dof] = by
    S = msx.Solver(X, conn, [(law, YOUNG, NU, 1000.0)], [], 0.0, 1e30, 0.5)
    f = S.internal_force(u)
    S.close()
    check(f, X, u, conn, law)


@pytest.mark.parametrize("law", LAWS)
def test_run_and_pool(law):
    X, conn, dof, by = mesh()
    nodes = np.arange(X.shape[1])
    bcs = [(int(d), msx.BC_INST, float(v), 0) for d, v in zip(dof, by)]
    S = msx.Solver(X, conn, [(law, YOUNG, NU, 1000.0)], bcs, 0.0, 1e30, 0.5, max_steps=3)
    S.run(1)
    u = S.state()[0]
    assert np.array_equal(u[dof], by)
    check(np.stack([S.node_values(msx.FIELD_INTERNAL_FORCE, c, nodes) for c in range(3)]), X, u, conn, law)
    S.run()
    state = S.state()
    S.close()
    P = msx.Pool(max_slots=1, precision=msx.FP64, elems_per_block=256)
    t = P.submit(X, conn, (law, YOUNG, NU, 1000.0), bcs, 3)
    P.wait(t)
    pooled = P.fetch(t)
    P.close()
    for a, b in zip(state, pooled):
        assert np.array_equal(a, b)

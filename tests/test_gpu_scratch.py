"""Device memory that the compute-and-copy-out calls of a handle keep: what the
largest of them needed, no more, and given back with the handle."""
import numpy as np
import pytest

import msx

pytestmark = pytest.mark.gpu

MAPPING = 2 << 20   # the device maps memory in pieces of this size


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_a_handle_keeps_what_its_calls_need():
    X, conn = msx.mesh_cube(2)
    S = msx.Solver(X, conn, [(msx.STVK, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)   # the kernels are loaded
    S.internal_force(np.zeros(3 * X.shape[1]))
    S.element_values("VOLUME")
    S.close()
    X, conn = msx.mesh_cube(60, 3, 0.1)
    need = 2 * 24 * X.shape[1]   # displacement in, force out: 10.9 MB
    u = 1e-4 * np.random.default_rng(2).uniform(-1, 1, 3 * X.shape[1])
    whole = free_bytes()
    S = msx.Solver(X, conn, [(msx.STVK, 1e6, 0.3, 1000.0)], [], 0.0, 1e30, 0.5)
    before = free_bytes()
    first = S.internal_force(u)
    assert before - free_bytes() <= need + MAPPING
    assert np.array_equal(first, S.internal_force(u))
    assert S.element_values("VOLUME").shape == (conn.shape[0],)   # 10.4 MB: the same scratch
    assert before - free_bytes() <= need + MAPPING
    S.close()
    assert whole - free_bytes() <= MAPPING

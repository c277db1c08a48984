"""The fixed-point corner forces compiled for the host, at and beyond the ends of
their range: whatever they accept has to be right, against the same formulas in
extended precision."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import test_gpu_fixed_point as cnh
import test_gpu_fixed_stress as svk
from test_gpu_fixed_point import EPS, N, rotation, tets

HERE = os.path.dirname(os.path.abspath(__file__))
YOUNG = 1e6


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed") / "fixed.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    os.path.join(HERE, "fixed_point_host.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def lame(nu):
    return YOUNG * nu / ((1 + nu) * (1 - 2 * nu)), YOUNG / (1 + nu)


def forces(lib, law, X, u, conn, nu):
    """(forces (N, 4, 3), accepted (N,)) of the host build; law: "cnh", "stvk" or "le"."""
    lam, mu2 = lame(nu)
    x, w = np.ascontiguousarray(X.T[conn]), np.ascontiguousarray(u.T[conn])
    f, taken = np.zeros(x.shape), np.zeros(len(x), np.int32)
    n = C.c_longlong(len(x))
    if law == "cnh":
        lib.fixed_cnh(n, _p(x), _p(w), C.c_double(lam), C.c_double(0.5 * mu2), _p(f), _p(taken))
    else:
        lib.fixed_svk(n, _p(x), _p(w), C.c_int(law == "le"), C.c_double(lam), C.c_double(mu2), _p(f), _p(taken))
    return f, taken.astype(bool)


def reference(law, X, u, conn, nu):
    lam, mu2 = lame(nu)
    if law == "cnh":
        return cnh.reference(X, u, conn, lam, 0.5 * mu2)
    return svk.reference(X, u, conn, law == "le", lam, mu2)


def check(lib, law, X, u, conn, nu):
    """How many are accepted; those have to be right to the GPU tests' bound."""
    f, taken = forces(lib, law, X, u, conn, nu)
    with np.errstate(invalid="ignore", divide="ignore"):
        want, scale = reference(law, X, u, conn, nu)
        err = np.abs((f - want).astype(float)).max(-1) / (64 * EPS * scale)
    assert not (~(err[taken] <= 1.0)).any(), (int((~(err[taken] <= 1.0)).any(1).sum()), int(taken.sum()))
    return int(taken.sum())


STRETCHES = [1.5, 2, 4, 8, 12, 16, 18, 20, 24, 28, 31, 32, 33, 63.5, 64, 65, 100, 128, 1000, 1e6, 1e30]


@pytest.mark.parametrize("law", ["cnh", "stvk", "le"])
@pytest.mark.parametrize("along", ["x", "y", "z", "all"])
@pytest.mark.parametrize("sign", [1, -1])
def test_stretches(lib, law, along, sign):
    rng = np.random.default_rng(7)
    X, conn = tets(rng, 1.0, 1.0)
    x = X.T[conn]
    for s in STRETCHES:
        F = np.eye(3)
        for i in range(3) if along == "all" else ["xyz".index(along)]:
            F[i, i] = sign * s
        y = np.einsum("ij,naj->nai", F, x - x[:, :1]) + x[:, :1]
        check(lib, law, X, np.ascontiguousarray((y - x).reshape(4 * N, 3).T), conn, 0.3)


@pytest.mark.parametrize("law", ["cnh", "stvk", "le"])
@pytest.mark.parametrize("component", [0, 1, 2])
@pytest.mark.parametrize("node", [0, 1, 2, 3])
def test_one_node_moved(lib, law, component, node):
    """Unit corner tets, one node of each displaced by just under, at and over multiples of the edge length."""
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    d = np.concatenate([k * np.array([0.97, 1 - 2.0 ** -20, 1, 1 + 2.0 ** -20, 1.03])
                        for k in (1, 2, 4, 8, 15, 16, 31, 32, 33, 48, 63.5, 64, 96, 128, 1000, 2.0 ** 20, 2.0 ** 40)])
    d = np.concatenate([d, -d])
    n = len(d)
    X = np.ascontiguousarray(np.tile(ref, (n, 1)).T)
    conn = np.arange(4 * n, dtype=np.int32).reshape(n, 4)
    u = np.zeros((3, 4 * n))
    u[component, node::4] = d
    check(lib, law, X, u, conn, 0.3)


@pytest.mark.parametrize("law", ["cnh", "stvk", "le"])
def test_graded_edges(lib, law):
    """Tets whose three edges differ by up to 1:12, stretched along each axis."""
    rng = np.random.default_rng(11)
    for grade in ([1, 1, 12], [1, 5, 12], [12, 1, 3]):
        X, conn = tets(rng, 1.0, 1.0)
        X = X * np.array(grade, float)[:, None]
        x = X.T[conn]
        for s in (1.01, 1.7, 2.5, 9, 17, 33, 65):
            for i in range(3):
                F = np.eye(3)
                F[i, i] = s
                y = np.einsum("ij,naj->nai", F, x - x[:, :1]) + x[:, :1]
                check(lib, law, X, np.ascontiguousarray((y - x).reshape(4 * N, 3).T), conn, 0.3)


# ------------------------------------------------------------------ accuracy against the FP64 forms
SPLIT = np.array([(1, 3, 4, 7), (1, 2, 3, 7), (4, 1, 7, 8), (1, 5, 7, 8), (1, 5, 6, 7), (2, 1, 6, 7)]) - 1
CORNER = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)])
SHEAR = np.zeros((3, 3))
SHEAR[0, 2] = 1
MOTIONS = {
    "simple shear": SHEAR,
    "pure shear": SHEAR + SHEAR.T,
    "shears in three planes": np.array([[0, 1, 0.3], [0.2, 0, -0.7], [0.5, 0.4, 0]]),
    "pulled": np.diag([-0.3, -0.3, 1]),
    "swollen": np.eye(3),
    "general": np.array([[0.3, 1, 0.3], [0.2, -0.4, -0.7], [0.5, 0.4, 0.6]]),
}


def grid(n, h, jitter):
    """n^3 hexes of sides h, six tets each, nodes jittered by `jitter` h; X (3, nn), conn."""
    rng = np.random.default_rng(1)
    at = np.stack(np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    X = at * np.array(h) + jitter * np.array(h) * rng.uniform(-1, 1, at.shape)
    cell = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 1, 1, 3) + CORNER[SPLIT][None]
    conn = ((cell[..., 0] * (n + 1) + cell[..., 1]) * (n + 1) + cell[..., 2]).reshape(-1, 4)
    return np.ascontiguousarray(X.T), conn.astype(np.int32)


def forces_fp64(lib, law, X, u, conn, nu):
    lam, mu2 = lame(nu)
    x, w = np.ascontiguousarray(X.T[conn]), np.ascontiguousarray(u.T[conn])
    f, n = np.zeros(x.shape), C.c_longlong(len(x))
    if law == "cnh":
        lib.fp64_cnh(n, _p(x), _p(w), C.c_double(lam), C.c_double(0.5 * mu2), _p(f))
    else:
        lib.fp64_svk(n, _p(x), _p(w), C.c_int(law == "le"), C.c_double(lam), C.c_double(mu2), _p(f))
    return f


def rms_errors(lib, law, h, jitter, motion, strain, nu):
    """Root mean squares of the fixed-point and of the FP64 form's corner-force errors over that of the forces."""
    X, conn = grid(4, h, jitter)
    u = strain * (MOTIONS[motion] @ X)
    f, taken = forces(lib, law, X, u, conn, nu)
    assert taken.all()
    want = reference(law, X, u, conn, nu)[0]
    rms = lambda e: float(np.sqrt((e ** 2).sum() / (want ** 2).sum()))
    return rms(f - want), rms(forces_fp64(lib, law, X, u, conn, nu) - want)


@pytest.mark.parametrize("motion", list(MOTIONS))
@pytest.mark.parametrize("h,jitter", [((0.1,) * 3, 0.0), ((0.1,) * 3, 0.1), ((0.125,) * 3, 0.0), ((0.1, 0.1, 0.3), 0.0),
                                      ((0.1, 0.1, 0.04), 0.0), ((0.1, 0.1, 0.02), 0.0), ((0.1, 0.1, 0.02), 0.1),
                                      ((0.1, 0.1, 1.0), 0.0)])
@pytest.mark.parametrize("law", ["le", "stvk"])
def test_no_less_accurate_than_fp64(lib, law, h, jitter, motion):
    """At or below the FP64 form's error at every strain, or below two roundings of the result (where the FP64 form's
    own products happen to be exact); twice its error at strains whose roundings both forms share (0.1)."""
    for nu in (0.0, 0.3, 0.49):
        for strain in (0.1, 1e-2, 1e-3, 1e-5, 1e-7, 1e-9, 1e-12):
            ours, theirs = rms_errors(lib, law, h, jitter, motion, strain, nu)
            assert ours <= max((2 if strain > 0.05 else 1) * theirs, 2 * EPS), (nu, strain, ours, theirs)


@pytest.mark.parametrize("motion", list(MOTIONS))
def test_no_less_accurate_than_fp64_cnh(lib, motion):
    for nu in (0.0, 0.3, 0.49):
        for strain in (1e-2, 1e-3, 1e-5, 1e-7, 1e-9):
            ours, theirs = rms_errors(lib, "cnh", (0.1,) * 3, 0.1, motion, strain, nu)
            assert ours <= max(theirs, 2 * EPS), (nu, strain, ours, theirs)


def test_integer_to_fp64(lib):
    lib.to_fp64.restype = C.c_double
    rng = np.random.default_rng(6)
    for bits in range(1, 64):
        for x in rng.integers(2 ** (bits - 1), 2 ** bits - 1, 50, dtype=np.int64, endpoint=True).tolist() + [2 ** bits - 1, 1 - 2 ** bits]:
            for k in (0, -57, 400, -900):
                got = lib.to_fp64(C.c_longlong(x), C.c_int(k))
                want = float(x) * 2.0 ** k   # float(): nearest, halves to even
                assert got == want or abs(got - want) <= 2.0 ** (bits - 53 + k) and (x >> max(bits - 54, 0)) & 1
    assert lib.to_fp64(C.c_longlong(0), C.c_int(5)) == 0.0

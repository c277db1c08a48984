"""The work a user of this library has it do, as cases that can be timed and checked.

The library advances explicit solid-mechanics solves on linear-tet meshes.  A
program that uses it does one of a few things, over and over: it advances a
resident solve by the steps between two outputs and reads the state back
("step"); it hands a whole job over and takes the result ("job"); it has many
small solves advanced together ("pool"); it asks for the internal force of a
displacement field ("force"); or it takes a step at a time and writes rows of
extracted quantities after each ("extract").

listed() names one case for each of them at the sizes the repository's
configurations and tests use (unit cubes of 2 to 100 hexes a side, six tets a
hex), in the four precision modes and the four laws, draw() gives others of the
same ranges, prepare() makes what the program has in hand (mesh, state, handle),
run() is one pass through the public API, exact() the same result in plain FP64
torch.  Meshes are boxes of hexes split into six tets, interior nodes jittered
by 0.1 h, numbered hex by hex or (as a mesher leaves them) in shuffled order.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "v.1.1_gb300"))
import msx  # noqa: E402

MODES = {"fp64": msx.FP64, "exact": msx.FP64_EXACT, "mixed": msx.MIXED, "dword": msx.DOUBLE_WORD}
LAWS = {"nh": msx.NEO_HOOKEAN, "cnh": msx.COMPRESSIBLE_NH, "stvk": msx.STVK, "le": msx.LINEAR_ELASTIC}
SCALE = 0.5            # dt = 0.5 CFL, as in every configuration
RAMP_STEPS = 200       # steps over which the top face's velocity is ramped
T_END = 1e30           # passes are bounded by steps, not by time
YOUNG, NU, RHO = 1e6, 0.3, 1000.0
PRESSURE, GRAVITY = 2e3, 9.81   # Pa on the top face, m/s^2


def _case(name, kind, mode, law, nx, ny, nz, steps, **more):
    c = {"name": name, "kind": kind, "mode": mode, "law": law, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
         "loads": False, "two_materials": False, "shuffled": False}
    c.update(more)
    return c


def listed():
    return [
        # the large configuration: 6M tets, plain FP64, compressible neo-Hookean, advanced between two read-backs
        _case("step_fp64_cnh_100", "step", "fp64", "cnh", 100, 100, 100, 20),
        # the same mesh in mixed precision, the precision study's workload
        _case("step_mixed_cnh_100", "step", "mixed", "cnh", 100, 100, 100, 20),
        # a mid-size solve wanted to 1e-12 but faster than FP64
        _case("step_dword_cnh_64", "step", "dword", "cnh", 64, 64, 64, 20),
        # a run that has to repeat the reference's operation order; St-Venant-Kirchhoff gives its bits
        _case("step_exact_stvk_40", "step", "exact", "stvk", 40, 40, 40, 20),
        # a ragged part as a mesher numbers it, under gravity and a follower pressure on its top
        _case("step_fp64_stvk_loads", "step", "fp64", "stvk", 37, 41, 29, 50, loads=True, shuffled=True),
        # two materials in one part, mixed precision, Belytschko neo-Hookean
        _case("step_mixed_nh_2mat", "step", "mixed", "nh", 23, 31, 27, 100, two_materials=True),
        # the small configuration: the 6000-tet cube, many steps of little work each
        _case("step_fp64_cnh_10", "step", "fp64", "cnh", 10, 10, 10, 200),
        # the smallest meshes users start with (a few dozen tets): latency alone
        _case("step_mixed_cnh_2", "step", "mixed", "cnh", 2, 2, 3, 200),
        # the batched configuration: independent cubes of log-uniform side in [8, 48], mixed precision, advanced
        # together from rest and fetched
        _case("pool_mixed", "pool", "mixed", "cnh", 8, 48, 24, 64),
        # one internal-force evaluation of a host displacement field (a caller's own integrator, a residual check)
        _case("force_fp64_cnh_33", "force", "fp64", "cnh", 33, 33, 33, 1),
        # a whole job from host buffers: mesh upload, set-up, a run, read-back, release
        _case("job_fp64_cnh_56", "job", "fp64", "cnh", 56, 56, 56, 20),
        # output rows every step, as a deck with *EXTRACTION blocks asks for
        _case("extract_fp64_cnh_20", "extract", "fp64", "cnh", 20, 20, 20, 1),
    ]


def draw(rng):
    def side(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))

    kind = rng.choice(["step"] * 7 + ["pool", "force", "job", "extract"])
    if kind == "pool":   # nx, ny: smallest and largest side; nz: number of solves
        return {"kind": "pool", "mode": rng.choice(["mixed", "mixed", "dword", "fp64"]), "law": "cnh", "nx": 8,
                "ny": rng.randint(20, 48), "nz": rng.randint(6, 24), "steps": rng.randint(16, 64), "loads": False,
                "two_materials": False, "shuffled": False}
    mode = rng.choice(["fp64", "fp64", "mixed", "mixed", "dword", "exact"])
    if kind in ("force", "job"):
        nx, ny, nz, steps = side(8, 48), side(8, 48), side(8, 48), rng.randint(5, 30) if kind == "job" else 1
    elif kind == "extract":
        nx, ny, nz, steps = side(4, 30), side(4, 30), side(4, 30), 1
    else:
        base = side(2, 64 if mode == "exact" else 92)   # sides around one size, so meshes of all sizes come up
        nx, ny, nz = (max(1, int(base * rng.uniform(0.7, 1.05))) for _ in range(3))
        cost = 6 * nx * ny * nz * {"fp64": 1.0, "mixed": 0.25, "dword": 0.45, "exact": 3.5}[mode]
        steps = max(10, min(rng.choice([20, 50, 100, 200]), int(8e7 / cost)))
    return {"kind": kind, "mode": mode, "law": rng.choice(["cnh", "cnh", "nh", "stvk", "le"]), "nx": nx, "ny": ny,
            "nz": nz, "steps": steps, "loads": kind == "step" and rng.random() < 0.25,
            "two_materials": kind != "pool" and rng.random() < 0.25, "shuffled": rng.random() < 0.3}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _mesh(nx, ny, nz, g, shuffled):
    """Node coordinates (3, nn) and tets (ne, 4) of the box [0, nx h] x [0, ny h] x [0, nz h], h = 1 / max side;
    the bottom (z = 0) and top nodes; on the GPU."""
    d = torch.device("cuda")
    h = 1.0 / max(nx, ny, nz)
    K, J, I = torch.meshgrid(torch.arange(nz + 1, device=d), torch.arange(ny + 1, device=d),
                             torch.arange(nx + 1, device=d), indexing="ij")
    i, j, k = I.reshape(-1), J.reshape(-1), K.reshape(-1)
    X = torch.stack([i, j, k]).double() * h
    inner = (i > 0) & (i < nx) & (j > 0) & (j < ny) & (k > 0) & (k < nz)
    X += (2 * torch.rand(X.shape, generator=g, device=d, dtype=torch.float64) - 1) * (0.1 * h) * inner
    m, mm = nx + 1, (nx + 1) * (ny + 1)
    base = (i + m * j + mm * k)[(i < nx) & (j < ny) & (k < nz)]
    corner = [None, 0, 1, 1 + m, m, mm, mm + 1, mm + 1 + m, mm + m]
    split = [(1, 3, 4, 7), (1, 2, 3, 7), (4, 1, 7, 8), (1, 5, 7, 8), (1, 5, 6, 7), (2, 1, 6, 7)]
    conn = torch.stack([torch.stack([base + corner[c] for c in t], 1) for t in split], 1).reshape(-1, 4)
    bottom, top = (k == 0).nonzero().reshape(-1), (k == nz).nonzero().reshape(-1)
    if shuffled:
        p = torch.randperm(X.shape[1], generator=g, device=d)   # node n becomes p[n]
        Y = torch.empty_like(X)
        Y[:, p] = X
        X, conn, bottom, top = Y, p[conn], p[bottom], p[top]
        conn = conn[torch.randperm(conn.shape[0], generator=g, device=d)]
    return X.contiguous(), conn.contiguous(), bottom.sort()[0], top.sort()[0], h


def _materials(case):
    mats = [(LAWS[case["law"]], YOUNG, NU, RHO)]
    if case["two_materials"]:
        mats.append((msx.COMPRESSIBLE_NH if case["law"] != "cnh" else msx.STVK, 2.5 * YOUNG, 0.4, 1.2 * RHO))
    return mats


def _field(X, g, amplitude, h):
    """A smooth vector field (3, nn), zero on the bottom: four low modes a component, gradients of order `amplitude`."""
    d, out = X.device, torch.zeros_like(X)
    for c in range(3):
        for _ in range(4):
            k = torch.randint(1, 4, (3,), generator=g, device=d).double() * math.pi
            phase = torch.rand(1, generator=g, device=d, dtype=torch.float64) * 2 * math.pi
            out[c] += torch.sin((k[:, None] * X).sum(0) + phase) / k.norm()
    return out * X[2] * (amplitude / 2)


def _sound(mats):
    return max(math.sqrt(E / rho) if law >= 2 else math.sqrt(E * (1 - nu) / ((1 + nu) * (1 - 2 * nu)) / rho)
               for law, E, nu, rho in mats)


def _inputs(case, seed):
    """Everything that the seed decides, on the GPU: mesh, materials, initial state, driven velocity."""
    g = _generator(seed)
    X, conn, bottom, top, h = _mesh(case["nx"], case["ny"], case["nz"], g, case["shuffled"])
    mats = _materials(case)
    mat = None
    if len(mats) == 2:   # the upper half is the second material
        mat = (X[2][conn].mean(1) > 0.5 * case["nz"] * h).to(torch.int32)
    amp = 2e-3 * float(torch.rand(1, generator=g, device="cuda") + 0.5)
    u = _field(X, g, amp, h)
    v = _field(X, g, amp, h) * _sound(mats)
    v_top = 0.0
    if case["kind"] == "job":   # from rest, driven
        u, v, v_top = None, None, 0.1 * (0.5 + float(torch.rand(1, generator=g, device="cuda")))
    elif not case["loads"]:
        # a drive so slow that the part may be advanced for as long as the process lives
        v_top = 1e-7 * (0.5 + float(torch.rand(1, generator=g, device="cuda")))
        for w in (u, v):
            w[2] *= 1 - X[2] / (case["nz"] * h)   # nothing on the driven DOFs
            w[2][top] = 0.0
    return {"X": X, "conn": conn, "bottom": bottom, "top": top, "h": h, "mats": mats, "mat": mat, "u": u, "v": v,
            "v_top": v_top, "g": g}


def _bcs(p, driven):
    nn = p["X"].shape[1]
    b, t = p["bottom"].cpu().numpy(), p["top"].cpu().numpy()
    dof = np.concatenate([b, b + nn, b + 2 * nn] + ([t + 2 * nn] if driven else []))
    held = 3 * len(b)
    rows = np.zeros(len(dof), dtype=msx.bc_array([]).dtype)
    rows["dof"] = dof
    rows["mode"] = msx.BC_RAMP
    rows["mode"][held:] = msx.BC_VEL_RAMP
    rows["ramp_steps"][held:] = RAMP_STEPS
    rows["value"][held:] = p["v_top"]
    return rows


def _top_faces(p):
    """{S: tets whose face S (1..4, the reference's numbering) lies in the top plane}."""
    is_top = torch.zeros(p["X"].shape[1], dtype=torch.bool, device="cuda")
    is_top[p["top"]] = True
    on = is_top[p["conn"]]
    return {S: on[:, list(f)].all(1).nonzero().reshape(-1) for S, f in _FACES.items()}


_FACES = {1: (0, 1, 2), 2: (0, 3, 1), 3: (1, 3, 2), 4: (0, 2, 3)}


def _pinned(shape, dtype):
    """A page-locked host array, as a program that moves data every pass keeps."""
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _host(t, dtype):
    a = _pinned(tuple(t.shape), dtype)
    a[...] = t.cpu().numpy()
    return a


def prepare(case, seed):
    if case["kind"] == "pool":
        return _prepare_pool(case, seed)
    p = _inputs(case, seed)
    nn = p["X"].shape[1]
    s = {"kind": case["kind"], "steps": case["steps"], "mats": p["mats"], "mode": MODES[case["mode"]],
         "X": _host(p["X"], torch.float64), "conn": _host(p["conn"], torch.int32),
         "mat": None if p["mat"] is None else p["mat"].cpu().numpy(),
         "bcs": _bcs(p, not case["loads"]),
         "out": tuple(_pinned((3 * nn,), torch.float64) for _ in range(3))}
    if case["kind"] == "job":
        return s
    S = msx.Solver(s["X"], s["conn"], s["mats"], s["bcs"], 0.0, T_END, SCALE, precision=s["mode"],
                   elem_material=s["mat"])
    s["solver"] = S
    if case["kind"] == "force":
        s["u"] = _host(p["u"].reshape(-1), torch.float64)
        return s
    if case["loads"]:
        S.set_load_blocks([("gravity", GRAVITY)] +
                          [("pressure_inst", 0.0, T_END, -PRESSURE, k, e.cpu().numpy())
                           for k, e in _top_faces(p).items() if len(e)])
    S.set_state(_host(p["u"].reshape(-1), torch.float64), _host(p["v"].reshape(-1), torch.float64))
    if case["kind"] == "extract":
        s["top"], s["bottom"] = p["top"].cpu().numpy(), p["bottom"].cpu().numpy()
    return s


def _pool_solves(case, seed):
    """The batch: [(inputs, material)], sides log-uniform in [nx, ny], parameters as in the batched configuration."""
    r = random.Random(int(seed) * 101 + 3)
    rs = random.Random(1000003 * case["ny"] + 101 * case["nz"] + case["steps"])   # the sizes are the case's, not the seed's
    out = []
    for k in range(case["nz"]):
        n = int(round(math.exp(rs.uniform(math.log(case["nx"]), math.log(case["ny"])))))
        g = _generator(int(seed) * 1009 + k)
        X, conn, bottom, top, h = _mesh(n, n, n, g, False)
        mat = (LAWS[case["law"]], math.exp(r.uniform(math.log(1e5), math.log(1e7))), r.uniform(0.25, 0.45), RHO)
        out.append({"X": X, "conn": conn, "bottom": bottom, "top": top, "h": h, "mats": [mat], "mat": None, "u": None,
                    "v": None, "v_top": r.uniform(0.01, 0.2)})
    return out


def _prepare_pool(case, seed):
    solves = _pool_solves(case, seed)
    s = {"kind": "pool", "steps": case["steps"], "pool": msx.Pool(max_slots=64, precision=MODES[case["mode"]]),
         "solves": []}
    total = sum(3 * p["X"].shape[1] for p in solves)
    s["out"] = tuple(_pinned((total,), torch.float64) for _ in range(3))
    at = 0
    for p in solves:
        n3 = 3 * p["X"].shape[1]
        s["solves"].append({"X": _host(p["X"], torch.float64), "conn": _host(p["conn"], torch.int32),
                            "mat": p["mats"][0], "bcs": _bcs(p, True),
                            "out": tuple(o[at:at + n3] for o in s["out"])})
        at += n3
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "step":
        s["solver"].run(s["steps"])
        return list(s["solver"].state(s["out"]))
    if kind == "job":
        S = msx.Solver(s["X"], s["conn"], s["mats"], s["bcs"], 0.0, T_END, SCALE, precision=s["mode"],
                       elem_material=s["mat"])
        S.run(s["steps"])
        out = list(S.state(s["out"]))
        S.close()
        return out
    if kind == "force":
        return [s["solver"].internal_force(s["u"])]
    if kind == "extract":
        S = s["solver"]
        S.run(1)
        return {"svm_mean": S.element_reduce("SVM", "Mean"), "pzz_max": S.element_reduce("PZZ", "Max"),
                "kinetic": S.element_reduce("KIN_ENERGY", "Sum"), "volume": S.element_reduce("VOLUME", "Sum"),
                "top_z": S.node_values(msx.FIELD_DISPLACEMENT, 2, s["top"]),
                "reaction_z": S.node_values(msx.FIELD_INTERNAL_FORCE, 2, s["bottom"])}
    P = s["pool"]
    tickets = [P.submit(q["X"], q["conn"], q["mat"], q["bcs"], s["steps"], tf=T_END, scale_factor=SCALE)
               for q in s["solves"]]
    for t, q in zip(tickets, s["solves"]):
        P.wait(t)
        P.fetch(t, q["out"])
    return list(s["out"])


# ------------------------------------------------------------------ what a pass cannot do without
# Per element and step: connectivity 16 B, shape-function gradients, quadrature weight and reference length in the
# mode's width; per node: X, u, v, a and the mass read, u, v, a written.
ELEMENT_BYTES = {"fp64": 16 + 72 + 8 + 8, "exact": 16 + 72 + 8 + 8, "mixed": 16 + 36 + 4 + 4, "dword": 16 + 72 + 8 + 4}
NODE_BYTES = {"fp64": 24 + 72 + 8 + 72, "exact": 24 + 72 + 8 + 72, "mixed": 24 + 60 + 8 + 60, "dword": 24 + 72 + 8 + 72}
ELEMENT_FLOPS = 250   # edges, F, the law, B^T P and the inscribed sphere, counted as the law's plain algebra


def _sizes(nx, ny, nz):
    return 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)


def work(case):
    if case["kind"] == "pool":
        b = f = 0
        rs = random.Random(1000003 * case["ny"] + 101 * case["nz"] + case["steps"])
        for _ in range(case["nz"]):
            n = int(round(math.exp(rs.uniform(math.log(case["nx"]), math.log(case["ny"])))))
            ne, nn = _sizes(n, n, n)
            b += case["steps"] * (ne * ELEMENT_BYTES[case["mode"]] + nn * NODE_BYTES[case["mode"]]) + 16 * ne + 96 * nn
            f += case["steps"] * ne * ELEMENT_FLOPS
        return {"bytes": b, "flops": f}
    ne, nn = _sizes(case["nx"], case["ny"], case["nz"])
    eb, nb = ELEMENT_BYTES[case["mode"]], NODE_BYTES[case["mode"]]
    if case["kind"] == "force":
        return {"bytes": ne * (eb - 8) + nn * 48, "flops": ne * ELEMENT_FLOPS}
    b, f = case["steps"] * (ne * eb + nn * nb), case["steps"] * ne * ELEMENT_FLOPS
    if case["kind"] == "extract":
        b, f = b + 4 * ne * (eb - 8), f + 4 * ne * ELEMENT_FLOPS
    elif case["kind"] == "job":   # the mesh in, the element data and the state out
        b += ne * (16 + eb) + nn * (24 + 72)
    else:
        b += 72 * nn
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ the same in plain FP64 torch
WEIGHT = 0.166666666667   # the one-point rule's weight as the method defines it


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


class _Model:
    """One part in FP64: the element data and the operations of an explicit step on it."""

    def __init__(self, p):
        self.X, self.conn = p["X"], p["conn"].long()
        self.nn, self.ne = self.X.shape[1], self.conn.shape[0]
        x = self.X[:, self.conn]                      # (3, ne, 4)
        e = [x[:, :, b] - x[:, :, 0] for b in (1, 2, 3)]
        det = (e[0] * _cross(e[1], e[2])).sum(0)
        # rows of the inverse of [e1 e2 e3] are the gradients of shape functions 1..3
        self.g = torch.stack([_cross(e[1], e[2]), _cross(e[2], e[0]), _cross(e[0], e[1])]) / det
        self.wJ = WEIGHT * det.abs()
        ids = torch.zeros(self.ne, dtype=torch.long, device="cuda") if p["mat"] is None else p["mat"].long()

        def per(f):
            return torch.tensor([f(*m) for m in p["mats"]], dtype=torch.float64, device="cuda")[ids]

        self.law = torch.tensor([m[0] for m in p["mats"]], device="cuda")[ids]
        self.laws = sorted({m[0] for m in p["mats"]})
        self.lam = per(lambda l, E, nu, r: E * nu / ((1 + nu) * (1 - 2 * nu)))
        self.mu = per(lambda l, E, nu, r: 0.5 * E / (1 + nu))
        self.bulk = per(lambda l, E, nu, r: E / (3 * (1 - 2 * nu)))
        self.rho = per(lambda l, E, nu, r: r)
        self.c = per(lambda l, E, nu, r: math.sqrt(E / r) if l >= 2
                     else math.sqrt((E * nu / ((1 + nu) * (1 - 2 * nu)) + E / (1 + nu)) / r))
        self.Lref = self.length(torch.zeros_like(self.X))
        self.mass = torch.zeros(self.nn, dtype=torch.float64, device="cuda")
        for a in range(4):
            self.mass.index_add_(0, self.conn[:, a], 0.25 * self.rho * self.wJ)

    def length(self, u):
        """Diameter of the inscribed sphere of every tet of X + u."""
        x = (self.X + u)[:, self.conn]
        p = [x[:, :, a] for a in range(4)]

        def area(a, b, c):
            return 0.5 * _cross(a - c, b - c).square().sum(0).sqrt()

        A = area(p[0], p[1], p[2]) + area(p[1], p[2], p[3]) + area(p[0], p[2], p[3]) + area(p[0], p[1], p[3])
        D = ((p[1] - p[0]) * _cross(p[2] - p[0], p[3] - p[0])).sum(0).abs()
        return D / A

    def cfl(self, u):
        return float((torch.minimum(self.length(u), self.Lref) / self.c).min())

    def H(self, u):
        du = u[:, self.conn]
        return torch.stack([torch.stack([sum((du[i, :, a + 1] - du[i, :, 0]) * self.g[a, j] for a in range(3))
                                         for j in range(3)]) for i in range(3)])   # (3, 3, ne)

    def kinematics(self, u):
        H = self.H(u)
        t = H[0, 0] + H[1, 1] + H[2, 2]
        I2 = (H[0, 0] * H[1, 1] - H[0, 1] * H[1, 0] + H[1, 1] * H[2, 2] - H[1, 2] * H[2, 1] +
              H[0, 0] * H[2, 2] - H[0, 2] * H[2, 0])
        I3 = (H[0, 0] * (H[1, 1] * H[2, 2] - H[1, 2] * H[2, 1]) - H[0, 1] * (H[1, 0] * H[2, 2] - H[1, 2] * H[2, 0]) +
              H[0, 2] * (H[1, 0] * H[2, 1] - H[1, 1] * H[2, 0]))
        return H, t, I2, t + (I2 + I3)

    def piola(self, u):
        """First Piola stress (3, 3, ne), through H = F - I."""
        H, t, I2, Jm1 = self.kinematics(u)
        J, lnJ = 1 + Jm1, torch.log1p(Jm1)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None]
        HT = H.transpose(0, 1)
        P = torch.zeros_like(H)
        for law in self.laws:
            if law == msx.LINEAR_ELASTIC:
                Q = self.mu * (H + HT) + eye * (self.lam * t)
            elif law == msx.STVK:
                E = 0.5 * (H + HT + torch.einsum("kie,kje->ije", H, H))
                S = 2 * self.mu * E + eye * (self.lam * (E[0, 0] + E[1, 1] + E[2, 2]))
                Q = S + torch.einsum("ike,kje->ije", H, S)
            else:
                D = eye * (t + I2) - (1 + t) * HT + torch.einsum("jke,kie->ije", H, H)   # cof(F) - I
                if law == msx.COMPRESSIBLE_NH:
                    Q = (self.mu * (Jm1 * eye + J * H - D) + self.lam * lnJ * (eye + D)) / J
                else:
                    beta = (2 * t + H.square().sum((0, 1))) / 3
                    Q = (self.mu * torch.exp(-2 / 3 * lnJ) / J * ((Jm1 - beta) * eye + J * H - (1 + beta) * D) +
                         self.bulk * Jm1 * (eye + D))
            P = torch.where(self.law == law, Q, P)
        return P

    def internal_force(self, u):
        P = self.piola(u) * self.wJ
        f = torch.zeros_like(u)
        f0 = 0
        for a in range(3):
            fa = torch.stack([(P[i] * self.g[a]).sum(0) for i in range(3)])
            f0 = f0 - fa
            f.index_add_(1, self.conn[:, a + 1], fa)
        f.index_add_(1, self.conn[:, 0], f0)
        return f

    def gravity(self):
        f = torch.zeros_like(self.X)
        for a in range(4):
            f[2].index_add_(0, self.conn[:, a], -0.25 * GRAVITY * self.rho * self.wJ)
        return f

    def pressure(self, u, faces):
        """Follower pressure on faces {S: tets}: area phi J P F^-T n0 on the face's nodes."""
        f = torch.zeros_like(self.X)
        F = self.H(u) + torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None]
        for S, tets in faces.items():
            if not len(tets):
                continue
            nodes = self.conn[tets][:, list(_FACES[S])]
            x = self.X[:, nodes]
            n0 = 0.5 * _cross(x[:, :, 1] - x[:, :, 0], x[:, :, 2] - x[:, :, 0])   # area * normal
            Ft = F[:, :, tets]
            cof = torch.stack([_cross(Ft[1], Ft[2]), _cross(Ft[2], Ft[0]), _cross(Ft[0], Ft[1])])   # J F^-T
            force = -PRESSURE * torch.einsum("ije,je->ie", cof, n0) / 3
            for a in range(3):
                f.index_add_(1, nodes[:, a], force)
        return f


def _simulate(p, steps, driven, faces=None):
    """`steps` steps of the central-difference scheme: dt = 0.5 CFL of the displacement before the step, prediction,
    Dirichlet values, internal force, a = f / m, v += dt/2 (a_old + a)."""
    M = _Model(p)
    u = torch.zeros_like(M.X) if p["u"] is None else p["u"].clone()
    v = torch.zeros_like(M.X) if p["v"] is None else p["v"].clone()
    a = torch.zeros_like(M.X)
    fixed = torch.zeros_like(M.X, dtype=torch.bool)
    fixed[:, p["bottom"]] = True
    if driven:
        fixed[2, p["top"]] = True
    grav = M.gravity() if faces is not None else None
    for step in range(1, steps + 1):
        dt = SCALE * M.cfl(u)
        u1 = u + dt * v + (0.5 * dt * dt) * a
        inc = torch.zeros_like(u)
        if driven:
            inc[2, p["top"]] = p["v_top"] * (step / RAMP_STEPS if step < RAMP_STEPS else 1.0) * dt
        u = torch.where(fixed, u + inc, u1)
        v = torch.where(fixed, inc, v)
        a = torch.where(fixed, torch.zeros_like(a), a)
        f = -M.internal_force(u)
        if faces is not None:
            f = f + (grav + M.pressure(u, faces))
        a1 = f / M.mass
        v = torch.where(fixed, v, v + (0.5 * dt) * (a + a1))
        a = torch.where(fixed, a, a1)
    return M, u, v, a


def exact(case, seed):
    if case["kind"] == "pool":
        got = [[x.reshape(-1) for x in _simulate(p, case["steps"], True)[1:]] for p in _pool_solves(case, seed)]
        return [torch.cat([r[k] for r in got]) for k in range(3)]
    p = _inputs(case, seed)
    if case["kind"] == "force":
        return [_Model(p).internal_force(p["u"]).reshape(-1)]
    faces = _top_faces(p) if case["loads"] else None
    M, u, v, a = _simulate(p, case["steps"], not case["loads"], faces)
    if case["kind"] != "extract":
        return [u.reshape(-1), v.reshape(-1), a.reshape(-1)]
    P = M.piola(u)
    F = M.H(u) + torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None]
    J = 1 + M.kinematics(u)[3]
    s = torch.einsum("ike,jke->ije", P, F) / J
    svm = (0.5 * ((s[0, 0] - s[1, 1]) ** 2 + (s[1, 1] - s[2, 2]) ** 2 + (s[2, 2] - s[0, 0]) ** 2 +
                  6 * (s[0, 1] ** 2 + s[0, 2] ** 2 + s[1, 2] ** 2))).sqrt()
    vc = v[:, M.conn].mean(2)
    return {"svm_mean": float((svm * M.wJ).sum() / M.wJ.sum()), "pzz_max": float(P[2, 2].max()),
            "kinetic": float((0.5 * M.rho * vc.square().sum(0) * M.wJ).sum()), "volume": float((M.wJ * J).sum()),
            "top_z": u[2][p["top"]], "reaction_z": M.internal_force(u)[2][p["bottom"]]}

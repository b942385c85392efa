"""Performance cases of the solver: what users of this framework run.

Every case is one simulation job through the public batch, seam or serving
entry points (fedem_gb300.batch): models set up from their solver-input text,
uploaded, advanced through a number of implicit HHT-alpha time steps and their
triad position matrices read back.  The models are the generators' own: beam
chains (the batched and served workloads and the cantilever), the space-frame
tower with joints, springs and dampers, and the chain of reduced parts.

kinds:
  chain   a batch of beam chains with log-uniform element counts, run to its
          end time from the initial state
  driven  the same, advanced one time step at a time with the positions read
          after each (co-simulation)
  frame   the space-frame tower, run to its end time
  parts   the chain of Craig-Bampton reduced blocks, run to its end time
  seam    one model's Newton matrix assembled, factored and solved for several
          right-hand sides (a host that drives its own Newton loop)
  served  a burst of requests through the continuous-batching server
"""
import math
import os
import re
import sys
import tempfile

import numpy as np

sys.path.insert(0, os.path.join(os.getcwd(), "fedem-solvers_gb300"))

from fedem_gb300 import models  # noqa: E402
from fedem_gb300.batch import Batch, Server, create_models  # noqa: E402

DT = 1.0e-3
SEAM_SCALES = (3.3e6, 1.8e3, 0.9)  # sM, sC, sK of an HHT-alpha step of 1 ms (alpha -0.1)


def listed():
    return [
        # the smallest call: the 20-beam cantilever driven step by step by a co-simulation
        {"name": "cantilever_driven_fp64", "kind": "driven", "models": 1, "n_min": 20, "n_max": 20, "steps": 8,
         "mixed": False},
        # the plain path on the cantilever's size: one model, FP64, to its end time
        {"name": "cantilever_fp64", "kind": "chain", "models": 1, "n_min": 20, "n_max": 20, "steps": 60,
         "mixed": False},
        # one long chain alone (the largest model of the batched workload, odd element count)
        {"name": "long_chain_mixed", "kind": "chain", "models": 1, "n_min": 3827, "n_max": 3827, "steps": 24,
         "mixed": True},
        # the largest request of the served workload: 200,000 degrees of freedom
        {"name": "largest_chain_mixed", "kind": "chain", "models": 1, "n_min": 33333, "n_max": 33333, "steps": 10,
         "mixed": True},
        # a small parameter study in full precision
        {"name": "batch16_fp64", "kind": "chain", "models": 16, "n_min": 10, "n_max": 1000, "steps": 40,
         "mixed": False},
        # the batched workload: 256 chains of 10 to 4,000 beams, in both precisions
        {"name": "batch256_mixed", "kind": "chain", "models": 256, "n_min": 10, "n_max": 4000, "steps": 40,
         "mixed": True},
        {"name": "batch256_fp64", "kind": "chain", "models": 256, "n_min": 10, "n_max": 4000, "steps": 40,
         "mixed": False},
        # the space-frame tower (12 storeys of 4 x 4 bays) in both precisions
        {"name": "tower_fp64", "kind": "frame", "storeys": 12, "bays": 4, "steps": 8, "mixed": False},
        {"name": "tower_mixed", "kind": "frame", "storeys": 12, "bays": 4, "steps": 8, "mixed": True},
        # the chain of 16 reduced parts: joints, damping, gravity
        {"name": "parts16_fp64", "kind": "parts", "parts": 16, "modes": 30, "steps": 20, "mixed": False},
        # assembly, factorisation and eight solves of the tower's Newton matrix
        {"name": "tower_seam_fp64", "kind": "seam", "storeys": 12, "bays": 4, "nrhs": 8, "mixed": False},
        # a burst of requests of 1,000 to 20,000 degrees of freedom, 10 to 100 steps each
        {"name": "served24_mixed", "kind": "served", "models": 24, "n_min": 167, "n_max": 3333, "steps_min": 10,
         "steps_max": 100, "mixed": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["driven", "chain", "chain", "chain", "frame", "frame", "parts", "seam", "served"])
    mixed = rng.random() < 0.5
    if kind == "driven":
        n = _logint(rng, 5, 2000)
        return {"kind": kind, "models": 1, "n_min": n, "n_max": n, "steps": rng.randint(4, 12), "mixed": mixed}
    if kind == "chain":
        m = _logint(rng, 1, 256)
        if m == 1 or rng.random() < 0.3:
            n = _logint(rng, 10, 33333 if m == 1 else 60000 // m)
            return {"kind": kind, "models": m, "n_min": n, "n_max": n, "steps": rng.randint(5, 10 if n > 8000 else 30),
                    "mixed": mixed}
        return {"kind": kind, "models": m, "n_min": 10, "n_max": _logint(rng, 100, 4000),
                "steps": rng.randint(5, 40), "mixed": mixed}
    if kind == "frame":
        return {"kind": kind, "storeys": rng.randint(3, 12), "bays": rng.randint(2, 4), "steps": rng.randint(3, 8),
                "mixed": mixed}
    if kind == "parts":
        return {"kind": kind, "parts": rng.randint(2, 16), "modes": rng.randint(6, 30), "steps": rng.randint(5, 20),
                "mixed": mixed}
    if kind == "seam":
        return {"kind": kind, "storeys": rng.randint(3, 12), "bays": rng.randint(2, 4), "nrhs": rng.randint(1, 8),
                "mixed": mixed}
    return {"kind": kind, "models": rng.randint(6, 24), "n_min": 167, "n_max": _logint(rng, 300, 3333),
            "steps_min": 10, "steps_max": rng.randint(20, 100), "mixed": True}


def _spread(lo, hi, k, n):
    """k-th of n values between lo and hi, evenly spaced in the logarithm."""
    return int(round(lo * (hi / lo) ** ((k + 0.5) / n)))


def _texts(case, seed, directory=None):
    """(solver-input text, options) of the case's models.  Element and step
    counts are those of the case, spread evenly over the logarithm of its range;
    sections, materials, clamps and loads come from the seed."""
    kind = case["kind"]
    if kind in ("chain", "driven", "served"):
        rng = np.random.default_rng(seed)
        out = []
        for k in range(case["models"]):
            n = _spread(case["n_min"], case["n_max"], k, case["models"])
            # the step counts in another order than the sizes
            steps = case.get("steps") or _spread(case["steps_min"], case["steps_max"], 7 * k % case["models"],
                                                 case["models"])
            out.append(models.batch_c4(1, seed=int(rng.integers(1 << 30)), n_min=n, n_max=n, steps=steps)[0][:2])
        return out
    if kind in ("frame", "seam"):
        floor_nodes = (case["bays"] + 1) ** 2
        extra = min(40, floor_nodes * case["storeys"] // 7)
        return [models.space_frame_c2(seed=seed, storeys=case["storeys"], bays=case["bays"], n_joints=extra,
                                      n_springs=extra, steps=case.get("steps", 1))]
    rng = np.random.default_rng(seed)
    fsi, opts, _ = models.superelement_chain_c3(
        directory, n_parts=case["parts"], n_modes=case["modes"], width=0.2 * rng.uniform(0.8, 1.2),
        height=0.2 * rng.uniform(0.8, 1.2), torque=500.0 * rng.uniform(0.5, 2.0), steps=case["steps"])
    return [(fsi, opts)]


def _rhs(case, seed, neq):
    return np.random.default_rng(seed + 1).standard_normal((case["nrhs"], neq)) * 1.0e4


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "parts":
        with tempfile.TemporaryDirectory() as directory:
            state["models"] = create_models(_texts(case, seed, directory))
    else:
        state["models"] = create_models(_texts(case, seed))
    if case["kind"] == "served":
        return state
    state["batch"] = Batch(state["models"], mixed=case["mixed"])
    state["batch"].snapshot()  # the initial state, for runs that start over
    if case["kind"] == "seam":
        state["rhs"] = _rhs(case, seed, state["models"][0].neq)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "served":
        server = Server(mixed=case["mixed"])
        ids = [server.submit(m) for m in state["models"]]
        left = len(ids)
        while left > 0:
            left -= server.pump()
        out = np.concatenate([server.result(i).reshape(-1) for i in ids])
        server.close()
        return out
    batch = state["batch"]
    if kind == "seam":
        batch.assemble_newton(0, *SEAM_SCALES)
        negative = batch.factor(0)
        return {"x": batch.solve(0, state["rhs"]), "negative_pivots": negative}
    batch.restore()
    if kind == "driven":
        path = []
        for _ in range(case["steps"]):
            batch.step(0)
            path.append(batch.triads(0))
        return np.stack(path)
    batch.run()
    return batch.all_triads()


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
# One Newton iteration reads and writes the models' state and reads their
# constant matrices once; a step takes at least two.  Per beam: K and M (26
# values each), reference data (36 values), positions, velocities and
# accelerations (24 values, read and written); about 3,000 operations in the
# element forces, the tangent and the block elimination of its triad.
_BEAM_BYTES = 8 * (52 + 36 + 48)
_BEAM_FLOPS = 3000


def work(case):
    kind = case["kind"]
    if kind in ("chain", "driven", "served"):
        lo, hi = case["n_min"], case["n_max"]
        mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
        steps = case.get("steps") or 0.5 * (case["steps_min"] + case["steps_max"])
        beams = case["models"] * mean * 2.0 * steps
        return {"bytes": beams * _BEAM_BYTES, "flops": beams * _BEAM_FLOPS}
    if kind in ("frame", "seam"):
        # envelope elimination storey by storey: bandwidth of one floor's equations
        floor = 6 * (case["bays"] + 1) ** 2
        neq = floor * case["storeys"]
        factor, solve = neq * floor ** 2, 4 * neq * floor
        if kind == "seam":
            return {"bytes": 8.0 * (neq * floor + 2 * neq * case["nrhs"]), "flops": factor + case["nrhs"] * solve}
        beams = 4 * (case["bays"] + 1) ** 2 * case["storeys"]
        return {"bytes": case["steps"] * (8.0 * neq * floor + 2.0 * beams * _BEAM_BYTES),
                "flops": case["steps"] * (factor + 2.0 * (solve + beams * _BEAM_FLOPS))}
    n = 12 + case["modes"]
    per = case["parts"] * 2.0 * case["steps"]
    return {"bytes": per * 8 * 3 * n * n, "flops": per * (n ** 3 / 3 + 10 * n * n)}


# ---------------------------------------------------------------------------
# the same results in plain numpy, in 64 bits
# ---------------------------------------------------------------------------
def _records(text, name):
    """The namelist records `name` of a solver-input text as {key: [values]}."""
    out = []
    for body in re.findall(r"&%s\n(.*?)\n/\n" % name, text, re.S):
        pairs = re.findall(r"(\w+)\s*=\s*((?:(?!\w+\s*=).)*)", body, re.S)
        out.append({k: v.replace(",", " ").split() for k, v in pairs})
    return out


def _num(values):
    return np.array([float(v) for v in values])


def _beam_matrices(prop, length):
    """12 x 12 Euler-Bernoulli stiffness and consistent mass, beam along x."""
    area, iy, iz, it = _num(prop["geometry"])[:4]
    rho, young, shear = _num(prop["material"])
    ea, gi = young * area / length, shear * it / length
    mass = rho * area * length
    polar = rho * (iy + iz) * length
    K, M = np.zeros((12, 12)), np.zeros((12, 12))
    for a, k, m in ((0, ea, mass), (3, gi, polar)):
        K[np.ix_([a, a + 6], [a, a + 6])] = [[k, -k], [-k, k]]
        M[np.ix_([a, a + 6], [a, a + 6])] = [[m / 3, m / 6], [m / 6, m / 3]]
    L = length
    for dofs, sign, inertia in (([1, 5, 7, 11], 1.0, iy), ([2, 4, 8, 10], -1.0, iz)):
        s = np.array([1.0, sign, 1.0, sign])
        k = young * inertia / L ** 3 * np.array(
            [[12, 6 * L, -12, 6 * L], [6 * L, 4 * L * L, -6 * L, 2 * L * L],
             [-12, -6 * L, 12, -6 * L], [6 * L, 2 * L * L, -6 * L, 4 * L * L]])
        m = mass / 420 * np.array(
            [[156, 22 * L, 54, -13 * L], [22 * L, 4 * L * L, 13 * L, -3 * L * L],
             [54, 13 * L, 156, -22 * L], [-13 * L, -3 * L * L, -22 * L, 4 * L * L]])
        K[np.ix_(dofs, dofs)] = s[:, None] * k * s
        M[np.ix_(dofs, dofs)] = s[:, None] * m * s
    return K, M


class _BlockTridiagonal:
    """Symmetric block-tridiagonal solve (6 x 6 blocks, one per triad)."""

    def __init__(self, diag, lower):
        self.lower, self.inv = lower, np.empty_like(diag)
        self.inv[0] = np.linalg.inv(diag[0])
        for k in range(1, len(diag)):
            low = lower[k - 1]
            self.inv[k] = np.linalg.inv(diag[k] - low @ self.inv[k - 1] @ low.T)

    def solve(self, b):
        y = b.copy()
        for k in range(1, len(y)):
            y[k] -= self.lower[k - 1] @ (self.inv[k - 1] @ y[k - 1])
        y[-1] = self.inv[-1] @ y[-1]
        for k in range(len(y) - 2, -1, -1):
            y[k] = self.inv[k] @ (y[k] - self.lower[k].T @ y[k + 1])
        return y


def _quaternion_matrix(q):
    w, x, y, z = np.moveaxis(q / np.linalg.norm(q, axis=-1, keepdims=True), -1, 0)
    rows = [[2 * (x * x + w * w) - 1, 2 * (x * y - z * w), 2 * (x * z + y * w)],
            [2 * (y * x + z * w), 2 * (y * y + w * w) - 1, 2 * (y * z - x * w)],
            [2 * (z * x - y * w), 2 * (z * y + x * w), 2 * (z * z + w * w) - 1]]
    return np.stack([np.stack(r, -1) for r in rows], -2)


def _rotation(v):
    """Rotation matrices of rotation vectors; sin(h)/h of half angles below
    5e-4 interpolated linearly, as the solver this models does."""
    half = 0.5 * np.linalg.norm(v, axis=-1, keepdims=True)
    small = half < 5.0e-4
    part = half / 5.0e-4
    with np.errstate(invalid="ignore", divide="ignore"):
        fac = np.where(small, part * (math.sin(5.0e-4) / 5.0e-4) + 1.0 - part, np.sin(half) / half)
    return _quaternion_matrix(np.concatenate([np.cos(half), 0.5 * fac * v], -1))


def _orthonormal(R):
    """Rotation matrices re-orthonormalised through their quaternions (rotations
    of less than a half turn)."""
    w = 0.5 * np.sqrt(1.0 + np.trace(R, axis1=-2, axis2=-1))
    f = 0.25 / w
    q = np.stack([w, (R[:, 2, 1] - R[:, 1, 2]) * f, (R[:, 0, 2] - R[:, 2, 0]) * f, (R[:, 1, 0] - R[:, 0, 1]) * f], -1)
    return _quaternion_matrix(q)


def _chain_positions(text, options, record=False):
    """Triad positions of a beam chain along X after all its time steps (3 x 4
    column by column per triad; or of every step, 3 x 4 row by row): HHT-alpha
    Newton steps of corotated beams, the tangent of the predictor kept."""
    triads = _records(text, "TRIAD")
    origin = np.array([_num(t["ur"]).reshape(3, 4)[:, 3] for t in triads])
    clamp = next(k for k, t in enumerate(triads) if "BC" in t)
    load = _records(text, "LOAD")[0]
    length = origin[1, 0] - origin[0, 0]
    K, M = _beam_matrices(_records(text, "ELEMENT_PROPERTY")[0], length)
    weight = _num(_records(text, "MECHANISM")[0]["weightTranslation"] + _records(text, "MECHANISM")[0]["weightRotation"])
    end = next(float(o.split("=")[1]) for o in options if o.startswith("-timeEnd"))
    tol = next(float(o.split("=")[1]) for o in options if o.startswith("-tolDispNorm"))
    alpha = -next(float(o.split("=")[1]) for o in options if o.startswith("-alphaNewmark"))
    n = len(triads)
    beta, gamma = (1.0 - alpha) ** 2 / 4.0, 0.5 - alpha
    s_acc, s_vel, s_stif = 1.0 / (beta * DT * DT), gamma / (beta * DT), 1.0 + alpha
    free = np.ones((n, 6))
    free[clamp] = 0.0
    w = np.repeat(weight, 3)
    Q = np.zeros((n, 6))
    Q[int(load["triadId"][0]) - 1, int(load["lDof"][0]) - 1] = float(load["f0"][0])
    x, R = origin.copy(), np.tile(np.eye(3), (n, 1, 1))
    v, a = np.zeros((n, 6)), np.zeros((n, 6))
    S = np.tile(np.eye(3), (n - 1, 1, 1))
    fin = np.zeros((n - 1, 12))
    undeformed = np.zeros((n - 1, 2, 3))
    undeformed[:, 1, 0] = length

    def to_local(u):
        ends = np.stack([u[:-1, :3], u[:-1, 3:], u[1:, :3], u[1:, 3:]], 1)
        return np.einsum("eji,egj->egi", S, ends).reshape(n - 1, 12)

    def to_system(f):
        g = np.einsum("eij,egj->egi", S, f.reshape(n - 1, 4, 3)).reshape(n - 1, 12)
        out = np.zeros((n, 6))
        out[:-1] += g[:, :6]
        out[1:] += g[:, 6:]
        return out

    inertia = np.zeros((n, 6))
    elastic = np.zeros((n, 6))
    path = []
    for _ in range(int(round(end / DT))):
        actual = inertia
        dk = (gamma / beta - 1.0) * v + (0.5 * gamma / beta - 1.0) * DT * a
        ak = v / (beta * DT) + (0.5 / beta - 1.0) * a
        total = np.zeros((n, 6))
        N = s_acc * M + s_stif * K
        blocks = np.einsum("eij,egjhk,elk->egihl", S, N.reshape(4, 3, 4, 3)[None].repeat(n - 1, 0), S,
                           optimize=True).reshape(n - 1, 12, 12)
        diag = np.zeros((n, 6, 6))
        diag[:-1] += blocks[:, :6, :6]
        diag[1:] += blocks[:, 6:, 6:]
        lower = blocks[:, 6:, :6].copy()
        diag[clamp] = np.eye(6)
        if clamp > 0:
            lower[clamp - 1] = 0.0
        if clamp < n - 1:
            lower[clamp] = 0.0
        tangent = _BlockTridiagonal(diag, lower)
        residual = s_stif * (Q - elastic) + to_system(to_local(ak) @ M) - alpha * actual
        for it in range(1, 100):
            inc = tangent.solve(residual * free)
            total = total + inc
            v = s_vel * total - dk
            a = s_acc * total - ak
            x = x + inc[:, :3]
            R = _rotation(inc[:, 3:]) @ R
            accel = to_local(a)  # in the frames of the last iterate
            ex = x[1:] - x[:-1]
            ez = np.cross(ex, R[:-1, :, 1] * length)
            ex = ex / np.linalg.norm(ex, axis=1, keepdims=True)
            ez = ez / np.linalg.norm(ez, axis=1, keepdims=True)
            S = np.stack([ex, np.cross(ez, ex), ez], -1)
            for node, (xe, Re) in enumerate(((x[:-1], R[:-1]), (x[1:], R[1:]))):
                local = np.einsum("eji,ejk->eik", S, Re)
                shift = np.einsum("eji,ej->ei", S, xe - x[:-1]) - undeformed[:, node]
                turn = np.stack([local[:, 2, 1], local[:, 0, 2], local[:, 1, 0]], -1)
                fin[:, 6 * node:6 * node + 6] = np.concatenate([shift, turn], 1)
            elastic = to_system(fin @ K)
            inertia = to_system(accel @ M)
            norm = math.sqrt(((w * inc * free) ** 2).sum() / ((w * free) ** 2).sum())
            if it >= 2 and norm < tol:
                break
            residual = s_stif * (Q - elastic) - inertia - alpha * actual
        R = _orthonormal(R)
        if record:
            path.append(np.concatenate([R, x[:, :, None]], 2))
    if record:
        return np.stack(path)
    return np.concatenate([R.transpose(0, 2, 1).reshape(n, 9), x], 1).reshape(-1)


def _frame_solutions(text, rhs):
    """Solutions of the tower's Newton matrix in its start position: beams,
    springs and dampers, dependent triads eliminated through their joints."""
    s_mass, s_damp, s_stif = SEAM_SCALES
    triads = _records(text, "TRIAD")
    ids = {t["id"][0]: k for k, t in enumerate(triads)}
    pos = np.array([_num(t["ur"]).reshape(3, 4)[:, 3] for t in triads])
    fixed = ["BC" in t for t in triads]
    joints = _records(text, "MASTERSLAVEJOINT")
    slave = {ids[j["slaveId"][0]]: k for k, j in enumerate(joints)}
    eq, neq = {}, 0
    for k in range(len(triads)):
        if not fixed[k] and k not in slave:
            eq[k] = neq
            neq += 6
    T = np.zeros((6 * len(triads), neq + len(joints)))
    for k in eq:
        T[6 * k:6 * k + 6, eq[k]:eq[k] + 6] = np.eye(6)
    for k, j in slave.items():
        joint = joints[j]
        m = eq.get(ids[joint["masterId"][0]])
        if m is not None:
            T[6 * k:6 * k + 6, m:m + 6] = np.eye(6)
        T[6 * k + 3:6 * k + 6, neq + j] = _num(joint["initPosInGlobal"]).reshape(3, 4)[:, 2]
    N = np.zeros((6 * len(triads),) * 2)
    props = {p["id"][0]: p for p in _records(text, "ELEMENT_PROPERTY")}
    for e in _records(text, "SUP_EL"):
        a, b = (ids[t] for t in e["triadIds"])
        K, M = _beam_matrices(props[e["elPropId"][0]], np.linalg.norm(pos[b] - pos[a]))
        G = np.kron(np.eye(4), _num(e["supPos"]).reshape(3, 4)[:, :3])
        dofs = np.r_[6 * a:6 * a + 6, 6 * b:6 * b + 6]
        N[np.ix_(dofs, dofs)] += G @ (s_mass * M + s_stif * K) @ G.T
    stiffness = {b["id"][0]: float(b["s0"][0]) for b in _records(text, "SPRING_BASE")}
    axial = [(e["triadIDs"], s_stif * stiffness[e["springBaseId"][0]]) for e in _records(text, "SPRING_ELEMENT")]
    axial += [((e["triad1Id"][0], e["triad2Id"][0]), s_damp * float(e["d0"][0])) for e in _records(text, "DAMPER")]
    for ends, k in axial:
        a, b = (ids[t] for t in ends)
        d = (pos[b] - pos[a]) / np.linalg.norm(pos[b] - pos[a])
        d = np.concatenate([-d, d])
        dofs = np.r_[6 * a:6 * a + 3, 6 * b:6 * b + 3]
        N[np.ix_(dofs, dofs)] += k * np.outer(d, d)
    return np.linalg.solve(T.T @ N @ T, rhs.T).T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chain", "driven"):
        texts = _texts(case, seed)
        if case["steps"] * sum(len(_records(t, "TRIAD")) for t, _ in texts) > 300000:
            return None  # more than about 20 seconds
        parts = [_chain_positions(t, o, record=kind == "driven") for t, o in texts]
        return parts[0] if kind == "driven" else np.concatenate(parts)
    if kind == "seam":
        text = _texts(case, seed)[0][0]
        fixed = sum("BC" in t for t in _records(text, "TRIAD"))
        joints = len(_records(text, "MASTERSLAVEJOINT"))
        neq = 6 * (len(_records(text, "TRIAD")) - fixed - joints) + joints
        return {"x": _frame_solutions(text, _rhs(case, seed, neq)), "negative_pivots": None}
    return None

"""The workloads this library is timed on: calls that hand the simulator a state
(positions and velocities on the host), step it and take the new positions
back, and one that differentiates a rollout.

The scenes are those of the package's own configurations and tests
(pdipc.scenes): square cloths of a regular grid split along alternating
diagonals, pinned at two corners, over an icosphere; a stack of cloths; a batch
of independent cloths of uneven sizes; a tetrahedral block with a cloth.  The
states are made in closed form from the seed:

  * "flight": the cloth has swung down about its pinned edge like a flap (an
    isometry of the rest shape, so nothing is stretched) and swings on;
  * "touch": the flap has reached the sphere: its plane is a fraction of dhat
    away and moves towards it, so the step is cut by the time of impact and the
    contact projections act.

Both carry a smooth random velocity field of a few modes.  exact() restates the
contact-free step (prediction, local step, Chebyshev-accelerated Jacobi sweeps,
the stopping rule) in 64-bit torch, and the rollout's gradients by automatic
differentiation.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "pd-ipc-armadillodemo_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pdipc  # noqa: E402
from pdipc import scenes  # noqa: E402


def listed():
    return [
        # the smallest cloth of the batched configuration, alone: launches and latency
        {"name": "drop16_mixed", "scene": "drop", "n": 16, "sphere": 2, "precision": "mixed", "state": "flight"},
        # configuration 0 in its own precision
        {"name": "drop64_fp64", "scene": "drop", "n": 64, "sphere": 4, "precision": "fp64", "state": "flight"},
        # configuration 0 in the mixed mode, on the sphere: an interactive single cloth
        {"name": "drop64_mixed_touch", "scene": "drop", "n": 64, "sphere": 4, "precision": "mixed", "state": "touch"},
        # the library's default precision (the reference's arithmetic), the autotuner test's mesh
        {"name": "drop96_fp32", "scene": "drop", "n": 96, "sphere": 3, "precision": "fp32", "state": "flight"},
        # a ragged size in between: 181 is prime, so no row of the grid is aligned
        {"name": "drop181_mixed_touch", "scene": "drop", "n": 181, "sphere": 5, "precision": "mixed", "state": "touch"},
        # the plain FP64 form past one wave of blocks
        {"name": "drop257_fp64", "scene": "drop", "n": 257, "sphere": 5, "precision": "fp64", "state": "flight"},
        # configuration 1, the headline: in flight, and when the cloth lies on the sphere
        {"name": "drop512_mixed", "scene": "drop", "n": 512, "sphere": 6, "precision": "mixed", "state": "flight"},
        {"name": "drop512_mixed_touch", "scene": "drop", "n": 512, "sphere": 6, "precision": "mixed", "state": "touch"},
        # configuration 4: four layers on one another and on the sphere (self-collision)
        {"name": "stack4x256_mixed_touch", "scene": "stack", "n": 256, "layers": 4, "sphere": 5, "precision": "mixed",
         "state": "touch"},
        # configuration 2 at 40 of its 256 drops, uneven sides 16 to 128, per-instance stopping
        {"name": "batch40_mixed", "scene": "batch", "count": 40, "precision": "mixed", "state": "flight"},
        # a tetrahedral block above a cloth: strain constraints by SVD, the kind of the reference's example
        {"name": "block8_cloth64_mixed", "scene": "block", "n": 8, "cloth": 64, "sphere": 4, "precision": "mixed",
         "state": "flight"},
        # configuration 3: a rollout of the 128x128 cloth forward and its adjoint backward
        {"name": "rollout128_fp64", "scene": "rollout", "n": 128, "steps": 2, "precision": "fp64", "state": "flight"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop", "drop", "drop", "stack", "batch", "block", "rollout"])
    state = rng.choice(["flight", "touch"])
    if kind == "drop":
        precision = rng.choice(["mixed", "mixed", "fp32", "fp64"])
        n = _log_int(rng, 16, 512 if precision == "mixed" else 256)
        sphere = 2 if n < 32 else 3 if n < 64 else 4 if n < 128 else 5 if n < 320 else 6
        return {"scene": "drop", "n": n, "sphere": sphere, "precision": precision, "state": state}
    if kind == "stack":
        return {"scene": "stack", "n": _log_int(rng, 20, 256), "layers": rng.randint(2, 4), "sphere": rng.randint(3, 5),
                "precision": "mixed", "state": state}
    if kind == "batch":
        return {"scene": "batch", "count": _log_int(rng, 4, 40), "precision": "mixed", "state": state}
    if kind == "block":
        return {"scene": "block", "n": rng.randint(2, 8), "cloth": _log_int(rng, 16, 64), "sphere": rng.randint(2, 4),
                "precision": rng.choice(["mixed", "fp64"]), "state": "flight"}
    return {"scene": "rollout", "n": _log_int(rng, 10, 128), "steps": rng.randint(1, 3), "precision": "fp64",
            "state": "flight"}


# ---------------------------------------------------------------- scenes and states
def _scene(case):
    kind = case["scene"]
    if kind == "drop":  # 20 local-global iterations at the large sizes, 10 else, as the configurations have it
        return scenes.cloth_drop(case["n"], case["sphere"], lg=20 if case["n"] > 256 else 10)
    if kind == "stack":
        return scenes.stack(case["layers"], case["n"], case["sphere"], dhat=5e-4)
    if kind == "batch":
        return scenes.batched(case["count"], 16, 128)
    if kind == "block":
        return scenes.block_drop(case["n"], case["sphere"], cloth_n=case["cloth"])
    return scenes.cloth_drop(case["n"], 1, with_sphere=False)


def _params(case):
    if case["scene"] == "batch":
        return {"instance_stop": 1}
    if case["scene"] == "rollout":
        return {"fixed_outer": 2}
    return {}


def _waves(X, rng, amplitude):
    """A smooth vector field of four modes over the model's own extent."""
    lo = X.min(0)
    size = max(float((X.max(0) - lo).max()), 1e-9)
    U = (X - lo) / size
    out = np.zeros_like(X)
    for _ in range(4):
        k = rng.integers(1, 4, 3) * math.pi
        out += np.sin(U @ k + rng.uniform(0, 2 * math.pi))[:, None] * rng.normal(size=3)[None, :]
    return out * (amplitude / 4.0)


def _flap(C, sphere, case, dhat, rng):
    """One pinned cloth swung about the x axis through its first row."""
    X0 = C.X
    ox, oz = X0[:, 0].min(), X0[:, 2].min()
    a = math.radians(rng.uniform(3.0, 12.0))
    if sphere is not None:
        # the angle at which the cloth's plane is `gap` short of the sphere (its
        # distance to the centre (y, z) is -(y cos a + z sin a)), or part of the way
        c = sphere.X.mean(0)
        r = float(np.linalg.norm(sphere.X - c, axis=1).max())
        gap = rng.uniform(0.3, 0.8) * dhat
        y, z = float(c[1]), float(c[2] - oz)
        touch = math.atan2(-z, -y) + math.acos((r + gap) / math.hypot(y, z))
        a = touch if case["state"] == "touch" else rng.uniform(0.2, 0.7) * touch
    w = math.sqrt(3.0 * 9.8 * math.sin(a)) * rng.uniform(0.8, 1.0)  # a plate swinging from rest
    ys, zs = X0[:, 1], X0[:, 2] - oz
    X = X0.copy()
    X[:, 1] = ys * math.cos(a) - zs * math.sin(a)
    X[:, 2] = ys * math.sin(a) + zs * math.cos(a) + oz
    V = np.zeros_like(X)
    V[:, 1] = -w * (X[:, 2] - oz)
    V[:, 2] = w * X[:, 1]
    V += _waves(X0 - np.array([ox, 0.0, oz]), rng, 0.02)
    X[C.pins] = X0[C.pins]
    V[C.pins] = 0.0
    return X, V


def _state(case, sc, seed):
    """Positions of every vertex and velocities of the simulated ones."""
    rng = np.random.default_rng(seed)
    Xs, Vs = [], []
    kind = case["scene"]
    if kind in ("drop", "batch"):
        for C, S in zip(sc.cloths, sc.statics):
            x, v = _flap(C, S, case, sc.dhat, rng)
            Xs.append(x)
            Vs.append(v)
    elif kind == "stack":
        # layers above one another, falling: "touch" has them within dhat of
        # the sphere and of one another, "flight" 5 mm apart and above it
        touch = case["state"] == "touch"
        top = float(sc.statics[0].X[:, 1].max())
        y = top + (rng.uniform(0.4, 0.8) * sc.dhat if touch else 0.05) + 1e-4
        for C in sc.cloths:
            x = C.X.copy()
            x[:, 1] += y - C.X[:, 1].mean()
            v = _waves(x, rng, 0.01)
            v[:, 1] -= 1.0
            Xs.append(x)
            Vs.append(v)
            y += (rng.uniform(1.2, 1.6) * sc.dhat if touch else 5e-3)
    else:
        for M in list(sc.cloths) + list(sc.solids):
            v = _waves(M.X, rng, 0.1)
            v[M.pins] = 0.0
            Xs.append(M.X.copy())
            Vs.append(v)
    Xs += [S.X for S in sc.statics]
    return np.concatenate(Xs), np.concatenate(Vs)


def prepare(case, seed):
    sc = _scene(case)
    X, V = _state(case, sc, seed)
    sim = pdipc.create_simulator("pd_ipc_simulator", sc, precision=case["precision"], **_params(case))
    state = {"case": case, "sim": sim, "X": X, "V": V}
    if case["scene"] == "rollout":
        # the loss of the rollout: squared distance to a displaced grid
        state["target"] = X + np.random.default_rng(seed + 1).uniform(-0.05, 0.05, X.shape)
    return state


def run(state):
    sim, case = state["sim"], state["case"]
    sim.set_state(state["X"], state["V"])
    if case["scene"] == "rollout":
        sim.adjoint_record(1)
        sim.step(case["steps"])
        x = sim.positions()
        gx, gv, gk = sim.adjoint_backward(2.0 * (x - state["target"]))
        return {"x": x, "gx": gx, "gv": gv, "gk": gk}
    x = sim.animate()
    # the FP32 mode's state is 32-bit: the array it hands over widens it
    return {"x": x.astype(np.float32) if case["precision"] == "fp32" else x.copy()}


def _sizes(case):
    kind = case["scene"]
    if kind == "drop" or kind == "rollout":
        return case["n"] ** 2
    if kind == "stack":
        return case["layers"] * case["n"] ** 2
    if kind == "batch":
        return case["count"] * 5200
    return case["cloth"] ** 2 + (case["n"] + 1) ** 3


def work(case):
    """Per simulated vertex: the state in and the positions out, its stencil
    (7 entries) and matrix row (22 entries) once; the sweeps' multiply-adds over
    the fewest outer iterations the stopping rule lets a step have (it stops
    after the second at the earliest; a step in contact mostly runs all 30)."""
    n = _sizes(case)
    v = 8 if case["precision"] == "fp64" else 4
    lg = 20 if case["scene"] in ("drop", "stack") and (case["n"] > 256 or case["scene"] == "stack") else 10
    outer = 30 if case["state"] == "touch" else 2
    sweeps = outer * lg * 30
    if case["scene"] == "rollout":
        sweeps = case["steps"] * 2 * lg * 30 * 3  # forward, and backward through both factors
    return {"bytes": n * (48.0 + 24.0 + 7 * (4 + 3 * v) + 22 * (4 + v)), "flops": float(sweeps) * n * (22 * 6 + 12)}


# ---------------------------------------------------------------- the step in 64 bits
class _Exact:
    """Cloths without contact, in 64-bit torch (autograd passes through)."""

    def __init__(self, sc, device):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)  # noqa: E731
        src, dst, rest, lbo, ks, mass, bend, cn, pink, model = [], [], [], [], [], [], [], [], [], []
        o = 0
        for m, C in enumerate(sc.cloths):
            X, F, n = C.X, C.F.astype(np.int64), C.X.shape[0]
            area = np.zeros(n)
            e = [X[F[:, (k + 1) % 3]] - X[F[:, k]] for k in range(3)]
            fa = 0.5 * np.linalg.norm(np.cross(e[0], -e[2]), axis=1)
            for k in range(3):
                np.add.at(area, F[:, k], fa / 3.0)
            # half the cotangent of the angle at corner k weighs the opposite edge
            w, pairs = [], []
            for k in range(3):
                u, v = X[F[:, (k + 1) % 3]] - X[F[:, k]], X[F[:, (k + 2) % 3]] - X[F[:, k]]
                w.append(-0.5 * (u * v).sum(1) / np.linalg.norm(np.cross(u, v), axis=1))
                pairs.append(np.sort(np.stack([F[:, (k + 1) % 3], F[:, (k + 2) % 3]], 1), axis=1))
            pairs, w = np.concatenate(pairs), np.concatenate(w)
            uniq, inv = np.unique(pairs[:, 0] * n + pairs[:, 1], return_inverse=True)
            we = np.bincount(inv.reshape(-1), weights=w, minlength=uniq.size)
            a, b = uniq // n, uniq % n
            i, j = np.concatenate([a, b]), np.concatenate([b, a])
            wl = np.concatenate([we, we]) / area[i]
            cv = np.zeros((n, 3))
            np.add.at(cv, i, wl[:, None] * (X[j] - X[i]))
            pk = np.zeros(n)
            pk[C.pins] = C.k_pin
            src.append(i + o), dst.append(j + o), lbo.append(wl), rest.append(np.linalg.norm(X[i] - X[j], axis=1))
            ks.append(np.full(i.size, C.k_stretch)), mass.append(area * C.density), bend.append(area * C.k_bend)
            cn.append(np.linalg.norm(cv, axis=1)), pink.append(pk), model.append(np.full(n, m))
            o += n
        cat = lambda l: t(np.concatenate(l))  # noqa: E731
        self.n, self.i, self.j = o, cat(src), cat(dst)
        self.rest, self.k, self.bend, self.cn, self.pin = cat(rest), cat(ks), cat(bend), cat(cn), cat(pink)
        self.model, self.nmodel = cat(model), len(sc.cloths)
        self.free = self.pin == 0
        lbo = cat(lbo)
        ident = torch.arange(o, device=device)

        def sparse(row, col, val):
            return torch.sparse_coo_tensor(torch.stack([row, col]), val, (o, o), check_invariants=False).coalesce()

        diag = torch.zeros(o, dtype=torch.float64, device=device).index_add_(0, self.i, lbo)
        self.L = sparse(torch.cat([ident, self.i]), torch.cat([ident, self.j]), torch.cat([-diag, lbo]))
        self.Lt = self.L.t().coalesce()
        deg = torch.zeros(o, dtype=torch.float64, device=device).index_add_(0, self.i, self.k)
        self.De = self.pin + deg + torch.sparse.mm(self.Lt * self.Lt, self.bend[:, None])[:, 0]
        self.K = sparse(torch.cat([ident, self.i]), torch.cat([ident, self.j]), torch.cat([self.pin + deg, -self.k]))
        self.Xrest = t(sc.initial_positions()[:o])
        dt, self.dt, self.lg = sc.dt, sc.dt, sc.lg_iterations
        mass = cat(mass)
        self.Di = torch.where(self.free, mass / (dt * dt), torch.zeros_like(mass))
        self.g = sc.gravity

    def neg_offdiag(self, x):  # N x, N = -offdiag(A)
        return self.De[:, None] * x - (torch.sparse.mm(self.K, x) +
                                       torch.sparse.mm(self.Lt, self.bend[:, None] * torch.sparse.mm(self.L, x)))

    def solve(self, x, y, cheby=15, rho=0.9992, w=2.0 / 3.0):
        iD = 1.0 / (self.De + self.Di)[:, None]
        for _ in range(self.lg):
            d = x[self.i] - x[self.j]
            f = (self.k * self.rest / d.norm(dim=1))[:, None] * d
            b = torch.zeros_like(x).index_add(0, self.i, f)
            q = torch.sparse.mm(self.L, x)
            s = q.norm(dim=1)
            q = q * torch.where(s >= 1e-10, self.cn / s.clamp_min(1e-10), torch.ones_like(s))[:, None]
            b = b + torch.sparse.mm(self.Lt, self.bend[:, None] * q)
            b = b + self.Di[:, None] * y + self.pin[:, None] * self.Xrest

            def S(z):
                return (1.0 - w) * z + w * iD * (self.neg_offdiag(z) + b)

            prev, cur, om = x, S(S(x)), 2.0 / (2.0 - rho * rho)
            for _ in range(cheby - 1):
                prev, cur = cur, om * (S(S(cur)) - prev) + prev
                om = 4.0 / (4.0 - rho * rho * om)
            x = cur
        return x

    def step(self, x, v, outer=0, per_model=False, tol=1e-5):
        dt, f = self.dt, self.free[:, None].to(x.dtype)
        v = v * f
        grav = torch.tensor([0.0, self.g, 0.0], dtype=x.dtype, device=x.device)
        y = torch.where(self.free[:, None], x + dt * (v + dt * grav), x)
        cur = y
        run = torch.ones(self.nmodel, dtype=torch.bool, device=x.device)
        for k in range(outer or 30):
            new = self.solve(cur, y)
            if per_model:
                new = torch.where(run[self.model][:, None], new, cur)
            d2 = (new - (x if k == 0 else cur)).detach().square().sum(1)
            cur = new
            if outer or k == 0:
                continue
            if per_model:
                run = run & ~(torch.zeros(self.nmodel, dtype=x.dtype, device=x.device).index_add_(0, self.model, d2) < tol)
                if not bool(run.any()):
                    break
            elif float(d2.sum()) < tol:
                break
        return cur, (cur - x) * ((1.0 - dt) / dt)


def exact(case, seed):
    # contact is left out here (and with it the layers and the block, which meet the sphere or the cloth)
    if case["state"] != "flight" or case["scene"] not in ("drop", "batch", "rollout"):
        return None
    sc = _scene(case)
    X, V = _state(case, sc, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    E = _Exact(sc, device)
    x, v = torch.as_tensor(X[:E.n], device=device), torch.as_tensor(V, device=device)
    if case["scene"] == "rollout":
        x.requires_grad_(), v.requires_grad_()
        a, b = x, v
        for _ in range(case["steps"]):
            a, b = E.step(a, b, outer=2)
        target = X + np.random.default_rng(seed + 1).uniform(-0.05, 0.05, X.shape)
        gx, gv = torch.autograd.grad((a - torch.as_tensor(target, device=device)).square().sum(), (x, v))
        return {"x": a.detach(), "gx": gx, "gv": gv, "gk": None}
    with torch.no_grad():
        a, _ = E.step(x, v, per_model=case["scene"] == "batch")
    return {"x": np.concatenate([a.cpu().numpy(), X[E.n:]])}

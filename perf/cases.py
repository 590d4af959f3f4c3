"""The work a user of the XPBD library has it do, as cases that can be timed and compared.

A pass goes through the Python binding the way a host application does: the positions (and the velocities)
of the frame go in from host arrays, the spheres or the kinematic offset of the frame are set, the collisions
are detected where there are any, some substeps run, and the positions come back into the host's own array.
Every pass starts from the same state, so passes can be repeated.

Positions are what comes back. The velocities are their differences over the time step: they hold no more,
and at a time step of 0.2 ms one rounding of a position is a percent of them; they reach the outputs through
the next substep's prediction.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "xpbd-tissue-sim_gb300"))
import xpbd_gb300 as G  # noqa: E402

GRAVITY = 9.81
DENSITY = 1000.0


def solid(name, nx, ny, nz, h, iters, steps, *, young=3e3, spread=1.0, nu=0.45, dt_us=1000, solver="Gauss-Seidel",
          gather=False, form="Stable-Neohookean-Combined", residual="Never", spheres=0, pull=0.0, learned=False):
    """One mesh of nx x ny x nz hexes of edge h, five tets each. young: the softest tet's modulus, spread: the
    stiffest's over it. spheres: how many press on the top; pull: how far the top face is moved, in h."""
    return {"name": name, "kind": "solid", "nx": nx, "ny": ny, "nz": nz, "h": h, "iters": iters, "steps": steps,
            "young": young, "spread": spread, "nu": nu, "dt_us": dt_us, "solver": solver, "gather": gather,
            "form": form, "residual": residual, "spheres": spheres, "pull": pull, "learned": learned}


def listed():
    return [
        # a toy mesh, a single substep: what one call costs
        solid("sliver", 3, 5, 2, 0.02, 5, 1),
        # the 5,000-tet unit cube at 10 sweeps, ten substeps between two reads: an interactive loop
        solid("cube", 10, 10, 10, 0.1, 10, 10),
        # the 50,000-tet beam under a sphere, one collision period (10 substeps, one detection)
        solid("beam_sphere", 10, 100, 10, 0.005, 20, 10, young=1e4, nu=0.49, spheres=1),
        # the 1.3M-tet block with per-tet stiffness at the sweeps it needs to 1e-3, the top pulled up
        solid("block", 64, 64, 64, 0.1 / 64, 88, 1, young=1e3, spread=100.0, pull=0.064),
        # the same mesh under the parallel solver, on a material on which it is stable
        solid("block_jacobi", 64, 64, 64, 0.1 / 64, 30, 2, dt_us=200, solver="Jacobi", pull=0.064),
        # the parallel solver's deterministic form on an odd mesh
        solid("odd_jacobi_gather", 37, 23, 31, 0.1 / 64, 20, 4, dt_us=200, solver="Jacobi", gather=True),
        # the two element constraints projected one after the other
        solid("odd_separate", 33, 17, 21, 0.004, 10, 5, young=1e4, form="Stable-Neohookean"),
        # convergence studies: the residual before every sweep
        solid("history", 40, 40, 40, 0.0025, 30, 1, young=1e3, spread=10.0, residual="Every-Iteration"),
        # the learned warm start (network, residual test, fall-back) before the sweeps
        solid("learned_start", 48, 48, 48, 0.1 / 48, 10, 2, young=1e3, spread=10.0, learned=True),
        # many patients or parameters at once: 96 uneven instances with their own spheres
        {"name": "batch", "kind": "batch", "instances": 96, "sizes": 0, "tets_lo": 2000, "tets_hi": 100000, "iters": 20,
         "steps": 2},
        # two parts of one mesh pressed into each other: self-collisions
        {"name": "fold", "kind": "fold", "n": 12, "iters": 8, "steps": 2},
        # one training batch of the warm start's network: loss and gradient
        {"name": "train", "kind": "train", "rows": 65536},
    ]


def draw(rng):
    def odd(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solid"] * 4 + ["contact"] * 2 + ["jacobi"] * 2 + ["separate", "history", "batch", "fold", "train"])
    if kind == "batch":
        return {"kind": "batch", "instances": odd(3, 64), "sizes": rng.randrange(1 << 20), "tets_lo": 500,
                "tets_hi": odd(5000, 50000), "iters": rng.randint(5, 20), "steps": rng.randint(1, 3)}
    if kind == "fold":
        return {"kind": "fold", "n": odd(5, 16), "iters": rng.randint(4, 10), "steps": rng.randint(1, 3)}
    if kind == "train":
        return {"kind": "train", "rows": odd(300, 200000)}
    hexes = odd(24, 200000 if kind in ("solid", "jacobi") else 40000)
    long = rng.choice([1, 1, 3, 8])  # a cube or a beam
    n = max(2.0, (hexes / long) ** (1 / 3))
    nx, nz = (max(1, int(round(n * rng.uniform(0.8, 1.25)))) for _ in range(2))
    ny = max(2, int(round(hexes / (nx * nz))))
    c = solid("", nx, ny, nz, rng.uniform(0.002, 0.02), rng.randint(5, 30), rng.randint(1, 4),
              young=rng.uniform(1e3, 1e4), spread=rng.choice([1.0, 10.0]), nu=rng.uniform(0.40, 0.49))
    if kind == "contact":
        c["spheres"] = rng.randint(1, 4)
    elif kind == "jacobi":
        c.update(h=0.1 / 64, young=3e3, spread=1.0, nu=0.45, dt_us=200, solver="Jacobi", gather=rng.random() < 0.4)
    elif kind == "separate":
        c["form"] = "Stable-Neohookean"
    elif kind == "history":
        c["residual"] = rng.choice(["Every-Substep", "Every-Iteration"])
    elif rng.random() < 0.25:
        c["pull"] = 0.05
    del c["name"]
    return c


# ---- meshes and inputs ----
def hex_mesh(nx, ny, nz, h):
    """A grid of hexes, five tets each in two mirrored splits: vertices (z fastest, then x, then y), tets hex by
    hex in that order, and the surface triangles."""
    y, x, z = np.meshgrid(np.arange(ny + 1), np.arange(nx + 1), np.arange(nz + 1), indexing="ij")
    X = np.stack([x, y, z], -1).reshape(-1, 3) * h

    def vid(i, j, k):
        return k + i * (nz + 1) + j * (nx + 1) * (nz + 1)

    j, i, k = (a.ravel() for a in np.meshgrid(np.arange(ny), np.arange(nx), np.arange(nz), indexing="ij"))
    c = np.stack([vid(i + a, j + b, k + d) for a, b, d in
                  ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))], 1)
    A = np.array([[0, 1, 2, 5], [0, 2, 3, 7], [0, 5, 4, 7], [2, 5, 6, 7], [0, 2, 5, 7]])
    B = np.array([[0, 3, 1, 4], [1, 3, 2, 6], [1, 5, 4, 6], [3, 4, 7, 6], [1, 3, 4, 6]])
    first = (i + j + k) % 2 == 0
    tets = np.where(first[:, None, None], c[:, A], c[:, B]).reshape(-1, 4).astype(np.int32)

    faces = []
    for axis, n in ((1, ny), (0, nx), (2, nz)):
        for at in (0, n):
            p, q = [a for a in (0, 1, 2) if a != axis]
            dims = (nx, ny, nz)
            u, v = (a.ravel() for a in np.meshgrid(np.arange(dims[p]), np.arange(dims[q]), indexing="ij"))

            def corner(du, dv):
                w = [None] * 3
                w[axis], w[p], w[q] = np.full_like(u, at), u + du, v + dv
                return vid(*w)

            a, b, d, e = corner(0, 0), corner(1, 0), corner(1, 1), corner(0, 1)
            ac = ((u + v + at) % 2 == 0)[:, None]  # the diagonal that the tets below have
            t1 = np.where(ac, np.stack([a, b, d], 1), np.stack([a, b, e], 1))
            t2 = np.where(ac, np.stack([a, d, e], 1), np.stack([b, d, e], 1))
            faces.append(np.stack([t1, t2], 1).reshape(-1, 3))
    return X, tets, np.concatenate(faces).astype(np.int32)


def bodies(case):
    """The meshes of a case: dicts of the hex counts, the edge, young, nu and the spheres (centres, radii)."""
    if case["kind"] == "solid":
        b = {k: case[k] for k in ("nx", "ny", "nz", "h", "young", "spread", "nu")}
        n, w = case["spheres"], case["nx"] * case["h"]
        r = np.full(n, 0.6 * w)
        at = (np.arange(n) + 0.5) / max(n, 1) * case["ny"] * case["h"]
        b["spheres"] = (np.stack([np.full(n, w / 2), at, case["nz"] * case["h"] + r - 0.4 * case["h"]], 1), r)
        return [b]
    if case["kind"] == "fold":
        return [dict(nx=case["n"], ny=case["n"], nz=case["n"], h=0.1 / case["n"], young=2e4, spread=1.0, nu=0.45,
                     spheres=None)] * 2
    rng, out = np.random.default_rng(case["sizes"]), []
    for _ in range(case["instances"]):
        target = np.exp(rng.uniform(np.log(case["tets_lo"]), np.log(case["tets_hi"]))) / 5.0
        long = 1 if rng.random() < 0.5 else 4
        m = max(2, int(round((target / long) ** (1 / 3))))
        h = 0.05 / m
        ns = int(rng.integers(1, 5))
        r = rng.uniform(0.2, 0.4, ns) * m * h
        out.append(dict(nx=m, ny=long * m, nz=m, h=h, young=float(np.exp(rng.uniform(np.log(1e3), np.log(1e5)))),
                        spread=1.0, nu=float(rng.uniform(0.40, 0.49)),
                        spheres=(np.stack([rng.uniform(0.2, 0.8, ns) * m * h, rng.uniform(0.2, 0.8, ns) * long * m * h,
                                           m * h + 0.9 * r], 1), r)))
    return out


def inputs(case, seed):
    """Everything a pass works on, from the seed: meshes, materials, positions, velocities, spheres."""
    rng = np.random.default_rng(seed)
    s = {"meshes": [], "spheres": [], "x": [], "v": [], "fixed": [], "top": [], "voff": [0]}
    for n, b in enumerate(bodies(case)):
        X, tets, faces = hex_mesh(b["nx"], b["ny"], b["nz"], b["h"])
        h, T = b["h"], len(tets)
        E = b["young"] * np.exp(rng.uniform(0.0, np.log(b["spread"]) + 1e-3, T)) if b["spread"] > 1 else \
            np.full(T, b["young"] * (1 + 0.1 * rng.random()))
        # a state in motion: a smooth bend of a tenth of an edge, every vertex off by up to a thousandth
        bend = 0.1 * h * np.sin(X @ rng.uniform(-1, 1, (3, 3)) * (2 / np.abs(X).max()))
        x = X + bend * (X[:, 2:] > 0) + rng.uniform(-1e-3, 1e-3, X.shape) * h
        v = rng.uniform(-0.05, 0.05, 3) * (X[:, 2:] / X[:, 2].max()) + rng.uniform(-1e-3, 1e-3, X.shape)
        if case["kind"] == "fold":
            # two cubes side by side, pushed into each other by a sixth of an edge, meeting at 2 m/s
            shift = np.array([0.1 - h / 6, 0.013, 0.007]) * n
            X, x = X + np.array([0.102, 0.013, 0.007]) * n, X + shift + rng.uniform(-0.01, 0.01, X.shape) * h
            v = v + np.array([1.0 - 2.0 * n, 0.0, 0.0])
        x, v = x.astype(np.float32), v.astype(np.float32).astype(np.float64)
        s["meshes"].append((X, tets, faces, E, np.full(T, b["nu"]), np.full(T, DENSITY)))
        if b["spheres"] is not None and len(b["spheres"][1]):
            c, r = b["spheres"]
            s["spheres"].append((c + rng.uniform(-0.05, 0.05, c.shape) * h, r))
        s["x"].append(x)
        s["v"].append(v)
        s["fixed"].append((X[:, 2] == 0) if case["kind"] != "fold" else np.zeros(len(X), bool))
        s["top"].append(np.nonzero(X[:, 2] == X[:, 2].max())[0].astype(np.int32))
        s["voff"].append(s["voff"][-1] + len(X))
    for k in ("x", "v", "fixed"):
        s[k] = np.concatenate(s[k])
    return s


def he_network(seed):
    """The network's parameters as a flat vector (W1 64x16, b1, W2, b2, W3, b3 64x64, W4 2x64, b4)."""
    rng = np.random.default_rng(seed)
    W1 = rng.standard_normal((64, 16)) * math.sqrt(2 / 14)
    W1[:, 14:] = 0
    W2, W3 = (rng.standard_normal((64, 64)) * math.sqrt(2 / 64) for _ in range(2))
    W4 = rng.standard_normal((2, 64)) * 0.1 * math.sqrt(2 / 64)
    b = [0.05 * rng.standard_normal(n) for n in (64, 64, 64, 2)]
    return np.concatenate([p.ravel() for p in (W1, b[0], W2, b[1], W3, b[2], W4, b[3])]).astype(np.float32)


def rows(case, seed):
    """Training rows as the solver records them: F near the identity, scaled multipliers, log10(E)/5, nu, 1e3 dt;
    the targets near the multipliers of the substep before."""
    rng, n = np.random.default_rng(seed), case["rows"]
    X = np.zeros((n, 16), np.float32)
    X[:, :9] = (np.eye(3)[None] + 0.05 * rng.standard_normal((n, 3, 3))).reshape(n, 9)
    X[:, 9] = -math.sqrt(3) + 0.1 * rng.standard_normal(n)
    X[:, 10] = rng.uniform(0.02, 0.25, n)
    X[:, 11] = rng.uniform(0.6, 1.0, n)
    X[:, 12] = rng.uniform(0.40, 0.49, n)
    X[:, 13] = 1.0
    return X, (X[:, 9:11] + 0.02 * rng.standard_normal((n, 2))).astype(np.float32)


# ---- the passes ----
def prepare(case, seed):
    if case["kind"] == "train":
        X, tets, _ = hex_mesh(2, 2, 2, 0.1)
        s = G.XPBDSolver(X, tets, None, 3e3, 0.45, DENSITY, dt=1e-3)
        s.set_mlp_params(he_network(seed))
        X, Y = rows(case, seed)
        return {"kind": "train", "solver": s, "X": X, "Y": Y}
    d = inputs(case, seed)
    p = dict(num_iters=case["iters"], dt=case.get("dt_us", 1000) * 1e-6, g_accel=GRAVITY, collision_rate=0.0)
    if case["kind"] == "solid":
        p.update(solver_type=case["solver"], constraint_type=case["form"], residual_policy=case["residual"],
                 jacobi_variant=G.JACOBI_GATHER if case["gather"] else G.JACOBI_ATOMIC)
    if case["kind"] == "fold":
        p.update(self_collisions=1, g_accel=0.0)
    touching = bool(d["spheres"]) or case["kind"] == "fold"
    s = G.XPBDSolver(instances=[m if touching else m[:2] + (None,) + m[3:] for m in d["meshes"]], **p)
    s.fix_vertices(d["fixed"])
    state = {"kind": case["kind"], "solver": s, "x": d["x"], "v": d["v"], "steps": case["steps"],
             "spheres": d["spheres"], "detect": touching, "out": np.zeros_like(d["x"]), "offset": None,
             "history": case.get("residual", "Never") != "Never"}
    if case.get("pull"):
        s.set_kinematic_group(d["top"][0])
        state["offset"] = np.array([0.0, 0.0, case["pull"] * case["h"]])
    if case.get("learned"):
        s.set_mlp_params(he_network(seed))
        s.set_warm_start(G.WARM_MLP)
    return state


def run(state):
    s = state["solver"]
    if state["kind"] == "train":
        loss, grad = s.mlp_loss_grad(state["X"], state["Y"])
        return {"loss": loss, "grad": grad}
    s.set_positions_f32(state["x"])
    s.set_velocities(state["v"])
    if state["offset"] is not None:
        s.set_kinematic_offset(state["offset"])
    for k, (c, r) in enumerate(state["spheres"]):
        s.set_spheres(c, r, instance=k)
    if state["detect"]:
        s.detect_collisions()
    s.step(state["steps"])
    out = {"x": s.positions_f32(out=state["out"])}
    if state["history"]:
        out["history"] = s.residual_history()
    if state["kind"] == "fold":
        out["pairs"] = s.self_contacts()[0]
    return out


def work(case):
    """Per sweep: a tet's four indices, its 48 bytes of rest shape and compliance and its two multipliers (read
    and written), and per vertex its position (read and written) and inverse mass; per substep the prediction
    and the velocities. About 400 operations a projection."""
    if case["kind"] == "train":
        n = case["rows"]  # three times the forward pass's products; rows in, gradient out
        return {"bytes": n * (64 + 8) + 9538 * 8, "flops": 6.0 * n * (14 * 64 + 2 * 64 * 64 + 2 * 64)}
    T = V = 0
    for b in bodies(case):
        T += 5 * b["nx"] * b["ny"] * b["nz"]
        V += (b["nx"] + 1) * (b["ny"] + 1) * (b["nz"] + 1)
    n = case["steps"]
    return {"bytes": n * (case["iters"] * (80 * T + 28 * V) + 84 * V) + 48 * V, "flops": 400.0 * n * case["iters"] * T}


# ---- the same in 64 bits, in plain torch ----
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=DEVICE)


class Tissue:
    """The concatenated meshes of a case: rest shapes, compliances, masses and the hexes' colours."""

    def __init__(self, case, d):
        self.dt = case.get("dt_us", 1000) * 1e-6
        off = d["voff"]
        X = _t(np.concatenate([m[0] for m in d["meshes"]]))
        self.idx = torch.cat([_t(m[1], torch.int64) + o for m, o in zip(d["meshes"], off)])
        E, nu, rho = (_t(np.concatenate([m[k] for m in d["meshes"]])) for k in (3, 4, 5))
        D = (X[self.idx[:, :3]] - X[self.idx[:, 3:]]).transpose(1, 2)  # columns: the rest edges
        det = torch.linalg.det(D)
        self.Q = torch.linalg.inv(D)
        vol = det.abs() / 6
        mu, la = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        self.at = torch.stack([1 / (mu * vol), 1 / (la * vol)], 1) / self.dt ** 2
        self.gamma = mu / la
        mass = torch.zeros(len(X), dtype=torch.float64, device=DEVICE)
        mass.index_add_(0, self.idx.reshape(-1), (vol * rho / 4).repeat_interleave(4))
        self.w = 1 / mass
        # colours of the hexes in index order, each the smallest free one: the parities of the axes that have
        # more than one hex, the fastest axis first
        colour = []
        for b in bodies(case):
            c, bit = 0, 1
            g = np.meshgrid(np.arange(b["ny"]), np.arange(b["nx"]), np.arange(b["nz"]), indexing="ij")
            for axis, n in ((2, b["nz"]), (1, b["nx"]), (0, b["ny"])):
                if n > 1:
                    c, bit = c + bit * (g[axis] % 2), 2 * bit
            colour.append(np.zeros(g[0].shape, int).ravel() + np.ravel(c))
        colour = _t(np.concatenate(colour), torch.int64)
        self.groups = [[h * 5 + k for k in range(5)] for h in
                       (torch.nonzero(colour == q).ravel() for q in range(int(colour.max()) + 1))]
        self.data = [[(self.idx[t], self.Q[t], self.at[t], self.gamma[t], t) for t in g] for g in self.groups]

    @staticmethod
    def constraints(p, Q, gamma):
        """Values and gradients of |F| and of log J (its cubic below J = 1) less gamma."""
        F = (p[:, :3] - p[:, 3:]).transpose(1, 2) @ Q
        f0, f1, f2 = F[:, :, 0], F[:, :, 1], F[:, :, 2]
        cof = torch.stack([torch.linalg.cross(f1, f2), torch.linalg.cross(f2, f0), torch.linalg.cross(f0, f1)], 2)
        Cd = F.square().sum((1, 2)).sqrt()
        J = (f0 * cof[:, :, 0]).sum(1)
        d = J - 1
        Ch = torch.where(J >= 1, torch.log(J.clamp(min=1)), d - d * d / 2 + d ** 3 / 3) - gamma
        fac = torch.where(J >= 1, 1 / J.clamp(min=1), 1 - d + d * d)
        g = torch.stack([F / Cd[:, None, None], cof * fac[:, None, None]], 1) @ Q[:, None].transpose(2, 3)
        g = torch.cat([g, -g.sum(3, keepdim=True)], 3).transpose(2, 3)  # tet, constraint, vertex, coordinate
        return torch.stack([Cd, Ch], 1), g

    def project(self, x, lam, data, which=None):
        """The vertex updates of some tets from one state; their multipliers move."""
        e, Q, at, gamma, t = data
        w = self.w[e]
        C, g = self.constraints(x[e], Q, gamma)
        wg = g * w[:, None, :, None]
        r = C + at * lam[t]
        if which is None:
            L = torch.einsum("tavk,tbvk->tab", wg, g)
            a, b, d = L[:, 0, 0] + at[:, 0], L[:, 0, 1], L[:, 1, 1] + at[:, 1]
            dl = torch.stack([r[:, 1] * b - r[:, 0] * d, r[:, 0] * b - r[:, 1] * a], 1) / (a * d - b * b)[:, None]
        else:
            dl = torch.zeros_like(r)
            dl[:, which] = -r[:, which] / ((wg * g).sum((2, 3))[:, which] + at[:, which])
        lam[t] = lam[t] + dl
        return (wg * dl[:, :, None, None]).sum(1)

    def residual(self, x, lam):
        return float((self.constraints(x[self.idx], self.Q, self.gamma)[0] + self.at * lam).square().sum().sqrt())

    def sweep(self, x, lam, separate):
        for which in ((0, 1) if separate else (None,)):
            for group in self.data:
                for data in group:
                    d = self.project(x, lam, data, which)
                    at = data[0].reshape(-1)
                    x[at] = x[at] + d.reshape(-1, 3)

    def jacobi(self, x, lam):
        every = slice(None)
        d = self.project(x, lam, (self.idx, self.Q, self.at, self.gamma, every))
        x.index_add_(0, self.idx.reshape(-1), d.reshape(-1, 3))


def greedy(items, n):
    """The smallest colour that no earlier item on a shared vertex has, item by item."""
    used, out = [0] * n, []
    for a, b, c in items.tolist():
        m = used[a] | used[b] | used[c]
        k = (~m & (m + 1)).bit_length() - 1
        out.append(k)
        m = 1 << k
        used[a] |= m
        used[b] |= m
        used[c] |= m
    return np.array(out, dtype=np.int64)


class Pressed:
    """The contacts of the surface with spheres: the least distance over each triangle by 32 Frank-Wolfe steps,
    the contact's barycentric point and the sphere's surface point and normal."""

    def __init__(self, d, x):
        faces = np.concatenate([m[2].astype(np.int64) + o for m, o in zip(d["meshes"], d["voff"])])
        inst = np.repeat(np.arange(len(d["meshes"])), [len(m[2]) for m in d["meshes"]])
        colour = _t(greedy(faces, len(d["x"])), torch.int64)
        faces, self.groups = _t(faces, torch.int64), []
        p = x[faces]
        found = []
        for s in range(max(len(r) for _, r in d["spheres"])):
            c = _t(np.stack([m[0][s] if s < len(m[1]) else np.zeros(3) for m in d["spheres"]]))[inst]
            r = _t(np.array([m[1][s] if s < len(m[1]) else -1.0 for m in d["spheres"]]))[inst]

            def sdf(q):
                return (q - c).norm(dim=1) - r

            edge = torch.stack([(p[:, a] - p[:, b]).square().sum(1) for a, b in ((0, 1), (0, 2), (1, 2))]).amax(0)
            near = (sdf(p.mean(1)).square() <= edge) & (r >= 0)
            q = p[torch.arange(len(p), device=DEVICE), torch.stack([sdf(p[:, k]) for k in range(3)]).argmin(0)]
            for i in range(32):
                g = (q - c) / (q - c).norm(dim=1, keepdim=True)
                to = p[torch.arange(len(p), device=DEVICE), (p * g[:, None]).sum(2).argmin(1)]
                q = q + 2.0 / (i + 3) * (to - q)
            far = sdf(q)
            f = torch.nonzero(near & (far <= 1e-4)).ravel()
            u, v, t = (p[:, 1] - p[:, 0])[f], (p[:, 2] - p[:, 0])[f], (q - p[:, 0])[f]
            uu, uv, vv, tu, tv = ((a * b).sum(1) for a, b in ((u, u), (u, v), (v, v), (t, u), (t, v)))
            den = uu * vv - uv * uv
            bv, bw = (vv * tu - uv * tv) / den, (uu * tv - uv * tu) / den
            n = ((q - c) / (q - c).norm(dim=1, keepdim=True))[f]
            found.append((f, torch.stack([1 - bv - bw, bv, bw], 1), q[f] - n * far[f, None], n))
        for k in range(int(colour.max()) + 1):
            for f, bary, at, n in found:
                m = colour[f] == k
                if bool(m.any()):
                    self.groups.append((faces[f[m]], bary[m], at[m], n[m]))

    def project(self, x, w):
        for e, b, at, n in self.groups:
            C = (n * ((b[:, :, None] * x[e]).sum(1) - at)).sum(1)
            dl = torch.where(C > 0, 0.0, -C / (w[e] * b * b).sum(1))
            x[e] = x[e] + (w[e] * b * dl[:, None])[:, :, None] * n[:, None]


def crossing(d, x):
    """Self-collisions: for each surface vertex the lowest tet holding it, and the rest face closest to the
    vertex mapped back through that tet. Returns (vertex, face vertices) rows in vertex order."""
    faces = _t(np.concatenate([m[2].astype(np.int64) + o for m, o in zip(d["meshes"], d["voff"])]), torch.int64)
    tets = torch.cat([_t(m[1], torch.int64) + o for m, o in zip(d["meshes"], d["voff"])])
    X = _t(np.concatenate([m[0] for m in d["meshes"]]))
    # tets and vertices in the box that the two parts share
    k = d["voff"][1]
    lo, hi = torch.maximum(x[:k].amin(0), x[k:].amin(0)), torch.minimum(x[:k].amax(0), x[k:].amax(0))
    q = x[tets]
    t = torch.nonzero(((q.amin(1) <= hi) & (q.amax(1) >= lo)).all(1)).ravel()
    verts = torch.unique(faces)
    verts = verts[((x[verts] >= lo) & (x[verts] <= hi)).all(1)]
    out = []
    p = x[tets[t]]
    for v in verts.tolist():
        inside = ~(tets[t] == v).any(1)
        for a, b, c, e in ((0, 1, 2, 3), (0, 1, 3, 2), (0, 2, 3, 1), (1, 2, 3, 0)):
            n = torch.linalg.cross(p[:, b] - p[:, a], p[:, c] - p[:, a])
            inside &= (n * (x[v] - p[:, a])).sum(1) * (n * (p[:, e] - p[:, a])).sum(1) >= 0
        hit = torch.nonzero(inside).ravel()
        if not len(hit):
            continue
        e = tets[t[hit[0]]]
        F = (x[e[:3]] - x[e[3]]).T @ torch.linalg.inv((X[e[:3]] - X[e[3]]).T)
        m = torch.linalg.solve(F, x[v] - x[e[3]]) + X[e[3]]
        A, B, C = X[faces[:, 0]], X[faces[:, 1]], X[faces[:, 2]]
        best = None
        for a, b in ((A, B), (B, C), (C, A)):  # the edges
            s = (((m - a) * (b - a)).sum(1) / (b - a).square().sum(1)).clamp(0, 1)
            dist = (m - a - s[:, None] * (b - a)).square().sum(1)
            best = dist if best is None else torch.minimum(best, dist)
        n = torch.linalg.cross(B - A, C - A)
        within = torch.stack([(torch.linalg.cross(b - a, m - a) * n).sum(1) >= 0 for a, b in ((A, B), (B, C), (C, A))]).all(0)
        best = torch.where(within, ((m - A) * n).sum(1).square() / n.square().sum(1), best)
        out.append([v] + faces[int(best.argmin())].tolist())
    return out


def press_pairs(pairs, lam, x, w, at):
    """The vertex-face pairs one after the other: C = (q - p1) . a / |a| + 1e-5, a = (p2 - p1) x (p3 - p1)."""
    for j, ids in enumerate(pairs):
        q, p1, p2, p3 = x[ids]
        a = np.cross(p2 - p1, p3 - p1)
        n = np.linalg.norm(a)
        C = (q - p1) @ a / n + 1e-5
        if C > 0:
            continue
        r1, r2 = ((u / n - a * (a @ u) / n ** 3) for u in (q - p1, q - p2))
        g = np.stack([a / n, -a / n + np.cross(r1, p3 - p2), np.cross(r1, p1 - p3), np.cross(r2, p2 - p1)])
        dl = (-C - at * lam[j]) / (at + (w[ids] * (g * g).sum(1)).sum())
        lam[j] += dl
        x[ids] += w[ids, None] * g * dl


def exact(case, seed):
    if case["kind"] == "train":
        X, Y = (_t(a) for a in rows(case, seed))
        p, at, W = _t(he_network(seed)).requires_grad_(True), 0, []
        for n, k in ((64, 16), (64, 0), (64, 64), (64, 0), (64, 64), (64, 0), (2, 64), (2, 0)):
            W.append(p[at:at + n * max(k, 1)].reshape((n, k) if k else (n,)))
            at += n * max(k, 1)
        a = X
        for k in range(4):
            a = a @ W[2 * k].T + W[2 * k + 1]
            a = torch.nn.functional.silu(a) if k < 3 else a
        loss = (a - Y).square().sum(1).mean()
        loss.backward()
        return {"loss": loss.detach(), "grad": p.grad}
    d = inputs(case, seed)
    if DEVICE == "cpu" and work(case)["flops"] > 3e10:
        return None
    m = Tissue(case, d)
    x, v, fixed = _t(d["x"]), _t(d["v"]), _t(d["fixed"], torch.bool)
    g = 0.0 if case["kind"] == "fold" else GRAVITY
    if case.get("pull"):
        top = _t(d["top"][0], torch.int64)
        # the group's rest positions are the mesh's, rounded as the library keeps them
        x[top] = _t(d["meshes"][0][0].astype(np.float32))[top] + _t([0.0, 0.0, case["pull"] * case["h"]])
        fixed[top] = True
    touch = Pressed(d, x) if d["spheres"] else None
    pairs = crossing(d, x) if case["kind"] == "fold" else []
    history, residual = [], case.get("residual", "Never")
    for _ in range(case["steps"]):
        before = x.clone()
        x = x + m.dt * v
        x[:, 2] -= g * m.dt ** 2
        lam, plam, history = torch.zeros_like(m.at), np.zeros(len(pairs)), []
        for it in range(case["iters"]):
            if residual == "Every-Iteration" or (residual == "Every-Substep" and it == 0):
                history.append(m.residual(x, lam))
            if case.get("solver") == "Jacobi":
                m.jacobi(x, lam)
            else:
                m.sweep(x, lam, case.get("form") == "Stable-Neohookean")
            if touch:
                touch.project(x, m.w)
            if pairs:
                xn = x.cpu().numpy().copy()
                press_pairs(pairs, plam, xn, m.w.cpu().numpy(), 1e-8 / m.dt ** 2)
                x = _t(xn)
        if residual != "Never":
            history.append(m.residual(x, lam))
        x[fixed] = before[fixed]
        v = (x - before) / m.dt
    out = {"x": x}
    if residual != "Never":
        out["history"] = _t(history)
    if case["kind"] == "fold":
        out["pairs"] = None
    return out

"""The work that users of this package have it do, as cases that can be timed and checked.

A case names a discretization (law, volume form, dimension, polynomial order N, elements K
per side, kind of grid, precision) and what is done with it: LSRK(5,4) steps, one tendency,
or a batch of solves through the serving loop.  ``prepare`` makes what a user's program
holds before the call (grid, DGSEM handle, state, solver, or a running server), ``run`` is
one pass through the public entry points, and ``exact`` is the same result from a plain
torch restatement of the scheme in 64 bits.
"""

import functools
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch


def _package():
    """The package directory ``raven.jl_b200`` as module ``raven_b200``."""
    if "raven_b200" not in sys.modules:
        pkg = os.path.join(os.getcwd(), "raven.jl_b200")
        spec = importlib.util.spec_from_file_location("raven_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        sys.modules["raven_b200"] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules["raven_b200"])
    return sys.modules["raven_b200"]


GAMMA = 1.4
ADV_VELOCITY = (1.0, 0.5, 0.25)
MAX_NODES = 32**3 * 8**3  # nodes of the largest grid: 32^3 elements at N = 7
L2_BYTES = 126e6


def _case(name, do, law, form, dim, N, K, grid="brick", precision="fp64", steps=1):
    c = {"do": do, "law": law, "form": form, "dim": dim, "N": N, "K": K, "grid": grid, "precision": precision,
         "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one right-hand side of a small 2-D problem, as a driver with its own time stepper
        # or a test calls it: the smallest call, launch and host latency
        _case("rhs_euler2d_ec_n4_5", "tendency", "euler", "ec", 2, 4, 5),
        # 100 time steps of 2-D linear advection on 16^2 elements: a small solve in one call
        _case("adv2d_weak_n4_16_100steps", "steps", "adv", "weak", 2, 4, 16, steps=100),
        # the entropy-conservative 2-D vortex at its third refinement level, ten steps and
        # the norm that a driver reports
        _case("euler2d_ec_n4_40", "steps+norm", "euler", "ec", 2, 4, 40, steps=10),
        # the same scheme in 3-D at the order of the reference's tests (odd Nq)
        _case("euler3d_ec_n4_18", "steps", "euler", "ec", 3, 4, 18),
        # 3-D Euler, Kennedy-Gruber, N = 7: the headline workload, in both precisions
        _case("euler3d_kg_n7_32_fp64", "steps", "euler", "kg", 3, 7, 32),
        _case("euler3d_kg_n7_32_fp32bulk", "steps", "euler", "kg", 3, 7, 32, precision="fp32_bulk"),
        # the same scheme on warped geometry, in both precisions
        _case("euler3d_kg_n7_16_warped_fp32bulk", "steps", "euler", "kg", 3, 7, 16, "warped", "fp32_bulk"),
        _case("euler3d_kg_n7_13_warped_fp64", "steps", "euler", "kg", 3, 7, 13, "warped"),
        # adapted grid with hanging faces, small enough for the L2 cache: many short launches
        _case("euler3d_kg_n5_adapted_fp32bulk", "steps", "euler", "kg", 3, 5, 4, "adapted", "fp32_bulk", 20),
        # 3-D advection at the headline size: one field, bytes only
        _case("adv3d_weak_n7_32_fp64", "steps", "adv", "weak", 3, 7, 32),
        # a weak-form 3-D Euler operator at even order, ragged size
        _case("euler3d_weak_n6_15", "steps", "euler", "weak", 3, 6, 15),
        # sixteen independent solves of mixed dimension, order, size and law served together
        dict(do="serve", mix=4, solves=16, steps=40, precision="fp32_bulk", name="serve_mix_16"),
    ]


def draw(rng):
    """One more case of the ranges above: elements per side log-uniform up to 16.8 M nodes
    (2-D 4..128, 3-D 3..32; warped, whose metrics the host computes, to 14), N = 3..7."""
    do = rng.choice(["steps"] * 12 + ["tendency"] * 3 + ["serve"])
    if do == "serve":
        return dict(do="serve", mix=rng.randrange(1 << 20), solves=rng.randint(6, 16), steps=rng.randint(15, 40),
                    precision="fp32_bulk")
    dim = rng.choice([2, 3, 3])
    law = rng.choice(["euler", "euler", "euler", "adv"])
    form = "weak" if law == "adv" else rng.choice(["kg", "kg", "ec", "weak"])
    N = rng.choice([3, 4, 5, 6, 7, 7])
    grid = rng.choice(["brick"] * 3 + ["warped"]) if form == "kg" else "brick"
    lo, hi = (4, 128) if dim == 2 else (3, 14 if grid == "warped" else 32)
    K = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    precision = rng.choice(["fp64", "fp32_bulk"])
    nodes = K**dim * (N + 1) ** dim
    steps = 1 if do == "tendency" else max(1, min(rng.choice([1, 2, 5, 10, 50]), int(1e7 / nodes)))
    return _case(None, do, law, form, dim, N, K, grid, precision, steps)


# ----------------------------------------------------------------------- nodes and states


@functools.lru_cache(maxsize=None)
def _lobatto(nq):
    """LGL nodes, weights and the derivative matrix D[i, j] = l_j'(r_i) (numpy, 64 bits)."""
    N = nq - 1
    P = np.polynomial.legendre.Legendre.basis(N)
    dP, ddP = P.deriv(), P.deriv(2)
    x = -np.cos(np.pi * np.arange(nq) / N)
    for _ in range(50):
        x[1:-1] -= dP(x[1:-1]) / ddP(x[1:-1])
    x = (x - x[::-1]) / 2
    w = 2 / (N * nq * P(x) ** 2)
    lam = np.array([1 / np.prod(x[j] - np.delete(x, j)) for j in range(nq)])
    D = np.zeros((nq, nq))
    for i in range(nq):
        for j in range(nq):
            if i != j:
                D[i, j] = lam[j] / lam[i] / (x[i] - x[j])
    D[0, 0], D[N, N] = -N * nq / 4, N * nq / 4
    return x, w, D


def _morton(xyz, dim):
    key = np.zeros(xyz.shape[1], dtype=np.int64)
    for b in range(16):
        for d in range(dim):
            key |= ((xyz[d] >> b) & 1) << (dim * b + d)
    return key


@functools.lru_cache(maxsize=4)
def _lattice(dim, K, adapted):
    """The elements in the grid's order: lower corners in units of the finest element and
    levels.  A brick is one level; the adapted grid has K^dim trees refined twice within a
    quarter side of the centre, and a tree that touches the finest level refined once."""
    fine = 4 if adapted else 1
    cells = np.array(np.meshgrid(*[np.arange(K)] * dim, indexing="ij")).reshape(dim, -1)
    if not adapted:
        xyz, lev = cells, np.zeros(cells.shape[1], dtype=np.int64)
    else:
        def near(c, h):  # boxes of side h (in trees) closer to the centre than K/4
            q = np.clip(K / 2, c * h, (c + 1) * h)
            return ((K / 2 - q) ** 2).sum(0) < (K / 4) ** 2

        def split(c):
            kids = np.array(np.meshgrid(*[[0, 1]] * dim, indexing="ij")).reshape(dim, 1, -1)
            return (2 * c[:, :, None] + kids).reshape(dim, -1)

        ref = near(cells, 1.0)
        one = split(cells[:, ref])
        ref1 = near(one, 0.5)
        two = split(one[:, ref1])
        # 2:1 balance: a level-0 cell with a level-2 cell across a face is split
        finest = {tuple(c) for c in two.T}
        touch = np.zeros(cells.shape[1], dtype=bool)
        for i in np.nonzero(~ref)[0]:
            lo = cells[:, i] * 4
            for f in range(2 * dim):
                d, side = divmod(f, 2)
                r = [range(lo[e], lo[e] + 4) for e in range(dim)]
                r[d] = [(lo[d] + (4 if side else -1)) % (4 * K)]
                touch[i] |= any(tuple(c) in finest for c in np.array(np.meshgrid(*r)).reshape(dim, -1).T)
        zero = cells[:, ~ref & ~touch]
        one = np.concatenate([one[:, ~ref1], split(cells[:, touch])], axis=1)
        xyz = np.concatenate([zero * 4, one * 2, two], axis=1)
        lev = np.repeat([0, 1, 2], [zero.shape[1], one.shape[1], two.shape[1]])
    order = np.argsort(_morton(xyz, dim), kind="stable")
    return xyz[:, order], lev[order], fine


def _box(case):
    return 10.0 if case["law"] == "euler" and case["grid"] != "adapted" else 1.0


def _points(case, device):
    """Node coordinates, a list of dim tensors (E, Np)."""
    dim, nq, L = case["dim"], case["N"] + 1, _box(case)
    xyz, lev, fine = _lattice(dim, case["K"], case["grid"] == "adapted")
    h = L / (case["K"] * 2.0 ** torch.as_tensor(lev, device=device, dtype=torch.float64))
    r = torch.as_tensor(_lobatto(nq)[0], device=device)
    X = []
    for d in range(dim):
        lo = torch.as_tensor(xyz[d], device=device, dtype=torch.float64) * (L / (case["K"] * fine))
        x = lo[:, None] + h[:, None] * ((r[None, :] + 1) / 2)
        shape = [1] * dim
        shape[dim - 1 - d] = nq
        X.append(x.reshape([-1] + shape).expand([-1] + [nq] * dim).reshape(len(lev), -1))
    if case["grid"] == "warped":
        X = _warp(L)(*X)
    return X


def _warp(L):
    """x' = x + 0.1 L sin(pi x / L) sin(pi y / L) [sin(pi z / L)] in every direction."""

    def warp(*x):
        lib = torch if isinstance(x[0], torch.Tensor) else np
        s = 1.0
        for v in x:
            s = s * lib.sin(math.pi * (v / L))
        return [v + (0.1 * L) * s for v in x]

    return warp


def _modes(rng, X, L, count=3):
    """A smooth periodic perturbation of size 1: a few random Fourier modes."""
    s = 0.0
    for _ in range(count):
        phase = 2 * math.pi * rng.random()
        for x in X:
            phase = phase + (2 * math.pi / L * rng.choice([-2, -1, 1, 2])) * x
        s = s + torch.sin(phase) / count
    return s


def _initial(case, seed, device="cuda"):
    """Initial data (E, Ns, Np).  Euler: an isentropic vortex carried by a background of
    Mach 0.3-0.6 (adapted grid: a density pulse), advection: a sine and a Gaussian; the
    seed sets place, strength and direction, and smooth perturbations along all directions."""
    rng = random.Random(seed)
    dim, L = case["dim"], _box(case)
    X = _points(case, device)
    if case["law"] == "adv":
        q = 0.1 * _modes(rng, X, L)
        s, r2 = 1.0, 0.0
        for x in X:
            s = s * torch.sin(2 * math.pi * (x / L + rng.random()))
            r2 = r2 + (x - L * rng.uniform(0.4, 0.6)) ** 2
        return (q + s + torch.exp(-r2 / (2 * (0.05 * L) ** 2)))[:, None, :].contiguous()
    speed, angle = rng.uniform(0.3, 0.6) * math.sqrt(GAMMA), rng.uniform(0, 2 * math.pi)
    u = [speed * math.cos(angle) + 0.01 * _modes(rng, X, L), speed * math.sin(angle) + 0.01 * _modes(rng, X, L)]
    if dim == 3:
        u.append(0.05 * _modes(rng, X, L))
    if case["grid"] == "adapted":
        r2 = sum((x - L * rng.uniform(0.45, 0.55)) ** 2 for x in X)
        rho = 1 + rng.uniform(0.1, 0.2) * torch.exp(-r2 / 0.01) + 0.01 * _modes(rng, X, L)
        p = 1 + 0.01 * _modes(rng, X, L)
    else:
        beta = rng.uniform(0.8, 1.6)
        r0, r1 = X[0] - L * rng.uniform(0.4, 0.6), X[1] - L * rng.uniform(0.4, 0.6)
        f = beta * torch.exp(1 - (r0 * r0 + r1 * r1))
        rho = (1 - (GAMMA - 1) * f * f / (16 * GAMMA * math.pi**2)) ** (1 / (GAMMA - 1))
        p = rho**GAMMA * (1 + 0.01 * _modes(rng, X, L))
        u[0] = u[0] - f * r1 / (2 * math.pi)
        u[1] = u[1] + f * r0 / (2 * math.pi)
    E = p / (GAMMA - 1) + rho * sum(v * v for v in u) / 2
    return torch.stack([rho] + [rho * v for v in u] + [E], dim=1)


def _dt(case):
    r = _lobatto(case["N"] + 1)[0]
    h = _box(case) / case["K"] / (4 if case["grid"] == "adapted" else 1)
    dmin = h * (r[1] - r[0]) / 2 * (0.6 if case["grid"] == "warped" else 1.0)
    return 0.4 * dmin / (2.8 if case["law"] == "euler" else math.hypot(*ADV_VELOCITY[: case["dim"]]))


# ------------------------------------------------------------------------- prepare and run


@functools.lru_cache(maxsize=1)
def _grid(dim, N, K, kind, L):
    """The generated grid, which a program keeps while it solves on it."""
    rb = _package()
    coords = tuple(rb.jl_range(0.0, L, K + 1) for _ in range(dim))
    gm = rb.GridManager(rb.LobattoCell(*([N + 1] * dim)), rb.brick(coords, (True,) * dim))
    if kind == "adapted":
        from raven_b200.forest import sphere_refinement_flags

        for _ in range(2):
            rb.adapt(gm, sphere_refinement_flags(gm.forest, coords, (L / 2,) * dim, L / 4))
    return rb.generate(_warp(L), gm) if kind == "warped" else rb.generate(gm)


def _solves(case):
    """The batch of a serving case: laws, dimensions, orders, sizes and step counts drawn
    from the case alone (2-D 8..40 and 3-D 4..14 elements per side)."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["solves"]):
        dim, law = rng.choice([2, 3]), rng.choice(["adv", "euler"])
        lo, hi = (8, 40) if dim == 2 else (4, 14)
        K = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        out.append({"law": law, "form": "kg" if law == "euler" else "weak", "dim": dim, "N": rng.choice([3, 5, 7]),
                    "K": K, "grid": "brick", "precision": case["precision"],
                    "steps": rng.randint(case["steps"] // 2, case["steps"])})
    return out


def prepare(case, seed):
    rb = _package()
    if case["do"] == "serve":
        from raven_b200 import serving

        specs = []
        for i, c in enumerate(_solves(case)):
            dim, L = c["dim"], _box(c)
            q0 = _initial(c, 1000 * seed + i).cpu().numpy().transpose(2, 1, 0)
            specs.append(serving.SolveSpec(
                dim=dim, nq=c["N"] + 1, law=rb.AdvectionLaw.code if c["law"] == "adv" else rb.EulerLaw.code,
                K=(c["K"],) * dim, lo=(0.0,) * dim, hi=(L,) * dim, nsteps=c["steps"], dt=_dt(c),
                precision=rb._lib.PRECISION_FP32_BULK, gamma=GAMMA, advection_velocity=ADV_VELOCITY[:dim],
                q0=np.asfortranarray(q0)))
        return {"do": "serve", "server": serving.Server(arena_bytes=2 << 30), "specs": specs}
    dim = case["dim"]
    law = rb.AdvectionLaw(dim, ADV_VELOCITY[:dim]) if case["law"] == "adv" else rb.EulerLaw(dim, gamma=GAMMA)
    form = {"weak": rb.WeakForm, "kg": lambda: rb.FluxDifferencingForm(rb.KennedyGruberFlux()),
            "ec": lambda: rb.FluxDifferencingForm(rb.EntropyConservativeFlux())}[case["form"]]()
    grid = _grid(dim, case["N"], case["K"], case["grid"], _box(case))
    dg = rb.DGSEM(law=law, grid=grid, volume_form=form, surface_numericalflux=rb.RusanovFlux(),
                  precision=case["precision"])
    q = rb.GridArray(_initial(case, seed), law.ns, grid.np, grid.E)
    return {"do": case["do"], "steps": case["steps"], "dg": dg, "q": q, "dq": q.similar(),
            "solver": rb.LSRK54(dg, q, _dt(case))}


def run(state):
    if state["do"] == "serve":
        tickets = [state["server"].submit(s) for s in state["specs"]]
        return [state["server"].wait(t)[0] for t in tickets]
    dg, q = state["dg"], state["q"]
    if state["do"] == "tendency":
        return dg(state["dq"], q, 0.0, increment=False).data
    solver = state["solver"]
    solver.dostep(q, state["steps"])
    out = [q.data] + ([solver.dq.data] if dg.precision == "fp64" else [])
    if state["do"] == "steps+norm":
        out.append(_package().weightednorm(dg, q))
    return out


def work(case):
    """Bytes and flops of one pass.  A state that fits the L2 cache is read and written
    once; a larger one is read and written by each stage, with the register (not read by
    the first stage) and, on warped grids, the metrics (9 + 1 doubles a node and 4 a face
    node)."""
    if case["do"] == "serve":
        parts = [work(dict(c, do="steps")) for c in _solves(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    dim, nq, grid = case["dim"], case["N"] + 1, case["grid"]
    nodes = _lattice(dim, case["K"], grid == "adapted")[0].shape[1] * nq**dim
    ns = 1 if case["law"] == "adv" else dim + 2
    reg = 8 if case["precision"] == "fp64" else 4
    pair = {"weak": 2 * ns, "kg": 20, "ec": 40}[case["form"]]
    flops = nodes * (dim * (nq - 1) * pair + (2 * dim / nq) * (8 if ns == 1 else 80) + 10 * ns)
    geo = (8 * (dim * dim + 1) + 16 * dim * (dim + 1) / nq) if grid == "warped" else 0
    if case["do"] == "tendency":
        return {"bytes": nodes * (16 * ns + geo), "flops": flops}
    stages = 5 * case["steps"]
    once = nodes * (16 + 2 * reg) * ns + nodes * geo
    per_stage = nodes * ((16 + reg + 0.8 * reg) * ns + geo)
    return {"bytes": once if once < L2_BYTES else stages * per_stage, "flops": stages * flops}


# ----------------------------------------------------------- the same results in 64 bits

_RKA = [0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
        -1275806237668 / 842570457699]
_RKB = [1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
        3134564353537 / 4481467310338, 2277821191437 / 14882151754819]


class _Plain:
    """The scheme of a case with plain torch operations in 64 bits.  Fields are tensors
    (E, nq, .., nq), x the last axis; directions d = 0, 1, 2 are the axes -1, -2, -3."""

    def __init__(self, case, device="cuda"):
        self.case, self.dim, self.nq = case, case["dim"], case["N"] + 1
        dim, nq = self.dim, self.nq
        r, w, D = _lobatto(nq)
        self.w, self.D = torch.as_tensor(w, device=device), torch.as_tensor(D, device=device)
        xyz, lev, fine = _lattice(dim, case["K"], case["grid"] == "adapted")
        self.E = len(lev)
        self.shape = (self.E,) + (nq,) * dim
        W = self.along(self.w, 0)
        for d in range(1, dim):
            W = W * self.along(self.w, d)
        h = torch.as_tensor(_box(case) / (case["K"] * 2.0**lev), device=device).reshape((-1,) + (1,) * dim)
        if case["grid"] == "warped":
            self.Ja, J = self.curved([x.reshape(self.shape) for x in _points(case, device)])
        else:  # J a^dir on the diagonal
            J = (h / 2) ** dim
            self.Ja = [[(J * 2 / h) if c == d else None for c in range(dim)] for d in range(dim)]
        self.W, self.MJI = W, 1 / (W * J)
        self.connect(xyz, lev, fine, device)

    def along(self, v, d):
        shape = [1] * (self.dim + 1)
        shape[-1 - d] = -1
        return v.reshape(shape)

    def diff(self, f, d):
        return torch.movedim(torch.movedim(f, -1 - d, -1) @ self.D.T, -1, -1 - d)

    def curved(self, X):
        """J a^dir_c of the mapping (3-D: curl-invariant form) and J."""
        if self.dim == 2:
            xr, xs, yr, ys = self.diff(X[0], 0), self.diff(X[0], 1), self.diff(X[1], 0), self.diff(X[1], 1)
            return [[ys, -xs], [-yr, xr]], xr * ys - yr * xs

        def cross(a, b):
            return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]

        dX = [[self.diff(x, d) for x in X] for d in range(3)]
        C = [cross(X, dX[d]) for d in range(3)]
        Ja = []
        for d in range(3):
            e, f = (d + 1) % 3, (d + 2) % 3
            Ja.append([(self.diff(C[f][c], e) - self.diff(C[e][c], f)) / 2 for c in range(3)])
        s = cross(dX[1], dX[2])
        return Ja, sum(dX[0][c] * s[c] for c in range(3))

    def connect(self, xyz, lev, fine, device):
        """Same-size neighbours per face, and per face direction the hanging faces: large
        element and its 2^(dim-1) small neighbours (first in-face direction fastest)."""
        n = self.case["K"] * fine
        where = {(int(l),) + tuple(int(v) for v in c): i for i, (l, c) in enumerate(zip(lev, xyz.T))}
        self.nbr, self.hang = [], []
        for f in range(2 * self.dim):
            d, side = divmod(f, 2)
            same, large, small = [], [], []
            for i in range(self.E):
                size = fine >> int(lev[i])
                c = [int(v) for v in xyz[:, i]]
                c[d] = (c[d] + (size if side else -size)) % n
                same.append(where.get((int(lev[i]),) + tuple(c), -1))
                if same[-1] < 0 and size > 1:
                    half = size // 2
                    c[d] = (c[d] + (0 if side else half)) % n
                    inface = [e for e in range(self.dim) if e != d]
                    kids = []
                    for b in range(1 << (self.dim - 1)):
                        k = list(c)
                        for m, e in enumerate(inface):
                            k[e] = (k[e] + half * ((b >> m) & 1)) % n
                        kids.append(where.get((int(lev[i]) + 1,) + tuple(k), -1))
                    if min(kids) >= 0:
                        large.append(i)
                        small.append(kids)
            self.nbr.append(torch.tensor(same, device=device))
            self.hang.append((torch.tensor(large, device=device), torch.tensor(small, device=device)) if large else None)
        if any(self.hang):
            r = _lobatto(self.nq)[0]
            w = self.w.cpu().numpy()

            def to_half(shift):
                t = (r + shift) / 2
                I = np.ones((self.nq, self.nq))
                for j in range(self.nq):
                    for k in range(self.nq):
                        if k != j:
                            I[:, j] *= (t - r[k]) / (r[j] - r[k])
                return I

            self.half = [torch.as_tensor(to_half(s), device=device) for s in (-1, 1)]
            self.back = [torch.as_tensor((to_half(s) * w[:, None] / (2 * w[None, :])).T.copy(), device=device)
                         for s in (-1, 1)]

    # -- physics
    def prim(self, q):
        rho, m, E = q[0], q[1:-1], q[-1]
        u = [v / rho for v in m]
        return rho, u, E, (GAMMA - 1) * (E - sum(v * w for v, w in zip(m, u)) / 2)

    def normal_flux(self, q, n):
        """Flux in direction n (a list; None: component 0) and the fastest wave speed."""
        if self.case["law"] == "adv":
            an = sum(a * c for a, c in zip(ADV_VELOCITY, n) if c is not None)
            return [an * q[0]], an.abs()
        rho, u, E, p = self.prim(q)
        un = sum(v * c for v, c in zip(u, n) if c is not None)
        F = [rho * un] + [rho * un * v + (p * c if c is not None else 0) for v, c in zip(u, n)] + [un * (E + p)]
        return F, un.abs() + torch.sqrt(GAMMA * p / rho)

    def rusanov(self, qm, qp, n):
        (Fm, cm), (Fp, cp) = self.normal_flux(qm, n), self.normal_flux(qp, n)
        c = torch.maximum(cm, cp)
        return [(a + b) / 2 - c * (y - x) / 2 for a, b, x, y in zip(Fm, Fp, qm, qp)]

    @staticmethod
    def logmean(a, b):
        f = (a - b) / (a + b)
        u = f * f
        s = torch.zeros_like(u)
        for k in range(9, -1, -1):
            s = s * u + 1 / (2 * k + 1)
        return (a + b) / (2 * torch.where(u < 0.01, s, torch.log(a / b) / (2 * torch.where(f == 0, 1.0, f))))

    def two_point(self, a, b, G):
        """Symmetric two-point flux of primitives a, b contracted with G (KG or EC)."""
        (r1, u1, E1, p1), (r2, u2, E2, p2) = a, b
        ub = [(v + w) / 2 for v, w in zip(u1, u2)]
        un = sum(v * g for v, g in zip(ub, G) if g is not None)
        if self.case["form"] == "kg":
            rb, eb, pb = (r1 + r2) / 2, (E1 / r1 + E2 / r2) / 2, (p1 + p2) / 2
            f = rb * un
            return [f] + [f * v + (pb * g if g is not None else 0) for v, g in zip(ub, G)] + [un * (rb * eb + pb)]
        b1, b2 = r1 / (2 * p1), r2 / (2 * p2)
        rl, bl = self.logmean(r1, r2), self.logmean(b1, b2)
        pt = (r1 + r2) / (2 * (b1 + b2))
        uu = sum(v * v + w * w for v, w in zip(u1, u2)) / 2
        f = rl * un
        e = 1 / (2 * (GAMMA - 1) * bl) - uu / 2 + sum(v * v for v in ub)
        return [f] + [f * v + (pt * g if g is not None else 0) for v, g in zip(ub, G)] + [un * (rl * e + pt)]

    # -- operators
    def rhs(self, q):
        dim, nq = self.dim, self.nq
        ns = len(q)
        acc = [torch.zeros(self.shape, dtype=torch.float64, device=q[0].device) for _ in range(ns)]
        weak = self.case["form"] == "weak"
        pr = None if weak else self.prim(q)
        for d in range(dim):
            ax = -1 - d
            lg = [None if g is None else self.W * g for g in self.Ja[d]]
            if weak:
                F, _ = self.normal_flux(q, lg)
                for s in range(ns):
                    acc[s] += torch.movedim(torch.movedim(F[s], ax, -1) @ self.D, -1, ax)
                continue

            def at(f, a):
                return f.narrow(ax, a, 1)

            for a in range(nq):
                Dai, Dia = self.along(self.D[a], d), self.along(self.D[:, a], d)
                G = [None if g is None else Dai * at(g, a) - Dia * g for g in lg]
                part = (at(pr[0], a), [at(v, a) for v in pr[1]], at(pr[2], a), at(pr[3], a))
                for s, f in enumerate(self.two_point(pr, part, G)):
                    acc[s] += f
        acc = [v * self.MJI for v in acc]
        for f in range(2 * dim):
            self.face(q, acc, f)
        return acc

    def face(self, q, acc, f):
        dim, nq = self.dim, self.nq
        d, side = divmod(f, 2)
        ax, end = -1 - d, (nq - 1 if side else 0)
        sn = 1.0 if side else -1.0

        def trace(v, at):
            return v.select(ax, at if v.shape[ax] > 1 else 0)

        Ja = [None if g is None else sn * trace(g, end) for g in self.Ja[d]]
        sJ = torch.sqrt(sum(g * g for g in Ja if g is not None))
        n = [None if g is None else g / sJ for g in Ja]
        scale = sJ * trace(self.W, end) / self.w[end] * trace(self.MJI, end)
        qm = [trace(v, end) for v in q]
        nb = self.nbr[f]
        ok = (nb >= 0).reshape((-1,) + (1,) * (dim - 1))
        qp = [torch.where(ok, trace(v, nq - 1 - end)[nb.clamp(min=0)], m) for v, m in zip(q, qm)]
        flux = self.rusanov(qm, qp, n)
        if self.hang[f] is not None:
            large, small = self.hang[f]
            self.mortar(q, flux, n, large, small, d, end, +1)
        if self.hang[f ^ 1] is not None:  # this face of the small elements
            large, small = self.hang[f ^ 1]
            self.mortar(q, flux, n, large, small, d, nq - 1 - end, -1)
        for s in range(len(q)):
            acc[s].select(ax, end).sub_(scale * flux[s])

    def mortar(self, q, flux, n, large, small, d, end, sign):
        """Fluxes of hanging faces: `end` is the large side's end of direction d; sign +1
        writes the large faces, -1 the small ones (whose normal n is the opposite)."""
        ax = -1 - d
        total = None
        for b in range(small.shape[1]):
            kid = small[:, b]
            bits = [(b >> m) & 1 for m in range(self.dim - 1)]

            def apply(op, v):  # first in-face direction is the last axis
                for m, bit in enumerate(bits):
                    v = torch.movedim(torch.movedim(v, -1 - m, -1) @ op[bit].T, -1, -1 - m)
                return v

            ql = [apply(self.half, v.select(ax, end)[large]) for v in q]
            qs = [v.select(ax, self.nq - 1 - end)[kid] for v in q]
            who = large if sign > 0 else kid
            nn = [None if g is None else sign * (g[who] if g.shape[0] > 1 else g) for g in n]
            F = self.rusanov(ql, qs, nn)
            if sign < 0:
                for s in range(len(q)):
                    flux[s][kid] = -F[s]
            else:
                part = [apply(self.back, v) for v in F]
                total = part if total is None else [x + y for x, y in zip(total, part)]
        if sign > 0:
            for s in range(len(q)):
                flux[s][large] = total[s]

    def steps(self, q, n, dt):
        dq = [torch.zeros_like(v) for v in q]
        for _ in range(n):
            for a, b in zip(_RKA, _RKB):
                k = self.rhs(q)
                dq = [a * x + y for x, y in zip(dq, k)]
                q = [x + (b * dt) * y for x, y in zip(q, dq)]
        return q, dq

    def load(self, q):
        return [q[:, s].reshape(self.shape) for s in range(q.shape[1])]

    def pack(self, q):
        return torch.stack([v.reshape(self.E, -1) for v in q], dim=1)

    def norm(self, q):
        m = 1 / self.MJI
        return math.sqrt(sum(float((m * v * v).sum()) for v in q))


def exact(case, seed):
    if case["do"] == "serve":
        out = []
        for i, c in enumerate(_solves(case)):
            p = _Plain(c)
            q, _ = p.steps(p.load(_initial(c, 1000 * seed + i)), c["steps"], _dt(c))
            out.append(p.pack(q).cpu().numpy().transpose(2, 1, 0))
        return out
    p = _Plain(case)
    q = p.load(_initial(case, seed))
    if case["do"] == "tendency":
        return p.pack(p.rhs(q))
    q, dq = p.steps(q, case["steps"], _dt(case))
    out = [p.pack(q)] + ([p.pack(dq)] if case["precision"] == "fp64" else [])
    if case["do"] == "steps+norm":
        out.append(p.norm(q))
    return out

"""Performance cases of the solver: what its users have it do, through the public entry points.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare(case, seed)`
makes what a program holds before the call (mesh, solver handle, inputs on the GPU, or in
pinned host memory where the call takes host arrays), `run(state)` is one pass, `work(case)`
the bytes and operations that a pass cannot do without and `exact(case, seed)` the same
outputs computed in 64 bits by plain torch.

Kinds of work:

  solve     Multigrid.solve_vcycle: one complete solve to a relative residual of 1e-10.  The
            precisions are the plain FP64 path, the FP64 performance mode and mixed precision.
  batch     BatchSolver.solve: many independent boxes of uneven sizes.
  autograd  PoissonSolve: a differentiable solve and its backward pass (the adjoint solve).
  smooth    Multigrid.rbgs_iterator: red-black sweeps on one level, as a user's own cycle or
            smoother calls them.
  transfer  Multigrid.residual, restriction and prolong_add between two levels, as a user's
            own cycle calls them.
  cg        Multigrid.cg_iterator: conjugate-gradient iterations on one level.
"""
import math

import numpy as np
import torch

import peps_mg_gb300 as pmg

TOL = 1e-10


# ---------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------
def _solve(nx, ny, nz, levels, precision, mesh, method="cgs", inner=0, omega=1.0, warm=False, host=False):
    return {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "levels": levels, "precision": precision, "mesh": mesh,
            "method": method, "inner": inner, "omega": omega, "warm": warm, "host": host}


def listed():
    return [
        # The small benchmark problem in plain FP64: a latency-bound solve, such as the
        # pressure step of a small simulation.
        dict(_solve(64, 64, 64, 4, "fp64", "uniform"), name="solve_64_fp64"),
        # Wall-bounded flow: z clustered at both walls, coarse levels aggregated.
        dict(_solve(256, 256, 256, 7, "fp64", "tanh_z", method="cga"), name="solve_256_tanh_fp64"),
        # The headline: a 512^3 box in mixed precision, four FP32 cycles per correction.
        dict(_solve(512, 512, 512, 8, "mixed", "uniform", inner=4), name="solve_512_mixed"),
        # A time step of a simulation on a stretched box of uneven sides: the last step's
        # solution as initial guess, non-zero Dirichlet faces, default cycle count.
        dict(_solve(224, 160, 96, 5, "mixed", "stretched", warm=True), name="solve_ragged_mixed"),
        # The FP64 performance mode on an ordinary box.
        dict(_solve(320, 256, 192, 6, "fp64_fast", "uniform"), name="solve_320_fast"),
        # A host program (the Fortran caller's situation) whose arrays stay in pinned memory.
        dict(_solve(256, 192, 128, 5, "mixed", "uniform", inner=4, host=True), name="solve_host_mixed"),
        # The 128-problem batch of uneven boxes.
        dict({"kind": "batch", "count": 128, "inner": 4, "pick": 4}, name="batch_128"),
        # Learning and inverse problems: forward solve and gradients.
        dict({"kind": "autograd", "nx": 256, "ny": 256, "nz": 256, "levels": 7, "mesh": "uniform", "inner": 4},
             name="autograd_256_mixed"),
        # The smallest call: two over-relaxed sweeps on a small odd box.
        dict({"kind": "smooth", "nx": 63, "ny": 47, "nz": 31, "mesh": "stretched", "omega": 1.2, "iters": 2},
             name="smooth_small_odd"),
        # The smoother on a large level.
        dict({"kind": "smooth", "nx": 384, "ny": 384, "nz": 384, "mesh": "uniform", "omega": 1.0, "iters": 2},
             name="smooth_384"),
        # The level operations of a user's own cycle on a stretched box.
        dict({"kind": "transfer", "nx": 324, "ny": 258, "nz": 194, "mesh": "stretched"}, name="transfer_324"),
        # Conjugate gradients on an ordinary level.
        dict({"kind": "cg", "nx": 224, "ny": 160, "nz": 128, "mesh": "stretched", "iters": 16}, name="cg_224"),
    ]


def _cells(c):
    return c["nx"] * c["ny"] * c["nz"]


def draw(rng):
    """One more case: a kind, then sizes spread over its range (by their logarithm)."""
    kind = rng.choice(["solve", "solve", "solve", "batch", "autograd", "smooth", "transfer", "cg"])
    mesh = rng.choice(["uniform", "stretched", "tanh_z"])

    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "batch":
        return {"kind": "batch", "count": side(4, 128), "inner": rng.choice([2, 3, 4]), "pick": rng.randrange(1 << 20)}
    if kind in ("smooth", "transfer", "cg"):
        cap = {"smooth": 384 ** 3, "transfer": 352 ** 3, "cg": 192 ** 3}[kind]
        while True:
            n = [side(20, 448) for _ in range(3)]
            if kind == "transfer":
                n = [2 * (m // 2) for m in n]
            c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "mesh": mesh}
            if _cells(c) <= cap:
                break
        if kind == "smooth":
            c.update(omega=rng.choice([1.0, 1.0, 1.2, 1.5]), iters=rng.choice([1, 2, 3]))
        if kind == "cg":
            c.update(iters=rng.randrange(4, 24))
        return c
    # whole solves: sides m 2^L, so that the coarsest level is a few cells wide
    precision = "mixed" if kind == "autograd" else rng.choice(["fp64", "mixed", "mixed", "fp64_fast"])
    cap = {"fp64": 224 ** 3, "fp64_fast": 288 ** 3, "mixed": 416 ** 3}[precision]
    if kind == "autograd":
        cap = 256 ** 3
    while True:
        levels = rng.randrange(3, 8)
        n = [rng.choice([2, 3, 4, 5]) << levels for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        if 24 ** 3 <= cells <= cap and max(n) <= 2.5 * min(n):
            break
    if kind == "autograd":
        return {"kind": "autograd", "nx": n[0], "ny": n[1], "nz": n[2], "levels": levels, "mesh": mesh,
                "inner": rng.choice([2, 3, 4])}
    return _solve(n[0], n[1], n[2], levels, precision, mesh, method=rng.choice(["cgs", "cga"]),
                  inner=rng.choice([2, 3, 4]) if precision == "mixed" else 0, omega=rng.choice([1.0, 1.0, 1.15]),
                  warm=rng.random() < 0.4, host=cells <= 7e6 and rng.random() < 0.25)


# ---------------------------------------------------------------------------------------
# Meshes and inputs
# ---------------------------------------------------------------------------------------
def _axis(n, kind, length):
    """(dm, dg, xg) of one axis, 0..n+1, ghosts of zero width: the reference's mesh form."""
    if kind == "stretched":        # symmetric geometric stretch, adjacent widths within 1.5%
        d = np.minimum(np.arange(n), np.arange(n)[::-1]).astype(np.float64)
        w = 1.015 ** np.minimum(d, 40.0)
    elif kind == "tanh":           # clustered at both ends
        f = np.tanh(1.5 * (2.0 * np.arange(n + 1) / n - 1.0))
        w = np.diff(f)
    else:
        w = np.ones(n)
    dm = np.zeros(n + 2)
    dm[1:-1] = w * (length / w.sum())
    dg = np.zeros(n + 2)
    dg[1:] = 0.5 * (dm[1:] + dm[:-1])
    xg = np.cumsum(dg)
    return dm, dg, xg


def _mesh(c):
    n = (c["nx"], c["ny"], c["nz"])
    longest = float(max(n))        # nearly cubic cells: each side as long as its cell count
    kinds = {"uniform": ("u", "u", "u"), "stretched": ("stretched",) * 3, "tanh_z": ("u", "u", "tanh")}[c["mesh"]]
    return [_axis(m, k, m / longest) for m, k in zip(n, kinds)]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _field(c):
    return torch.zeros((c["nz"] + 2, c["ny"] + 2, c["nx"] + 2), dtype=torch.float64, device="cuda")


def _random(c, seed, ghosts=False):
    a = _field(c)
    g = _generator(seed)
    if ghosts:
        a.copy_(2.0 * torch.rand(a.shape, dtype=torch.float64, device="cuda", generator=g) - 1.0)
    else:
        i = a[1:-1, 1:-1, 1:-1]
        i.copy_(2.0 * torch.rand(i.shape, dtype=torch.float64, device="cuda", generator=g) - 1.0)
    return a


def _sources(c, mesh, seed):
    """A right-hand side of eight Gaussian sources (amplitudes of both signs) and a little noise."""
    b = 1e-3 * _random(c, seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    x = [torch.as_tensor(m[2][1:-1] / m[2][-1], device="cuda") for m in mesh]
    for _ in range(8):
        centre, amp = rng.uniform(0.1, 0.9, 3), float(rng.uniform(-10.0, 10.0))
        gx, gy, gz = (torch.exp(-(v - p) ** 2 / (2 * 0.05 ** 2)) for v, p in zip(x, centre))
        b[1:-1, 1:-1, 1:-1] += (amp * gz)[:, None, None] * (gy[None, :, None] * gx[None, None, :])
    return b


def _set_faces(a, g):
    for face, v in zip((a[:, :, 0], a[:, :, -1], a[:, 0, :], a[:, -1, :], a[0], a[-1]), g):
        face.fill_(float(v))


def _faces(seed):
    return np.random.Generator(np.random.PCG64(seed + 7)).uniform(-0.5, 0.5, 6)


def _guess(c, mesh, seed):
    """The initial guess: zero, or (warm) a smooth field with non-zero Dirichlet faces."""
    a = _field(c)
    if c["warm"]:
        _set_faces(a, _faces(seed))
        s = [torch.sin(math.pi * torch.as_tensor(m[2][1:-1] / m[2][-1], device="cuda")) for m in mesh]
        amp = 0.1 + 0.01 * (seed % 7)
        a[1:-1, 1:-1, 1:-1] = amp * s[2][:, None, None] * s[1][None, :, None] * s[0][None, None, :]
    return a


_BATCH_SIDES = (32, 48, 64, 96, 128, 192)


def _batch_dims(c):
    r = np.random.Generator(np.random.PCG64(c["pick"]))
    return r.choice(np.asarray(_BATCH_SIDES), size=(c["count"], 3))


def _handle(c, mesh, vcycles=50):
    method = c.get("method", "cgs")
    levels = c.get("levels", 2)
    return pmg.Multigrid(mesh, levels, vcycles, method, cga_level=max(1, levels - 2) if method == "cga" else 0,
                         precision=c.get("precision", "mixed" if c["kind"] == "autograd" else "fp64"),
                         mixed_inner_cycles=c.get("inner", 0))


def _halved(axis):
    """The axis with every cell split into two halves: its coarse level is the axis again."""
    dm = np.zeros(2 * axis[0].size - 2)
    dm[1:-1] = np.repeat(axis[0][1:-1], 2) * 0.5
    dg = np.zeros_like(dm)
    dg[1:] = 0.5 * (dm[1:] + dm[:-1])
    return dm, dg, np.cumsum(dg)


def _level_handle(c, mesh):
    """(handle, level) with the case's box on that level.  A handle has two coarse levels at
    least and some axis halves at the last one, so a box that cannot be halved far enough is
    itself a coarse level, as the odd boxes of a real hierarchy are."""
    n = (c["nx"], c["ny"], c["nz"])
    level = 0 if any(m % 4 == 0 for m in n) else 1 if any(m % 2 == 0 for m in n) else 2
    if level >= 1:
        mesh = [_halved(m) for m in mesh]
    if level == 2:
        mesh[0] = _halved(mesh[0])
    return pmg.Multigrid(mesh, 2, 1, "cgs", precision="fp64"), level


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        bs = pmg.BatchSolver(_batch_dims(c), mixed_inner_cycles=c["inner"])
        rhs, sol = bs.field(), bs.field()
        for p in range(bs.n):
            v = bs.view(rhs, p)[1:-1, 1:-1, 1:-1]
            v.copy_(2.0 * torch.rand(v.shape, dtype=torch.float64, device="cuda", generator=_generator(seed * 131 + p)) - 1.0)
        return {"case": c, "solver": bs, "sol": sol, "rhs": rhs}
    mesh = _mesh(c)
    if c["kind"] == "solve":
        mg = _handle(c, mesh)
        rhs, guess = _sources(c, mesh, seed), _guess(c, mesh, seed)
        s = {"case": c, "solver": mg, "rhs": rhs, "guess": guess if c["warm"] else None, "sol": torch.zeros_like(rhs),
             "rsd": torch.zeros_like(rhs)}
        if c["host"]:
            for k in ("rhs", "guess", "sol", "rsd"):
                s[k] = None if s[k] is None else s[k].cpu().pin_memory()
        return s
    if c["kind"] == "autograd":
        b, w = _sources(c, mesh, seed), _random(c, seed + 1, ghosts=True)
        g = torch.as_tensor(_faces(seed))
        return {"case": c, "solver": _handle(c, mesh), "b": b.requires_grad_(), "g": g.requires_grad_(), "w": w}
    mg, level = _level_handle(c, mesh)
    s = {"case": c, "solver": mg, "level": level, "b": _random(c, seed), "x0": _random(c, seed + 1, ghosts=True)}
    s["x"] = torch.empty_like(s["x0"])
    if c["kind"] == "transfer":
        coarse = {"nx": c["nx"] // 2, "ny": c["ny"] // 2, "nz": c["nz"] // 2}
        s["r"], s["bc"], s["xc"] = _field(c), _field(coarse), _random(coarse, seed + 2, ghosts=True)
    return s


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    mg = s["solver"]
    if c["kind"] == "batch":
        s["sol"].zero_()
        mg.solve(s["sol"], s["rhs"], 2, TOL, 1.0, max_cycles=50)
        return s["sol"]
    if c["kind"] == "solve":
        if s["guess"] is None:
            s["sol"].zero_()
        else:
            s["sol"].copy_(s["guess"])
        mg.solve_vcycle(s["sol"], s["rsd"], s["rhs"], 2, TOL, c["omega"])
        return {"sol": s["sol"], "rsd": s["rsd"]}
    if c["kind"] == "autograd":
        u = pmg.PoissonSolve.apply(s["b"], s["g"], mg, 2, TOL, 1.0)
        db, dg = torch.autograd.grad(u, (s["b"], s["g"]), s["w"])
        return {"u": u, "db": db, "dg": dg}
    l = s["level"]
    if c["kind"] == "transfer":
        s["x"].copy_(s["x0"])
        mg.residual(l, s["r"], s["x"], s["b"])
        mg.restriction(l, s["bc"], s["r"])
        mg.prolong_add(l, s["x"], s["xc"])
        return {"r": s["r"], "bc": s["bc"], "x": s["x"]}
    s["x"].copy_(s["x0"])
    if c["kind"] == "smooth":
        mg.rbgs_iterator(l, s["x"], s["b"], c["iters"], c["omega"])
    else:
        mg.cg_iterator(l, s["x"], s["b"], c["iters"])
    return s["x"]


# ---------------------------------------------------------------------------------------
# What a pass cannot do without: its inputs read once, its outputs written once, and the
# operations of the algorithm that the call names (a sweep, a cycle), counted per cell
# ---------------------------------------------------------------------------------------
def work(case):
    c = case
    # a V(2,2) cycle: 4 sweeps of 15 operations, a residual of 14, restriction 2 and
    # prolongation 8 per cell, and the coarse levels' 1/7 more
    cycle = (4 * 15 + 14 + 2 + 8) * 8.0 / 7.0
    if c["kind"] == "batch":
        n = float(np.prod(_batch_dims(c).astype(np.float64), axis=1).sum())
        return {"bytes": 24.0 * n, "flops": 11 * cycle * n}              # sol in and out, rhs in
    n = float(_cells(c))
    if c["kind"] == "solve":
        return {"bytes": 32.0 * n, "flops": 11 * cycle * n}              # sol in and out, rhs in, rsd out
    if c["kind"] == "autograd":
        return {"bytes": 32.0 * n, "flops": 22 * cycle * n}              # b, w in; u, db out
    if c["kind"] == "transfer":                                          # r, x read and written once, coarse arrays
        return {"bytes": (8 * 4 + 2.0) * n, "flops": (14 + 2 + 8) * n}
    if c["kind"] == "smooth":
        return {"bytes": 24.0 * n, "flops": 15.0 * c["iters"] * n}
    return {"bytes": 24.0 * n, "flops": 24.0 * c["iters"] * n}           # x in and out, b in


# ---------------------------------------------------------------------------------------
# The outputs in 64 bits, from the definitions
# ---------------------------------------------------------------------------------------
def _modes(dm, dg):
    """Eigenvectors, their inverse and the eigenvalues of the operator along one axis, which
    is symmetric after scaling with the square root of the widths."""
    r = dm.sqrt()
    m = torch.diag(-(1.0 / (dm * dg[:-1]) + 1.0 / (dm * dg[1:])))
    k = torch.arange(dm.numel() - 1, device="cuda")
    m[k, k + 1] = m[k + 1, k] = 1.0 / (dg[1:-1] * r[:-1] * r[1:])
    lam, q = torch.linalg.eigh(m)
    return q / r[:, None], q.T * r[None, :], lam


class _Operator:
    """The seven-point operator of one mesh: (A x)(i) = sum over faces of c (x_neighbour - x_cell)."""

    def __init__(self, mesh):
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.dm = [t(m[0][1:-1]) for m in mesh]
        self.dg = [t(m[1][1:]) for m in mesh]                                # faces 0..n
        shape = [(1, 1, -1), (1, -1, 1), (-1, 1, 1)]
        self.lo = [(1.0 / (d * g[:-1])).view(s) for d, g, s in zip(self.dm, self.dg, shape)]
        self.hi = [(1.0 / (d * g[1:])).view(s) for d, g, s in zip(self.dm, self.dg, shape)]

    @staticmethod
    def sides(x, axis):
        i = [slice(1, -1)] * 3
        lo, hi = list(i), list(i)
        lo[2 - axis], hi[2 - axis] = slice(0, -2), slice(2, None)
        return x[tuple(lo)], x[tuple(hi)]

    def neighbours(self, x):
        out = 0.0
        for a in range(3):
            lo, hi = self.sides(x, a)
            out = out + self.lo[a] * lo + self.hi[a] * hi
        return out

    def diagonal(self):
        return -sum(p + q for p, q in zip(self.lo, self.hi))

    def apply(self, x):
        m = x[1:-1, 1:-1, 1:-1]
        out = 0.0
        for a in range(3):
            lo, hi = self.sides(x, a)
            out = out + self.lo[a] * (lo - m) + self.hi[a] * (hi - m)
        return out

    def factor(self):
        modes = [_modes(dm, dg) for dm, dg in zip(self.dm, self.dg)]
        self.set_modes(modes, 1.0)

    def set_modes(self, modes, scale):
        self.vec, self.inv = [m[0] for m in modes], [m[1] for m in modes]
        lam = [m[2] * scale for m in modes]
        self.lam = lam[2].view(-1, 1, 1) + lam[1].view(1, -1, 1) + lam[0].view(1, 1, -1)

    @staticmethod
    def along(mats, f):
        f = torch.matmul(f, mats[0].T)
        f = torch.matmul(mats[1], f)
        return torch.matmul(mats[2], f.reshape(f.shape[0], -1)).view(f.shape)

    def solve(self, x, b):
        """x with its ghosts kept and its interior the solution of A x = b."""
        if not hasattr(self, "lam"):
            self.factor()
        x[1:-1, 1:-1, 1:-1] = 0.0
        for _ in range(2):         # the second time: refinement
            r = b - self.apply(x)
            x[1:-1, 1:-1, 1:-1] += self.along(self.vec, self.along(self.inv, r) / self.lam)
        return x


def _exact_transfer(c, mesh, s):
    op = _Operator(mesh)
    r = _field(c)
    r[1:-1, 1:-1, 1:-1] = s["b"][1:-1, 1:-1, 1:-1] - op.apply(s["x0"])
    # restriction: the mean of the children, weighted with their widths
    v = r[1:-1, 1:-1, 1:-1]
    for axis in range(3):
        dim, d = 2 - axis, op.dm[axis]
        shape = [1, 1, 1]
        shape[dim] = -1
        lo, hi = d[0::2].view(shape), d[1::2].view(shape)
        i = [slice(None)] * 3
        j = list(i)
        i[dim], j[dim] = slice(0, None, 2), slice(1, None, 2)
        v = (v[tuple(i)] * lo + v[tuple(j)] * hi) / (lo + hi)
    bc = torch.zeros_like(s["bc"])
    bc[1:-1, 1:-1, 1:-1] = v
    # prolongation: linear between coarse centres (the boundary's ghosts lie on the faces)
    v = s["xc"]
    for axis in range(3):
        dim, d = 2 - axis, torch.as_tensor(mesh[axis][0], device="cuda")
        n = d.numel() - 2
        shape = [1, 1, 1]
        shape[dim] = -1
        f = torch.arange(1, n + 1, 2, device="cuda")      # the lower child of each pair
        a, p = d[f - 1] + 0.5 * d[f], 0.5 * d[f]          # own and lower neighbour's weight
        q, e = d[f + 2] + 0.5 * d[f + 1], 0.5 * d[f + 1]  # the upper child's
        own, lo, hi = v.narrow(dim, 1, n // 2), v.narrow(dim, 0, n // 2), v.narrow(dim, 2, n // 2)
        child = torch.stack([(a.view(shape) * own + p.view(shape) * lo) / (a + p).view(shape),
                             (q.view(shape) * own + e.view(shape) * hi) / (q + e).view(shape)], dim=dim + 1)
        v = child.flatten(dim, dim + 1)
        if axis < 2:                                       # the other axes keep their ghosts
            v = v.contiguous()
    x = s["x0"].clone()
    x[1:-1, 1:-1, 1:-1] += v
    return {"r": r, "bc": bc, "x": x}


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        dims = _batch_dims(c)
        cells = np.cumsum([0] + [int(np.prod(d + 2)) for d in dims])
        out, axes = torch.zeros(int(cells[-1]), dtype=torch.float64, device="cuda"), {}
        for p, d in enumerate(dims):
            n = [int(v) for v in d]
            h = 1.0 / max(n)
            op = _Operator([_axis(m, "u", m * h) for m in n])
            for m in n:                                    # modes by size, for unit widths
                if m not in axes:
                    one = _axis(m, "u", float(m))
                    axes[m] = _modes(*(torch.as_tensor(one[k][s], device="cuda") for k, s in ((0, slice(1, -1)), (1, slice(1, None)))))
            op.set_modes([axes[m] for m in n], 1.0 / h ** 2)
            v = out[int(cells[p]):int(cells[p + 1])].view(n[2] + 2, n[1] + 2, n[0] + 2)
            b = 2.0 * torch.rand((n[2], n[1], n[0]), dtype=torch.float64, device="cuda", generator=_generator(seed * 131 + p)) - 1.0
            op.solve(v, b)
        return out
    mesh = _mesh(c)
    op = _Operator(mesh)
    if c["kind"] == "solve":
        sol = op.solve(_guess(c, mesh, seed), _sources(c, mesh, seed)[1:-1, 1:-1, 1:-1])
        return {"sol": sol.cpu() if c["host"] else sol, "rsd": None}      # the residual is what is left over
    if c["kind"] == "autograd":
        b, w, g = _sources(c, mesh, seed), _random(c, seed + 1, ghosts=True), _faces(seed)
        u = _field(c)
        _set_faces(u, g)
        op.solve(u, b[1:-1, 1:-1, 1:-1])
        # A = V^-1 S with S symmetric and V the cell volumes: A^-T w = V A^-1 (w / V)
        vol = op.dm[2].view(-1, 1, 1) * op.dm[1].view(1, -1, 1) * op.dm[0].view(1, 1, -1)
        db = op.solve(_field(c), w[1:-1, 1:-1, 1:-1] / vol)
        db[1:-1, 1:-1, 1:-1] *= vol
        lam = db[1:-1, 1:-1, 1:-1]
        dg = []
        for a in range(3):
            dim = 2 - a
            dg.append(-(op.lo[a].flatten()[0] * lam.select(dim, 0)).sum())
            dg.append(-(op.hi[a].flatten()[-1] * lam.select(dim, lam.shape[dim] - 1)).sum())
        own = [w[1:-1, 1:-1, 0], w[1:-1, 1:-1, -1], w[1:-1, 0, :], w[1:-1, -1, :], w[0], w[-1]]
        return {"u": u, "db": db, "dg": torch.stack([p + v.sum() for p, v in zip(dg, own)]).cpu()}
    b, x = _random(c, seed), _random(c, seed + 1, ghosts=True)
    if c["kind"] == "transfer":
        coarse = {"nx": c["nx"] // 2, "ny": c["ny"] // 2, "nz": c["nz"] // 2}
        return _exact_transfer(c, mesh, {"b": b, "x0": x, "bc": _field(coarse),
                                         "xc": _random(coarse, seed + 2, ghosts=True)})
    bi, xi = b[1:-1, 1:-1, 1:-1], x[1:-1, 1:-1, 1:-1]
    if c["kind"] == "smooth":
        k = torch.arange(1, max(xi.shape) + 1, device="cuda")
        parity = (k[:xi.shape[0]].view(-1, 1, 1) + k[:xi.shape[1]].view(1, -1, 1) + k[:xi.shape[2]].view(1, 1, -1)) % 2
        d = op.diagonal()
        for _ in range(c["iters"]):
            for colour in (1, 0):                           # odd index sums first
                new = c["omega"] * (bi - op.neighbours(x)) / d + (1.0 - c["omega"]) * xi
                xi.copy_(torch.where(parity == colour, new, xi))
        return x
    p = _field(c)                                           # conjugate gradients: p's ghosts are zero
    pi = p[1:-1, 1:-1, 1:-1]
    r = bi - op.apply(x)
    pi.copy_(r)
    rr = (r * r).sum()
    for _ in range(c["iters"]):
        q = op.apply(p)
        alpha = rr / (pi * q).sum()
        xi += alpha * pi
        r -= alpha * q
        new = (r * r).sum()
        pi.copy_(r + (new / rr) * pi)
        rr = new
    return x

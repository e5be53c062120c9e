"""Timed cases of the L-sweeps library: the calls its users make, through the
public Python API (`lsweeps.solver.Solver`), over the range of sizes, media,
precisions and batch sizes that the library's own workloads have.

A case is a dict of plain values.  `kind` names the call:

  matvec    Solver.apply_A: the FP64 5-point operator (residual checks)
  local     Solver.local_solve: one cell solve, the LocalLinearSolver::solve
            of the plugin API
  apply     Solver.apply_precond in complex128: the plain method, whose
            preconditioner callers take out of the solver and iterate themselves
  solve     Solver.gmres (or Solver.solve_host with host buffers) on a resident
            factorised operator: what a user of the library waits for
  operator  a new medium: Solver, factorize and gmres, as a serving loop does
            for a request whose operator is not resident

The reduced precisions (c64, bf16x2) exist for one use, the preconditioner
inside FP64 flexible GMRES, and are measured there.  Their wavefields are kept
in complex64, which holds what a 1e-6 residual determines.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "l-sweeps-2d_gb300"))

from lsweeps.problems import ProblemSpec, omega_for_ppw  # noqa: E402
from lsweeps.solver import Solver  # noqa: E402

DEV = "cuda:0"
F8, C16 = torch.float64, torch.complex128


def _case(name, kind, N, m, p, prec, medium="lens", ppw=8.0, nrhs=1, host=False):
    return dict(name=name, kind=kind, N=N, m=m, p=p, prec=prec, medium=medium, ppw=ppw, nrhs=nrhs, host=host)


def listed():
    return [
        # the FP64 operator on the 2048^2 grid, four wavefields at once
        _case("matvec_2048_x4", "matvec", 16, 128, 20, "c64", "layered", nrhs=4),
        # one cell of the 4 x 4 x 64^2 problem: the smallest call, all latency
        _case("local_64_fp64", "local", 4, 64, 10, "c128"),
        # the plain FP64 method on the 4 x 4 x 64^2 problem: one preconditioner apply, one solve
        _case("apply_256_fp64", "apply", 4, 64, 10, "c128", ppw=10.0),
        _case("solve_256_fp64", "solve", 4, 64, 10, "c128", ppw=10.0),
        # the serving stream's smallest grid through host buffers
        _case("solve_host_256", "solve", 2, 128, 16, "c64", host=True),
        # a 512^2 request with four sources, solved in lockstep
        _case("solve_512_x4", "solve", 4, 128, 16, "c64", "layered", ppw=9.0, nrhs=4),
        # the 1024^2 lens problem
        _case("solve_1024", "solve", 8, 128, 16, "c64"),
        # odd cells, a larger batch of sources, a layered medium (many iterations)
        _case("solve_500_x8_odd", "solve", 5, 99, 13, "c64", "layered", nrhs=8),
        # sixteen sources on bf16-split factors, odd cells
        _case("solve_700_x16_split", "solve", 6, 117, 18, "bf16x2", nrhs=16),
        # the 2048^2 high-contrast medium on bf16-split factors: HBM-bound
        _case("solve_2048_split", "solve", 16, 128, 20, "bf16x2", "random"),
        # new media: set up, factorise, solve
        _case("operator_512_x2", "operator", 4, 128, 16, "c64", nrhs=2),
        _case("operator_1024_split", "operator", 8, 128, 16, "bf16x2"),
    ]


def draw(rng):
    kind = rng.choice(["matvec", "local", "apply", "solve", "solve", "solve", "operator"])
    prec = {"apply": "c128", "matvec": "c64", "operator": rng.choice(["c64", "bf16x2"]),
            "local": "c128"}.get(kind) or rng.choice(["c64", "c64", "bf16x2", "bf16x2", "c128"])
    m = int(round(math.exp(rng.uniform(math.log(24), math.log(140)))))
    p = rng.randint(5, min(20, max(6, m // 4), (192 - m - 5) // 2))
    nrhs = rng.choice([1, 1, 1, 2, 3, 4, 7, 16])
    # cells per side such that the case stays below the largest listed one
    n_max = {"matvec": 16, "local": 4, "apply": 6, "operator": 8}.get(kind, 12 if prec != "c128" else 4)
    if kind != "matvec":
        n_max = min(n_max, max(2, int(n_max / math.sqrt(nrhs))))
    N = rng.randint(2, n_max)
    medium = rng.choice(["lens", "layered", "random"])
    return dict(kind=kind, N=N, m=m, p=p, prec=prec, medium=medium, ppw=round(rng.uniform(7.0, 10.0), 2),
                nrhs=nrhs, host=kind == "solve" and N <= 4 and rng.random() < 0.3)


# ---- inputs -----------------------------------------------------------------

def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _smooth(a, sigma):
    r = int(4 * sigma)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=DEV, dtype=F8) / sigma) ** 2)
    k = (k / k.sum()).reshape(1, 1, -1)
    for _ in range(2):
        rows = torch.nn.functional.pad(a[:, None, :], (r, r), mode="replicate")
        a = torch.nn.functional.conv1d(rows, k)[:, 0, :].T.contiguous()
    return a


def _velocity(case, seed):
    """A seeded medium on the global grid: a Gaussian lens, perturbed layers, or smoothed random regions."""
    N, m, p = case["N"], case["m"], case["p"]
    n_g = N * m + N - 1
    n = n_g + 2 * p - 1
    g = _gen(seed, 1)
    s = (torch.arange(n, device=DEV, dtype=F8) + 1 - p) / n_g
    u = torch.rand(8, generator=g, device=DEV, dtype=F8).tolist()
    if case["medium"] == "lens":
        x0, y0, amp, w = 0.35 + 0.3 * u[0], 0.35 + 0.3 * u[1], 0.3 + 0.1 * u[2], 0.08 + 0.04 * u[3]
        return 1 - amp * torch.exp(-((s[:, None] - x0) ** 2 + (s[None, :] - y0) ** 2) / (2 * w * w))
    if case["medium"] == "layered":
        vel = 1.5 + 3.0 * torch.rand(12, generator=g, device=DEV, dtype=F8)
        layer = ((1 - s).clamp(0, 1 - 1e-12) * 12).long().clamp(max=11)
        noise = _smooth(torch.randn(n, n, generator=g, device=DEV, dtype=F8), 4.0)
        return vel[layer][None, :] * (1 + 0.05 * noise / noise.std())
    pts = torch.rand(48, 2, generator=g, device=DEV, dtype=F8)
    val = torch.rand(48, generator=g, device=DEV, dtype=F8)
    best = torch.full((n, n), 1e30, device=DEV, dtype=F8)
    c = torch.zeros(n, n, device=DEV, dtype=F8)
    for q in range(48):
        d = (s[:, None] - pts[q, 0]) ** 2 + (s[None, :] - pts[q, 1]) ** 2
        c = torch.where(d < best, val[q], c)
        best = torch.minimum(best, d)
    c = _smooth(c, 8.0)
    return 1.5 + 3.5 * (c - c.min()) / (c.max() - c.min())


def _problem(case, seed):
    N, m, p = case["N"], case["m"], case["p"]
    h = 1.0 / (N * m + N - 1)
    c = _velocity(case, seed)
    spec = ProblemSpec(N=N, m=m, p=p, h=h, omega=omega_for_ppw(float(c.min()), case["ppw"], h))
    return spec, (1.0 / (c * c)).cpu().numpy()


def _sources(case, seed):
    """One point source per right-hand side, inside the domain."""
    u = torch.rand(case["nrhs"], 2, generator=_gen(seed, 2), device=DEV, dtype=F8)
    return (0.1 + 0.8 * u).tolist()


def _cell(case):
    """A cell in the middle of the checkerboard."""
    return (case["N"] // 2) * (case["N"] + 1)


def _vectors(case, seed, n):
    return torch.randn(case["nrhs"] * n, generator=_gen(seed, 3), device=DEV, dtype=C16)


def prepare(case, seed):
    spec, slow2 = _problem(case, seed)
    st = dict(case=case, spec=spec, slow2=slow2)
    S = Solver(spec, slow2, precision=case["prec"])
    if case["kind"] in ("solve", "operator"):
        st["b"] = torch.cat([S.assemble_rhs([q]) for q in _sources(case, seed)])
        if case["host"]:
            st["b"] = st["b"].cpu().numpy()
            st["x"] = np.empty_like(st["b"])
    if case["kind"] == "operator":
        S.close()
        return st
    if case["kind"] != "matvec":
        S.factorize()
    if case["kind"] == "local":
        st["cell"] = _cell(case)
        info = S.cell_info(st["cell"])
        st["b"] = _vectors(case, seed, info["nx"] * info["ny"])
    elif case["kind"] in ("matvec", "apply"):
        st["b"] = _vectors(case, seed, S.n2)
    st["S"] = S
    return st


def _wavefield(case, x):
    if case["prec"] == "c128":
        return x
    return x.astype(np.complex64) if case["host"] else x.to(torch.complex64)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "matvec":
        return st["S"].apply_A(st["b"])
    if kind == "local":
        return st["S"].local_solve(st["cell"], st["b"])
    if kind == "apply":
        return st["S"].apply_precond(st["b"])
    opts = dict(mode="flexible", tol=1e-6, max_iter=60, restart=30)
    if kind == "operator":
        S = Solver(st["spec"], st["slow2"], precision=case["prec"])
        S.factorize()
        x, _ = S.gmres(st["b"], **opts)
        S.close()
    elif case["host"]:
        x, _ = st["S"].solve_host(st["b"], x_host=st["x"], **opts)
    else:
        x, _ = st["S"].gmres(st["b"], **opts)
    return _wavefield(case, x)


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """A cell solve reads the cell's factor twice (forward, backward): per x-line the inverse of a complex symmetric
    block (up to a diagonal scaling), half of ny^2 entries.  An apply visits N^2 + 4 N (N - 1) + 4 (N - 1)^2 cells
    (stage 1, four sweeps, four L-sweeps) with four shifted decompositions per right-hand side.  Solves count a nominal
    number of iterations of the medium."""
    N, m, p, k = case["N"], case["m"], case["p"], case["nrhs"]
    n = N * m + N - 1 + 2 * p - 1
    s = 16 if case["prec"] == "c128" else 8
    nd = m + (6 if N > 2 else 3) + 2 * p - 1
    cell_bytes, cell_flops = nd * nd * (nd + 1) / 2 * s, 16.0 * nd ** 3
    if case["kind"] == "matvec":
        return {"bytes": n * n * (32 * k + 8), "flops": 40.0 * k * n * n}
    if case["kind"] == "local":
        return {"bytes": 2 * cell_bytes + 32 * k * nd * nd, "flops": k * cell_flops}
    visits = N * N + 4 * N * (N - 1) + 4 * (N - 1) ** 2
    apply = {"bytes": visits * 2 * cell_bytes + 32 * k * n * n, "flops": visits * 4 * k * cell_flops}
    if case["kind"] == "apply":
        return apply
    its = {"lens": 5, "layered": 20, "random": 12}[case["medium"]]
    w = {q: its * v for q, v in apply.items()}
    w["bytes"] += its * k * n * n * (40 + 24 * its)   # the operator, the orthogonalisation
    if case["kind"] == "operator":
        w["bytes"] += N * N * cell_bytes + 8 * n * n
        w["flops"] += 8.0 * N * N * nd ** 4
    return w


# ---- the same in plain 64-bit torch ------------------------------------------

def _profile(nel, p, h, C):
    """Couplings to the previous and next node and the diagonal share, along one direction, of the 5-point operator
    with a cubic PML of p cells outside nel interior elements."""
    q = torch.arange(1, nel + 2 * p, device=DEV, dtype=F8)
    d = (p - q).clamp(min=0) + (q - p - nel).clamp(min=0)
    sign = torch.sign(q - p - 0.5)
    sg, dsg = C * (d / p) ** 3, sign * 3 * C * d * d / (p ** 3 * h)
    a = 1 / (1 + 1j * sg)
    lam, beta = a * a, -1j * dsg * a ** 3
    return -lam / h ** 2 + beta / (2 * h), -lam / h ** 2 - beta / (2 * h), 2 * lam / h ** 2


class _Box:
    """Direct solver on one box: block elimination over its x-lines."""

    def __init__(self, px, py, diag):
        self.lo, self.hi, dx = px
        T = torch.diag(py[2]) + torch.diag(py[0][1:], -1) + torch.diag(py[1][:-1], 1)
        self.inv = []
        for k in range(len(dx)):
            A = T + torch.diag(dx[k] + diag[k])
            if k:
                A = A - self.lo[k] * self.hi[k - 1] * self.inv[-1]
            self.inv.append(torch.linalg.inv(A))

    def solve(self, b):
        """b: [lines][points][vectors]"""
        y = []
        for k, Si in enumerate(self.inv):
            y.append(Si @ (b[k] - self.lo[k] * y[-1] if k else b[k]))
        for k in range(len(y) - 2, -1, -1):
            y[k] = y[k] - self.hi[k] * (self.inv[k] @ y[k + 1])
        return torch.stack(y)


class _Grid:
    """The global grid, its checkerboard cells and the L-sweep preconditioner."""

    def __init__(self, case, seed):
        self.spec, slow2 = _problem(case, seed)
        s = self.spec
        self.N, self.m, self.p = s.N, s.m, s.p
        self.diag = -(s.omega ** 2) * torch.from_numpy(slow2).to(DEV)
        self.n_g, self.n = s.n_g, s.n_dof
        self.prof = self.profile(self.n_g)
        self.boxes = {}

    def profile(self, nel):
        return _profile(nel, self.p, self.spec.h, math.log(self.spec.omega))

    def side(self, J):
        """First node, interior elements, trace lines and owned range per shift of cell J along one direction."""
        ka, kb = (self.m + 1) * J, (self.m + 1) * J + self.m
        first, last = J == 0, J == self.N - 1
        lo = 0 if first else ka - 2
        nel = (self.n_g if last else kb + 4) - lo
        nd = nel + 2 * self.p - 1
        at = lambda k: k - lo + self.p - 1  # noqa: E731
        lines = [[None if first else at(ka - 1 + o), None if first else at(ka + o),
                  None if last else at(kb + o), None if last else at(kb + 1 + o)] for o in (0, 2)]
        own = [(0 if first else at(ka + o), nd - 1 if last else at(kb + o)) for o in (0, 2)]
        return lo, nel, nd, lines, own

    def box(self, I, J):
        if (I, J) not in self.boxes:
            (lx, nx, dx, _, _), (ly, ny, dy, _, _) = self.side(J), self.side(I)
            self.boxes[I, J] = _Box(self.profile(nx), self.profile(ny), self.diag[lx:lx + dx, ly:ly + dy])
        return self.boxes[I, J]

    def matvec(self, x):
        lo, hi, dg = self.prof
        y = (dg[:, None] + dg[None, :] + self.diag) * x
        y[:, 1:] += lo[1:, None] * x[:, :-1]
        y[:, :-1] += hi[:-1, None] * x[:, 1:]
        y[:, :, 1:] += lo[None, 1:] * x[:, :, :-1]
        y[:, :, :-1] += hi[None, :-1] * x[:, :, 1:]
        return y

    def interface(self, lo, nd):
        """Which nodes of a cell's side lie on an interface line pair."""
        g = torch.arange(nd, device=DEV) + lo - self.p + 1
        r = g % (self.m + 1)
        return ((r == self.m) | (r == 0)) & (g >= self.m) & (g <= (self.m + 1) * (self.N - 1))

    def precond(self, x):
        """x: [vectors][n][n]"""
        out = torch.zeros_like(x)
        for sx in (0, 1):
            for sy in (0, 1):
                self._sweeps(x, out, sx, sy)
        return out

    def _sweeps(self, x, out, sx, sy):
        N, k = self.N, x.shape[0]
        sides = [self.side(J) for J in range(N)]
        tr = {}

        def read(name, I, J, line, length):
            return tr.get((name, I, J, line), torch.zeros(length, k, device=DEV, dtype=C16))

        def cell(I, J):
            X, Y = sides[J], sides[I]
            return X, Y, X[3][sx], Y[3][sy], self.profile(X[1]), self.profile(Y[1])

        def add(I, J, u, lr=None, lr_lines=(), ud=None, ud_lines=(), value=lambda u: u):
            X, Y, lx, ly, _, _ = cell(I, J)
            (x0, x1), (y0, y1) = X[4][sx], Y[4][sy]
            out[:, X[0] + x0:X[0] + x1 + 1, Y[0] + y0:Y[0] + y1 + 1] += u[x0:x1 + 1, y0:y1 + 1].permute(2, 0, 1)
            v = value(u)
            for name, lines, at, pick in ((lr, lr_lines, lx, lambda q: v[q]), (ud, ud_lines, ly, lambda q: v[:, q])):
                for q in lines:
                    if name and at[q] is not None:
                        tr[name, I, J, q] = tr.get((name, I, J, q), 0) + pick(at[q])

        def blank(X, Y):
            return torch.zeros(X[2], Y[2], k, device=DEV, dtype=C16)

        # stage 1: every cell on its window of the input
        for I in range(N):
            for J in range(N):
                X, Y, _, _, _, _ = cell(I, J)
                (x0, x1), (y0, y1) = X[4][sx], Y[4][sy]
                keep = torch.zeros(X[2], Y[2], device=DEV, dtype=torch.bool)
                keep[x0:x1 + 1, y0:y1 + 1] = True
                keep &= (self.interface(X[0], X[2]) == bool(sx))[:, None] & (self.interface(Y[0], Y[2]) == bool(sy))[None]
                b = x[:, X[0]:X[0] + X[2], Y[0]:Y[0] + Y[2]].permute(1, 2, 0) * keep[:, :, None]
                add(I, J, self.box(I, J).solve(b), "LR", range(4), "UD", range(4))

        def ends(fwd):
            """Outer and inner source line, the neighbour's lines read, the lines passed on."""
            return (0, 1, (2, 3), (2, 3)) if fwd else (3, 2, (1, 0), (0, 1))

        def couple(prof, fwd, o, i):
            return (prof[1][o], prof[0][i]) if fwd else (prof[0][o], prof[1][i])

        # stage 2: the four directions
        for t in range(1, N):
            for q in range(N):
                for fwd, side in ((True, "UDR"), (False, "UDL")):
                    I, J, nb = q, (t if fwd else N - 1 - t), (t - 1 if fwd else N - t)
                    X, Y, lx, _, px, _ = cell(I, J)
                    o, i, src, on = ends(fwd)
                    coi, cio = couple(px, fwd, lx[o], lx[i])
                    b = blank(X, Y)
                    b[lx[o]] = coi * read("LR", I, nb, src[1], Y[2])
                    b[lx[i]] = -cio * read("LR", I, nb, src[0], Y[2])
                    add(I, J, self.box(I, J).solve(b), "LR", on, side, range(4))
                for fwd, side in ((True, "LRU"), (False, "LRD")):
                    J, I, nb = q, (t if fwd else N - 1 - t), (t - 1 if fwd else N - t)
                    X, Y, _, ly, _, py = cell(I, J)
                    o, i, src, on = ends(fwd)
                    coi, cio = couple(py, fwd, ly[o], ly[i])
                    b = blank(X, Y)
                    b[:, ly[o]] = coi * read("UD", nb, J, src[1], X[2])
                    b[:, ly[i]] = -cio * read("UD", nb, J, src[0], X[2])
                    add(I, J, self.box(I, J).solve(b), side, range(4), "UD", on)

        # stage 3: the four L-sweeps, diagonal by diagonal
        for dd in range(2 * N - 3):
            for lr, ud, right, top in (("LRU", "UDR", 1, 1), ("LRD", "UDL", 0, 0), ("LRU", "UDL", 0, 1),
                                       ("LRD", "UDR", 1, 0)):
                for a in range(1, N):
                    c = dd + 2 - a
                    if not 1 <= c < N:
                        continue
                    I, J = (a if top else N - 1 - a), (c if right else N - 1 - c)
                    X, Y, lx, ly, px, py = cell(I, J)
                    (ox, ix, sxl, onx), (oy, iy, syl, ony) = ends(right), ends(top)
                    xo, xi, yo, yi = lx[ox], lx[ix], ly[oy], ly[iy]
                    cxo, cxi = couple(px, right, xo, xi)
                    cyo, cyi = couple(py, top, yo, yi)
                    nbx, nby = (J - 1 if right else J + 1), (I - 1 if top else I + 1)
                    lr0, lr1 = (read(lr, I, nbx, sxl[w], Y[2]) for w in (0, 1))
                    ud0, ud1 = (read(ud, nby, J, syl[w], X[2]) for w in (0, 1))
                    inx = slice(xi + 1, None) if right else slice(0, xi)
                    iny = slice(yi + 1, None) if top else slice(0, yi)
                    b = blank(X, Y)
                    b[xo, iny], b[xo, yi] = cxo * lr1[iny], cxo * ud1[xi]
                    b[xi, iny], b[xi, yo] = -cxi * lr0[iny], cyo * ud1[xi]
                    b[xi, yi] = -cxi * lr0[yi] - cyi * ud0[xi]
                    b[inx, yo], b[inx, yi] = cyo * ud1[inx], -cyi * ud0[inx]

                    def incoming(u):
                        v = u.clone()
                        v[xo], v[:, yo] = lr0, ud0
                        return v

                    add(I, J, self.box(I, J).solve(b), lr, onx, ud, ony, incoming)


def exact(case, seed):
    k, n_cells = case["nrhs"], case["N"] ** 2
    G = _Grid(case, seed) if case["kind"] != "operator" else None
    if case["kind"] == "matvec":
        return G.matvec(_vectors(case, seed, G.n ** 2).reshape(k, G.n, G.n)).reshape(-1)
    if case["kind"] == "local":
        c = _cell(case)
        box = G.box(c // case["N"], c % case["N"])
        nx, ny = len(box.inv), len(box.inv[0])
        x = box.solve(_vectors(case, seed, nx * ny).reshape(k, nx, ny).permute(1, 2, 0))
        return x.permute(2, 0, 1).reshape(-1)
    if case["kind"] == "apply":
        if n_cells * (case["m"] + 2 * case["p"]) > 3000:
            return None
        return G.precond(_vectors(case, seed, G.n ** 2).reshape(k, G.n, G.n)).reshape(-1)
    G = G or _Grid(case, seed)
    if G.n > 640:
        return None
    at = (torch.arange(G.n, device=DEV, dtype=F8) + 1 - G.p) * G.spec.h
    b = []
    for x0, y0 in _sources(case, seed):
        r2 = (at[:, None] - x0) ** 2 + (at[None, :] - y0) ** 2
        b.append(torch.exp(-r2 / G.spec.h ** 2) / (math.pi * G.spec.h ** 2))
    whole = _Box(G.prof, G.prof, G.diag)
    x = whole.solve(torch.stack(b, 2).to(C16)).permute(2, 0, 1).reshape(-1)
    return x.cpu().numpy() if case["host"] else x

"""The symmetric-tile sweep kernels (complex64 and bf16 split) where they can go
wrong: points per line at and around multiples of the 16-point tiles and of the
four tile classes, the smallest and the largest cells, and right-hand-side
counts at the edges of the slot paddings.  One cell (N = 1), so the cell matrix
is the global operator; the reference is the complex128 solve of the same cell
(other factor layout, other kernel; pinned to SuperLU in test_gpu_parity.py),
at the parity tolerance of the reduced precisions (2e-4).  Rectangular cells
come with N = 3: edge and inner cells differ in lines and points."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 2e-4


def _vectors(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, device="cuda", dtype=torch.complex128)


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _pair(spec, med, prec):
    from lsweeps.solver import Solver
    out = []
    for p in ("c128", prec):
        S = Solver(spec, med, precision=p)
        S.factorize()
        out.append(S)
    return out


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
@pytest.mark.parametrize("side", [6, 15, 16, 17, 31, 33, 48, 49, 64, 65, 97, 128, 129, 160, 175, 177, 191, 192])
def test_cell_solve_at_tile_edges(side, prec):
    p = 1 if side < 12 else 4
    spec, med = small(N=1, m=side - 2 * p + 1, p=p, medium="lens")
    ref, S = _pair(spec, med, prec)
    assert S.cell_info(0)["ny"] == side
    for nrhs in (1, 2, 3, 5, 8, 9, 13, 16, 17):
        b = _vectors(nrhs * side * side, 100 * side + nrhs)
        x = S.local_solve(0, b)
        assert _rel(x, ref.local_solve(0, b)) <= TOL, nrhs
        assert torch.equal(S.local_solve(0, b), x)
    for s in (ref, S):
        s.close()


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
@pytest.mark.parametrize("shape", ["4x1", "4x2", "4x4", "8x1", "8x2", "16x1"])
@pytest.mark.parametrize("N,m,p", [(3, 11, 2), (2, 57, 9), (3, 33, 5)])
def test_preconditioner_in_every_launch_shape(N, m, p, shape, prec, monkeypatch):
    """Slots per item x CTAs per half chain imposed on every front, one launch per step and per sweep."""
    monkeypatch.setenv("LSW_FRONT_SHAPE", shape)
    spec, med = small(N=N, m=m, p=p, medium="layered", seed=3)
    ref, S = _pair(spec, med, prec)
    for nrhs in (1, 3):
        v = _vectors(nrhs * S.n2, N * m + nrhs)
        y = S.apply_precond(v)
        assert _rel(y, ref.apply_precond(v)) <= TOL
        assert torch.equal(S.apply_precond(v), y)
    for s in (ref, S):
        s.close()

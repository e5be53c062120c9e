"""The complex128 sweep kernel where its split over the lanes changes: points per
line around multiples of 32 and 128, from the smallest to the largest cells (one
to sixteen column slices), and right-hand-side counts at the edges of the slot
paddings and of an item.  One cell (N = 1), so the cell matrix is the global
operator; the check is the residual in FP64, at the 1e-10 to which the cell
solves are pinned against SuperLU in test_gpu_parity.py."""
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [6, 12, 31, 32, 33, 54, 64, 89, 96, 97, 127, 128, 129, 161, 191, 192])
def test_cell_solve_residual(side):
    from lsweeps.solver import Solver
    p = 1 if side < 12 else 4
    spec, med = small(N=1, m=side - 2 * p + 1, p=p, medium="lens")
    S = Solver(spec, med, precision="c128")
    S.factorize()
    assert S.cell_info(0)["ny"] == side
    for nrhs in (1, 2, 3, 8, 9):
        g = torch.Generator(device="cuda").manual_seed(100 * side + nrhs)
        b = torch.randn(nrhs * side * side, generator=g, device="cuda", dtype=torch.complex128)
        x = S.local_solve(0, b)
        r = S.apply_A(x) - b
        assert float(r.norm() / b.norm()) <= 1e-10
        assert torch.equal(S.local_solve(0, b), x)
    S.close()

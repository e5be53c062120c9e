"""Symmetric-tile sweeps of small cells, whose CTAs share an SM: a CTA has the warps
of its rows only and a ring that leaves room for others.  Batches large enough to
put several CTAs on every SM, for cells of one to seven tile rows, against the
complex128 preconditioner at the parity tolerance of the reduced precisions (2e-4)
and twice for equal bits; and a batch of sixteen costs less than six times one
vector on 16 x 16 cells of 21 points (with one CTA per SM it cost over ten times)."""
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
@pytest.mark.parametrize("shape", ["1x1", "4x1", "16x1", "2x2", "8x4"])
@pytest.mark.parametrize("N,m,p", [(6, 5, 1), (5, 11, 4), (4, 20, 6), (3, 40, 8), (3, 57, 9), (2, 84, 12)])
def test_many_vectors(N, m, p, shape, prec, monkeypatch):
    from lsweeps.solver import Solver
    spec, med = small(N=N, m=m, p=p, medium="lens")
    ref = Solver(spec, med, precision="c128")
    ref.set_tuning(False)
    monkeypatch.setenv("LSW_FRONT_SHAPE", shape)
    S = Solver(spec, med, precision=prec)
    for s in (ref, S):
        s.factorize()
    nrhs = 13
    g = torch.Generator(device="cuda").manual_seed(N * m)
    v = torch.randn(nrhs * S.n2, generator=g, device="cuda", dtype=torch.complex128)
    y, want = S.apply_precond(v), ref.apply_precond(v)
    assert float((y - want).norm() / want.norm()) <= 2e-4
    assert torch.equal(S.apply_precond(v), y)
    for s in (ref, S):
        s.close()


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
def test_small_cells_share_the_sms(prec, monkeypatch):
    from lsweeps.solver import Solver
    monkeypatch.setenv("LSW_FRONT_SHAPE", "4x1")
    monkeypatch.setenv("LSW_SWEEP_LANES", "0")
    spec, med = small(N=16, m=8, p=4, medium="lens")
    S = Solver(spec, med, precision=prec)
    S.factorize()

    def best(nrhs):
        x = torch.randn(nrhs * S.n2, device="cuda", dtype=torch.complex128)
        y, t = torch.empty_like(x), []
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            S.apply_precond(x, y)
            e[1].record()
            e[1].synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t[1:])

    assert best(16) < 6.0 * best(1)
    S.close()

"""Sweep fronts of one and two slots per item, imposed on every launch: per sweep
(one right-hand side) and per step (three), where a cell that several sweeps
reach in one front keeps a group of slots that no item may split.  Shapes only
change how right-hand sides share a launch, so the results agree with the
untuned schedule to the rounding of the sums that a shape reorders: 1e-12 in
complex128 and, several FP32 (split: 2^-16) roundings of a cell solve apart,
2e-4 in the reduced precisions."""
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("c128", 1e-12), ("c64", 2e-4), ("bf16x2", 2e-4)])
@pytest.mark.parametrize("shape", ["1x1", "1x2", "1x4", "2x1", "2x2", "2x4"])
@pytest.mark.parametrize("N,m,p", [(2, 21, 4), (3, 33, 5)])
def test_small_items_give_the_same_apply(N, m, p, shape, prec, tol, monkeypatch):
    from lsweeps.solver import Solver
    spec, med = small(N=N, m=m, p=p, medium="layered", seed=5)
    ref = Solver(spec, med, precision=prec)
    ref.set_tuning(False)
    ref.factorize()
    monkeypatch.setenv("LSW_FRONT_SHAPE", shape)
    S = Solver(spec, med, precision=prec)
    S.factorize()
    r, cl = (int(v) for v in shape.split("x"))
    for nrhs in (1, 3):
        g = torch.Generator(device="cuda").manual_seed(nrhs)
        v = torch.randn(nrhs * S.n2, generator=g, device="cuda", dtype=torch.complex128)
        y, want = S.apply_precond(v), ref.apply_precond(v)
        assert float((y - want).norm() / want.norm()) <= tol
        assert torch.equal(S.apply_precond(v), y)
        shapes, _ = S.front_shapes(nrhs)
        assert any(f["items"] > 0 and f["slots_cap"] == r and f["cluster"] == cl for f in shapes)
    for s in (ref, S):
        s.close()

"""The search for a per-sweep schedule (the first apply of one or two vectors on a
new problem shape) times a bounded number of schedules, whatever the clock says:
its kernel launches are counted.  One apply is launched untimed, then at most four
candidates and two mixes of them once each (applies of half a millisecond or more),
besides the apply that was asked for.  The tuned complex128 schedule agrees with the
cost model's to rounding (1e-12), and repeated applies are bit-identical."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

# (a process of its own: the process keeps what it has measured)
_CHILD = r"""
import json, sys
sys.path[:0] = [{root!r}, {pkg!r}]
import torch
from lsweeps.problems import small
from lsweeps.solver import Solver
spec, med = small(N={N}, m={m}, p={p}, medium="layered", seed=4)
v = torch.randn({nrhs} * spec.n_dof ** 2, device="cuda", dtype=torch.complex128)
out = dict()
y = dict()
for prec in ("c128", {prec!r}):
    for tune in (True, False):
        S = Solver(spec, med, precision=prec)
        S.set_tuning(tune)
        S.set_graphs(False)
        S.factorize()
        n0 = S.info()["kernel_launches"]
        y[prec, tune] = S.apply_precond(v)
        n1 = S.info()["kernel_launches"]
        again = S.apply_precond(v)
        n2 = S.info()["kernel_launches"]
        assert torch.equal(again, y[prec, tune])
        out[prec + ("_tuned" if tune else "")] = [n1 - n0, n2 - n1]
        S.close()
rel = lambda a, b: float((a - b).norm() / b.norm())
out["err"] = rel(y["c128", True], y["c128", False])
print(json.dumps(out))
"""


@pytest.mark.parametrize("N,m,p,nrhs,prec", [(4, 128, 16, 1, "c64"), (4, 128, 16, 2, "bf16x2"), (6, 99, 13, 1, "c64"),
                                             (1, 128, 16, 1, "bf16x2"), (2, 150, 18, 2, "c64")])
def test_search_is_bounded(N, m, p, nrhs, prec):
    code = _CHILD.format(root=str(ROOT), pkg=str(ROOT / "l-sweeps-2d_gb300"), N=N, m=m, p=p, nrhs=nrhs, prec=prec)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["err"] <= 1e-12, out
    twice = N == 1                          # (applies below half a millisecond are timed twice)
    for p_ in ("c128", prec):
        first, later = out[p_ + "_tuned"]
        assert later < first <= 2 + (2 + (13 if twice else 7)) * later, (p_, out)
        assert out[p_][0] == out[p_][1]


@pytest.mark.parametrize("N,nrhs,prec", [(16, 3, "c64"), (8, 4, "bf16x2"), (6, 5, "c128")])
def test_fronts_of_one_kind_are_measured_once(N, nrhs, prec):
    """One launch per step: of the N - 1 columns all but the last are alike (it has the
    cells of both edges; an odd N has a middle one, too), and are measured once: they
    hold the same time and shape."""
    from lsweeps.problems import small
    from lsweeps.solver import Solver
    spec, med = small(N=N, m=6, p=2, medium="layered", seed=4)
    S = Solver(spec, med, precision=prec)
    S.factorize()
    fronts = [(f["tuned_ms"], f["slots_cap"], f["cluster"], f["items"]) for f in S.front_shapes(nrhs)[0]]
    assert len(fronts) == 1 + (N - 1) + (2 * N - 3) and all(f[0] > 0 for f in fronts)
    assert len(set(fronts[1:N - 1])) == 1
    S.close()

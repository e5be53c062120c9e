"""The global operator for several vectors at once, where its kernel can go wrong:
vector counts at and around the groups of four, points per line that fill no
block, and the profile's edges (real coefficients inside, complex ones in the
PML).  The reference is the NumPy oracle of the same problem; the kernel does
about 20 multiply-adds in FP64 per point, so 1e-13 of the vector's norm is some
twenty times its rounding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402
from oracle.lsweeps_oracle import OracleProblem  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("N,m,p", [(1, 6, 2), (2, 29, 3), (3, 43, 5)])
def test_operator_on_several_vectors(N, m, p, nrhs):
    from lsweeps.solver import Solver
    spec, med = small(N=N, m=m, p=p, medium="lens")
    S = Solver(spec, med, precision="c64")
    P = OracleProblem(spec.N, spec.m, spec.p, spec.h, spec.omega, med)
    rng = np.random.default_rng(17 * nrhs + m)
    v = rng.standard_normal((nrhs, S.n2)) + 1j * rng.standard_normal((nrhs, S.n2))
    y = S.apply_A(torch.from_numpy(v.reshape(-1)).cuda()).cpu().numpy().reshape(nrhs, -1)
    for r in range(nrhs):
        want = P.apply_A_global(v[r])
        assert np.linalg.norm(y[r] - want) <= 1e-13 * np.linalg.norm(want)
    S.close()

"""The serving loop's estimate of an operator's device memory, against what the
library holds after a factorisation and a solve of a full batch: never below it (the
estimate is what a budget admits operators by), and not more than twice it, for
small and large cells, each precision, one vector and a batch."""
import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402
from lsweeps.serving import estimate_bytes  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["c128", "c64", "bf16x2"])
@pytest.mark.parametrize("N,m,p,batch,restart", [(16, 8, 4, 1, 5), (12, 16, 6, 1, 2), (6, 16, 6, 8, 30), (4, 64, 10, 1, 2),
                                                 (4, 64, 10, 4, 30), (2, 128, 16, 1, 30), (3, 128, 16, 3, 10)])
def test_estimate_covers_the_operator(N, m, p, batch, restart, prec):
    from lsweeps.solver import Solver
    spec, med = small(N=N, m=m, p=p, medium="lens")
    S = Solver(spec, med, precision=prec)
    S.factorize()
    b = torch.cat([S.assemble_rhs([(0.5 * spec.L, 0.4 * spec.L + 0.01 * r)]) for r in range(batch)])
    S.gmres(b, mode="flexible", tol=1e-30, max_iter=restart, restart=restart)
    held = S.info()["device_bytes"]
    est = estimate_bytes(spec, prec, batch, restart)
    print(f"N{N} m{m} {prec} batch {batch} restart {restart}: held {held / 1e6:.1f} MB estimate {est / 1e6:.1f} x{est / held:.2f}")
    assert held <= est <= 2 * held, (held, est)
    S.close()

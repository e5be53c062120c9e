"""Cell solves of several right-hand sides in the reduced precisions: the items
they are cut into follow a cost model, so that a batch does not wait on one
cluster while the other SMs idle.  Checked: solutions against the complex128
solve of the same cell at the parity tolerance of the reduced precisions (2e-4)
for counts at and around the item sizes; the allocation-free call gives the same
bits and takes and refuses the same counts as by its 8 MiB of forward storage,
(nx + 1) ny values of 8 bytes per right-hand side in groups of 16; and sixteen
right-hand sides, which fit on the device side by side, cost less than twice
four (as one item of sixteen slots they took four to five times as long)."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from lsweeps import capi  # noqa: E402
from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 2e-4


def _vectors(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, device="cuda", dtype=torch.complex128)


def _noalloc(S, cell, b, nrhs):
    from lsweeps.solver import _stream_ptr
    x = torch.empty_like(b)
    st = capi.lib().lsw_local_solve_noalloc(S.ctx, cell, C.c_void_p(b.data_ptr()), C.c_void_p(x.data_ptr()), nrhs,
                                            _stream_ptr(None))
    return st, x


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
@pytest.mark.parametrize("m,p", [(8, 2), (57, 9), (128, 16)])
def test_batches_of_one_cell(m, p, prec):
    from lsweeps.solver import Solver
    spec, med = small(N=2, m=m, p=p, medium="lens")
    ref, S = Solver(spec, med, precision="c128"), Solver(spec, med, precision=prec)
    for s in (ref, S):
        s.factorize()
    ci = S.cell_info(1)
    n = ci["nx"] * ci["ny"]
    per = (ci["nx"] + 1) * ci["ny"] * 8 * 16           # forward storage of sixteen right-hand sides
    limit = 16 * ((8 << 20) // per)                    # (the descriptors take less than what is left over)
    for nrhs in sorted({1, 4, 5, 16, 17, 33, min(limit, 200)}):
        b = _vectors(nrhs * n, nrhs)
        x = S.local_solve(1, b)
        want = ref.local_solve(1, b)
        assert float((x - want).norm() / want.norm()) <= TOL, nrhs
        if nrhs <= limit:
            st, y = _noalloc(S, 1, b, nrhs)
            assert st == 0 and torch.equal(x, y), nrhs
    if limit < 200:
        assert _noalloc(S, 1, _vectors((limit + 1) * n, 1), limit + 1)[0] == 1
    for s in (ref, S):
        s.close()


@pytest.mark.parametrize("prec", ["c64", "bf16x2"])
@pytest.mark.parametrize("m,p", [(64, 10), (128, 16)])
def test_sixteen_right_hand_sides_side_by_side(m, p, prec):
    from lsweeps.solver import Solver
    spec, med = small(N=2, m=m, p=p, medium="lens")
    S = Solver(spec, med, precision=prec)
    S.factorize()
    ci = S.cell_info(0)
    n = ci["nx"] * ci["ny"]

    def best(nrhs):
        b, t = _vectors(nrhs * n, 3), []
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(5):
                S.local_solve(0, b)
            e[1].record()
            e[1].synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t)

    assert best(16) < 2.0 * best(4)
    S.close()

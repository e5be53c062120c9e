"""The global operator is one launch whatever the number of vectors (the library
counts one), so that a small grid does not wait for a second one: the calls are
captured into a CUDA graph and its nodes counted.  Vector counts beyond
those of test_apply_operator_gpu.py, where the last group is short by up to three,
on grids around the widths of a block: against the vectors applied one at a time,
whose sums are the same operations in the same order (equal bits)."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from lsweeps.problems import small  # noqa: E402

pytestmark = pytest.mark.gpu


def _solver(side):
    from lsweeps.solver import Solver
    spec, med = small(N=1, m=side - 3, p=2, medium="lens")
    assert spec.n_dof == side
    return Solver(spec, med, precision="c64")


@pytest.mark.parametrize("nrhs", [1, 4, 5, 6, 7, 9, 13])
def test_one_launch(nrhs):
    S = _solver(40)
    x = torch.randn(nrhs * S.n2, device="cuda", dtype=torch.complex128)
    y = torch.empty_like(x)
    S.apply_A(x, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        S.apply_A(x, y)
    n = C.c_size_t(0)
    cudart = C.CDLL("libcudart.so.13")     # (loaded by torch)
    assert cudart.cudaGraphGetNodes(C.c_void_p(g.raw_cuda_graph()), None, C.byref(n)) == 0
    assert n.value == 1
    S.close()


@pytest.mark.parametrize("side", [8, 63, 65, 96, 97, 129, 140, 161, 190])
def test_short_last_groups(side):
    S = _solver(side)
    g = torch.Generator(device="cuda").manual_seed(side)
    for nrhs in (5, 6, 9, 10, 13):
        x = torch.randn(nrhs * S.n2, generator=g, device="cuda", dtype=torch.complex128)
        y = S.apply_A(x)
        for r in range(nrhs):
            assert torch.equal(y[r * S.n2:(r + 1) * S.n2], S.apply_A(x[r * S.n2:(r + 1) * S.n2].contiguous())), (nrhs, r)
    S.close()

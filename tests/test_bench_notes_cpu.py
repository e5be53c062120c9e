"""bench.py says truly how L2 is kept out of its timing: a workload whose cell factors,
as the library stores them, are not larger than L2 is flushed before each timed solve,
and only the others claim inputs larger than L2; the figures it names are theirs."""
import ctypes as C
import re
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))
import bench  # noqa: E402
from lsweeps import capi  # noqa: E402

L2 = 129e6
# (cells per side, elements per cell, PML) of the workloads
SIZES = {"C1": (4, 64, 10), "C2": (8, 128, 16), "C3": (16, 128, 20), "C4": (32, 128, 20)}


def factor_bytes(N, m, p):
    """Lower halves in 16 x 16 tiles of 8-byte values, nx lines per cell."""
    L, total = capi.lib(), 0
    g = capi.Geom(N, m, p, 2, 1.0 / (N * m + N - 1))
    for cell in range(N * N):
        o = capi.CellInfo()
        assert L.lsw_geometry_cell(C.byref(g), cell, C.byref(o)) == 0
        rows = (o.ny + 15) // 16
        total += o.nx * rows * (rows + 1) // 2 * 256 * 8
    return total


@pytest.mark.parametrize("name", sorted(SIZES))
def test_l2_note(name):
    held = factor_bytes(*SIZES[name])
    note = bench.L2_NOTE[name]
    assert (name in bench.L2_FLUSH) == (held <= L2)
    assert note.startswith("inputs larger than L2") == (held > L2)
    named = float(re.search(r"([0-9.]+) GB", note).group(1)) * 1e9
    assert abs(named - held) <= 0.05 * held, (held, named)

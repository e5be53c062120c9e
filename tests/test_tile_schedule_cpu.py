"""The sweep schedule for factors in symmetric tiles, on the CPU: the race checks of
test_schedule_cpu.py with items of one and two slots (several right-hand sides too),
and the scratch of the tile kernels, twice the rows on more than one CTA per half
(tests/host/tile_schedule_probe.cpp, compiled with csrc/geometry.cpp)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "l-sweeps-2d_gb300" / "csrc"


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    cuda_inc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if not (cuda_inc / "cuda_runtime.h").exists():
        pytest.skip("CUDA headers not found")
    out = tmp_path_factory.mktemp("tiles") / "tile_schedule_probe"
    cmd = [cxx, "-std=c++17", "-O2", str(ROOT / "tests" / "host" / "tile_schedule_probe.cpp"),
           str(CSRC / "geometry.cpp"), "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(cuda_inc), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("cl", [1, 2, 4])
@pytest.mark.parametrize("slots", [1, 2, 4, 16])
@pytest.mark.parametrize("N,m,p,nrhs", [(2, 10, 4, 1), (3, 12, 5, 3), (5, 7, 2, 2), (4, 16, 6, 8), (8, 128, 16, 2)])
def test_tile_schedules(probe, N, m, p, nrhs, slots, cl):
    r = subprocess.run([str(probe), str(N), str(m), str(p), str(nrhs), str(slots), str(cl)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    imposed = int(r.stdout.split("imposed=")[1])
    # per-sweep launches take the shape as it is: stage 1, then four per step
    assert imposed >= 1 + 4 * (N - 1) + 4 * (2 * N - 3), r.stdout

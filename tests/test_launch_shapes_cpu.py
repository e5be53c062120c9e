"""Rules that choose launch shapes on the host, on the CPU: a small program
(tests/host/shape_probe.cpp) compiled with csrc/geometry.cpp prints what they
choose over their whole range."""
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
    out = tmp_path_factory.mktemp("shapes") / "shape_probe"
    cmd = [cxx, "-std=c++17", "-O1", str(ROOT / "tests" / "host" / "shape_probe.cpp"), str(CSRC / "geometry.cpp"),
           "-I", str(ROOT / "include"), "-I", str(CSRC), "-I", str(cuda_inc), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(*args):
        r = subprocess.run([str(out), *args], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stdout + r.stderr
        return [[int(t) for t in line.split()] for line in r.stdout.splitlines()]
    return run


def test_complex128_slices_give_each_scheduler_two_warps(probe):
    """A line product of complex128 has more than one warp on each of the four
    schedulers wherever the columns, the lanes and the staging (64 KB) allow another
    slice, and never more than its bounds."""
    rows = probe("slices")
    assert len(rows) == 188 * 3 * 4
    for ny, cl, r, columns, q in rows:
        def fits(k):
            return k <= 16 and k * ny <= 384 and (k == 1 or (columns >= 2 * k and k * ny * r * 16 <= 65536))
        assert fits(q), (ny, cl, r, q)
        assert q * ny > 128 or not fits(q + 1), (ny, cl, r, q)

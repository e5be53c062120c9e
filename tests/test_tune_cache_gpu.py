"""The file of measured launch shapes (LSW_TUNE_CACHE): entries measured with other
kernels or another factor layout are not taken (their keys carry the revision of
what was measured), and a line of any length is read back whole."""
import json
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

_CHILD = r"""
import json, sys
sys.path[:0] = [{root!r}, {pkg!r}]
from lsweeps.problems import small
from lsweeps.solver import Solver
spec, med = small(N=3, m=12, p=4, medium="lens")
S = Solver(spec, med, precision="c64")
S.factorize()
print(json.dumps([S.front_shapes({nrhs})[1]]))
"""


def _tune_seconds(cache, nrhs):
    env = dict(os.environ, LSW_TUNE_CACHE=str(cache))
    code = _CHILD.format(root=str(ROOT), pkg=str(ROOT / "l-sweeps-2d_gb300"), nrhs=nrhs)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.strip().splitlines()[-1])[0]


@pytest.mark.parametrize("nrhs", [1, 3])
def test_entries_of_other_kernels_are_measured_again(nrhs, tmp_path):
    cache = tmp_path / "shapes.txt"
    assert _tune_seconds(cache, nrhs) > 0.0
    line = cache.read_text()
    assert _tune_seconds(cache, nrhs) == 0.0
    # the key as it was before revisions, and another revision's
    for other in (re.sub(r"\|rev\d+|\|tiles\d", "", line).replace("|sweeps", "|lanes"),
                  re.sub(r"\|rev\d+", "|rev1", line)):
        assert other != line
        cache.write_text(other)
        assert _tune_seconds(cache, nrhs) > 0.0


def test_long_lines_are_read_whole(tmp_path):
    cache = tmp_path / "shapes.txt"
    assert _tune_seconds(cache, 3) > 0.0
    cache.write_text(cache.read_text().replace(" ", " " * 70000, 1))
    assert _tune_seconds(cache, 3) == 0.0

"""Mixed solves without a preconditioner keep the rule's tile height, whatever the tuner measures or its cache file
holds: their iteration count follows the rounding, and so the tiling."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOLVE = f"""
import sys
sys.path.insert(0, {ROOT!r})
import cism_b200 as cg
from tests import problems
s = cg.DeviceSolver(problems.slab_2d(seed=1))
for precond in (0, 1):
    err, nit = s.solve(cg.ALG_MIXED_CHRONGEAR, precond, 5, 1e-8, 5000)
    print("RES", precond, err, nit, float(abs(s.x()[0]).sum()))
"""


def solve(cache, timing):
    env = dict(os.environ, CISMGPU_TILE_CACHE=str(cache), CISMGPU_TILE_TUNING=timing)
    r = subprocess.run([sys.executable, "-c", SOLVE], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    return dict(re.findall(r"RES (\d) (.*)", r.stdout))


def test_tile_height_without_a_preconditioner(gpu_lib, tmp_path):
    cache = tmp_path / "tiles.txt"
    rule = solve(cache, "0")
    assert not cache.exists()
    timed = solve(cache, "1")  # the diagonal solve meets the key and times it
    assert timed["0"] == rule["0"]
    key = cache.read_text().split()[0]
    for height in (6, 16):
        cache.write_text(f"{key} {height}\n")
        read = solve(cache, "0")
        assert read["0"] == rule["0"]
        assert read["1"] != rule["1"]  # the preconditioned solve follows the file

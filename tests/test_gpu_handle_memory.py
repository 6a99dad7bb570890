"""Device memory that handles leave behind: nothing stays with the library after the last handle, also in a
process that has made one-shot calls."""
import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import sys, gc
import numpy as np, torch
sys.path.insert(0, {root!r})
import cism_b200 as cg
from cism_b200 import assembly as asm
from tests import problems
MB = 1 << 20
def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free
small = problems.slab_3d(seed=1)
big = asm.ice_stream(96, 93, 11, seed=1)
def solve(P, alg=cg.ALG_CHRONGEAR):
    s = cg.DeviceSolver(P)
    s.solve(alg, 2, 5, 1e-6, 40)
    return s
def oneshot():
    xu, xv = np.zeros_like(small.bu), np.zeros_like(small.bv)
    cg.pcg_solver_chrongear_3d(small.nx, small.ny, small.nz, small.par, asm.indxA_2d(), asm.indxA_3d(),
                               small.active_vertex, small.Auu, small.Auv, small.Avu, small.Avv, small.bu, small.bv,
                               xu, xv, 2, 5, 1e-6, 40)
# kernels are loaded, and the staging buffers made, on first use
for alg in (cg.ALG_CHRONGEAR, cg.ALG_MIXED_CHRONGEAR):
    solve(big, alg).close()
"""


def run(body):
    env = dict(os.environ, CISMGPU_TILE_TUNING="0", CISMGPU_TILE_CACHE=os.devnull)
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT) + body], capture_output=True, text=True,
                       timeout=300, env=env)
    assert r.returncode == 0, r.stdout + r.stderr


def test_last_handle_returns_all(gpu_lib):
    run("""
base = used()
a, b = solve(big), solve(big)
size = (used() - base) // 2
assert size > 100 * MB
a.close(); b.close()
assert used() - base < 8 * MB
""")


def test_oneshot_call_keeps_nothing_of_handles(gpu_lib):
    run("""
oneshot()
base = used()
s = solve(big)
assert used() - base > 100 * MB
s.close()
assert used() - base < 8 * MB, (used() - base) / MB
""")


def test_server_budget_counts_what_requests_leave(gpu_lib):
    """Requests of falling sizes, whose blocks do not fit the next one, through a budget that holds the largest."""
    run("""
probs = [asm.ice_stream(n, n - 3, 11, seed=n) for n in (96, 84, 73, 64, 55)]
def nbytes(P):  # an upper bound of the largest request's bytes, as the server counts them
    return (P.nx - 1) * (P.ny - 1) * P.nz * (4 * 27 * 8 * 2 + 27 * 8 + 27 * 16 + 16 * 8 + 88) + 9 * MB
budget = nbytes(probs[0])
base = used()
srv = cg.Server(hbm_budget_bytes=budget)
peak = 0
for P in probs:
    rid = srv.submit(P, precond=2, ncheck=5, tol=1e-6, maxiters=200)
    srv.drain()
    assert srv.poll(rid)["done"]
    peak = max(peak, used() - base)
srv.close()
assert peak < budget + 16 * MB, (peak / MB, budget / MB)
assert used() - base < 8 * MB
""")

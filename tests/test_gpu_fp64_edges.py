"""FP64 solves where the fused kernels' dispatch changes: lines longer than one shared-memory chunk of
the line solver, level counts at the edges of the column solver's register variants (16, 32, more), and a
matrix above and below the size from which the symmetric half is read, exactly symmetric or not.  Bit
for bit against the oracle's restatement of the device reduction tree."""
import numpy as np
import pytest

import oracle
from cism_b200 import assembly as asm
from tests import problems

pytestmark = pytest.mark.gpu


def solve_both(alg, P, precond, maxiters):
    import cism_b200 as cg
    x0 = problems.random_x0(P, 3, 0.1)
    s = cg.DeviceSolver(P, x0=x0)
    try:
        err, nit = s.solve(cg.ALG_STANDARD if alg == "standard" else cg.ALG_CHRONGEAR, precond, 5, 1e-30, maxiters)
        xu, xv = s.x()
    finally:
        s.close()
    st, ou, ov, oerr, onit = oracle.pcg(alg, P, precond, maxiters=maxiters, tol=1e-30, x0=x0,
                                        summode=oracle.SUM_DDTREE)
    assert st == 0 and nit == onit and err == oerr
    assert np.array_equal(xu, ou) and np.array_equal(xv, ov)


@pytest.mark.parametrize("ewn,nsn", [(376, 7), (377, 8), (9, 753)])
@pytest.mark.parametrize("precond", [3, 4])
def test_long_lines(ewn, nsn, precond):
    """One chunk exactly, one position more, and three chunks."""
    solve_both("standard", problems.slab_2d(ewn, nsn, seed=5), precond, 6)


@pytest.mark.parametrize("nz", [2, 15, 16, 17, 32, 33])
@pytest.mark.parametrize("alg", ["standard", "chrongear"])
def test_level_counts(nz, alg):
    """Column solves in registers (up to 16, up to 32 levels) and through memory."""
    solve_both(alg, problems.slab_3d(7, 6, nz=nz, seed=nz), 2, 7)


@pytest.mark.parametrize("side,symmetric", [(78, True), (84, True), (84, False)])
def test_symmetric_half(side, symmetric):
    """The planes (below 64 MiB of blocks), the half, and the planes again for a matrix one bit off."""
    P = asm.ice_stream(side, side - 3, 11, seed=2)
    if not symmetric:
        P.Auv[side // 2, side // 2, 4, 17] = np.nextafter(P.Auv[side // 2, side // 2, 4, 17], np.inf)
    for alg in ("standard", "chrongear"):
        solve_both(alg, P, 2, 9)

"""The copies of a 3D matrix that a handle's solves make (the symmetric half, the full interleaved copy): what
they leave allocated, and solves while the matrix of a handle changes between exactly symmetric and not."""
import numpy as np
import pytest

from cism_b200 import assembly as asm

pytestmark = pytest.mark.gpu
SIDE, NZ = 84, 11


def matrix(symmetric, seed=2):
    """Above the size from which FP64 solves read the half; not symmetric: one coupling a bit off."""
    P = asm.ice_stream(SIDE, SIDE - 3, NZ, seed=seed)
    if not symmetric:
        P.Auv[SIDE // 2, SIDE // 2, 4, 17] = np.nextafter(P.Auv[SIDE // 2, SIDE // 2, 4, 17], np.inf)
    return P


def nodes(P):
    return P.bu.size


@pytest.mark.parametrize("symmetric", [True, False])
def test_half_is_held_only_for_a_symmetric_matrix(gpu_lib, symmetric):
    import cism_b200 as cg
    P = matrix(symmetric)
    half = 14 * 32 * nodes(P)
    s = cg.DeviceSolver(P)
    before = s.device_bytes()
    s.solve(cg.ALG_CHRONGEAR, 2, 5, 1e-30, 10)
    grown = s.device_bytes() - before
    assert grown >= half if symmetric else grown < half
    s.solve(cg.ALG_MIXED_CHRONGEAR, 2, 5, 1e-6, 200)
    full = s.device_bytes() - before
    assert s.mixed_symmetric_half() == symmetric
    s.close()
    f32 = (27 * 16 + 6 * 4 + 16 * 4) * nodes(P)
    copy = half if symmetric else 27 * 32 * nodes(P)
    assert f32 + copy <= full < f32 + copy + 64 * nodes(P) + (4 << 20)


@pytest.mark.parametrize("alg", ["chrongear", "mixed"])
def test_matrix_changes_on_a_handle(gpu_lib, alg):
    """Symmetric and not in turn on one handle: each solve as on a handle of its own."""
    import cism_b200 as cg
    a = cg.ALG_CHRONGEAR if alg == "chrongear" else cg.ALG_MIXED_CHRONGEAR

    def solve(s):
        r = s.solve(a, 2, 5, 1e-8, 60)
        return r, s.x()

    s = None
    for symmetric, seed in ((False, 2), (True, 3), (False, 4), (False, 5), (True, 2)):
        P = matrix(symmetric, seed)
        if s is None:
            s = cg.DeviceSolver(P)
        else:
            s.set_system(P.Auu, P.Auv, P.Avu, P.Avv, P.bu, P.bv, x0_from_solution=False)
        own = cg.DeviceSolver(P)
        got, want = solve(s), solve(own)
        own.close()
        assert got[0] == want[0]
        assert np.array_equal(got[1][0], want[1][0]) and np.array_equal(got[1][1], want[1][1])
    s.close()


@pytest.mark.parametrize("precond", [1, 2, 3, 4])
@pytest.mark.parametrize("reprosum", [0, 1])
def test_fp64_solve_takes_no_vectors_of_its_own(gpu_lib, precond, reprosum):
    """Below the half's size, a 3D solve's dot terms and column pivots add nothing to the handle (its bytes leave out the
    line preconditioners' planes and reprosum's product fields): where the handle fitted, so does its solve."""
    import cism_b200 as cg
    P = asm.ice_stream(40, 37, NZ, seed=3)
    P.par = dict(P.par, reprosum=reprosum)
    s = cg.DeviceSolver(P)
    before = s.device_bytes()
    s.solve(cg.ALG_CHRONGEAR, precond, 5, 1e-30, 10)
    s.solve(cg.ALG_STANDARD, precond, 5, 1e-30, 10)
    grown = s.device_bytes() - before
    s.close()
    assert grown == 0


@pytest.mark.parametrize("symmetric", [True, False])
def test_profiled_bytes_of_a_product(gpu_lib, symmetric):
    """The half's 14 couplings, or all 27: x and y, and r for the fused dot products."""
    import cism_b200 as cg
    P = matrix(symmetric)
    p = P.par
    own = P.active_vertex[p["staggered_jlo"] - 1:p["staggered_jhi"], p["staggered_ilo"] - 1:p["staggered_ihi"]]
    n = np.count_nonzero(own) * NZ
    s = cg.DeviceSolver(P)
    s.profile()
    s.solve(cg.ALG_CHRONGEAR, 2, 5, 1e-30, 10)
    _, launches, nbytes = s.profile_read()
    s.close()
    assert launches == 9
    assert nbytes == n * (4 * (14 if symmetric else 27) * 8 + 3 * 16)

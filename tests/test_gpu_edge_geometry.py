"""Owned vertices on the edge of the array, the geometry in which every coupling is tested against the
array: FP64 solves, products and residuals bit for bit against the oracle, and the mixed solver's full
layout.  The couplings that leave the array hold values that must not be read."""
import numpy as np
import pytest

import oracle
from cism_b200 import assembly as asm
from tests import problems

SHAPE = {2: (23, 19, 1), 3: (14, 12, 5)}


def system(dims, edges, bc="none", seed=1):
    """A symmetric, diagonally dominant matrix on all vertices but a few; edges: the owned sides on the edge."""
    nx, ny, nz = SHAPE[dims]
    NY, NX = ny - 1, nx - 1
    rng = np.random.default_rng(seed)
    nc = 27 if dims == 3 else 9
    A = 0.1 * rng.standard_normal((4, NY, NX, nz, nc))
    shape = (NY, NX, nz)
    for c in range(nc // 2 + 1):
        i, j, k = c % 3 - 1, c // 3 % 3 - 1, (c // 9 - 1 if nc == 27 else 0)
        to = tuple(slice(max(0, -o), n - max(0, o)) for o, n in zip((j, i, k), shape))
        at = tuple(slice(s.start + o, s.stop + o) for s, o in zip(to, (j, i, k)))
        for b, p in ((0, 0), (1, 2), (2, 1), (3, 3)):
            A[(b, *to, c)] = A[(p, *at, nc - 1 - c)]
    A[0, ..., nc // 2] += 12.0
    A[3, ..., nc // 2] += 12.0
    b = rng.standard_normal((2, NY, NX, nz))
    active = (rng.random((NY, NX)) > 0.1).astype(np.int32)
    par = dict(asm.default_par(nx, ny, bc="outflow"), periodic_bc=int(bc == "periodic"),
               outflow_bc=int(bc == "outflow"), no_ice_bc=int(bc == "no_ice"))
    par.update({"ilo": dict(staggered_ilo=1), "ihi": dict(staggered_ihi=nx - 1), "jlo": dict(staggered_jlo=1),
                "jhi": dict(staggered_jhi=ny - 1), "all": dict(staggered_ilo=1, staggered_ihi=nx - 1, staggered_jlo=1,
                                                               staggered_jhi=ny - 1)}[edges])
    on = np.zeros((NY, NX), dtype=bool)  # the unknowns
    on[par["staggered_jlo"] - 1:par["staggered_jhi"], par["staggered_ilo"] - 1:par["staggered_ihi"]] = True
    b *= (on & (active != 0))[..., None]
    if dims == 2:
        A, b = np.moveaxis(A[..., 0, :], -1, 1), b[..., 0]
    A, b = [np.ascontiguousarray(a) for a in A], [np.ascontiguousarray(v) for v in b]
    return asm.Problem("3d" if dims == 3 else "2d", nx, ny, nz, *A, *b, active, par)


def test_systems_are_solvable():
    for dims in (2, 3):
        st, *_, err, nit = oracle.pcg("chrongear", system(dims, "all"), 1, tol=1e-8, maxiters=100)
        assert st == 0 and err < 1e-8 and nit < 100


@pytest.mark.gpu
@pytest.mark.parametrize("alg", ["standard", "chrongear"])
@pytest.mark.parametrize("dims,precond", [(d, p) for d in (2, 3) for p in range(5) if (d, p) != (2, 2)])
@pytest.mark.parametrize("edges,bc", [("all", "none"), ("all", "no_ice"), ("all", "outflow"), ("jlo", "outflow"),
                                      ("all", "periodic"), ("ihi", "periodic"), ("ilo", "none"), ("ihi", "none"),
                                      ("jlo", "none"), ("jhi", "none")])
def test_fp64_solve(gpu_lib, dims, edges, bc, precond, alg):
    import cism_b200 as cg
    P = system(dims, edges, bc)
    x0 = problems.random_x0(P, 3, 0.1)
    st, ou, ov, oerr, onit = oracle.pcg(alg, P, precond, maxiters=9, tol=1e-30, x0=x0, summode=oracle.SUM_DDTREE)
    assert st == 0
    s = cg.DeviceSolver(P, x0=x0)
    err, nit = s.solve(cg.ALG_STANDARD if alg == "standard" else cg.ALG_CHRONGEAR, precond, 5, 1e-30, 9)
    xu, xv = s.x()
    s.close()
    assert (err, nit) == (oerr, onit)
    np.testing.assert_array_equal(xu, ou)
    np.testing.assert_array_equal(xv, ov)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [2, 3])
def test_product_and_residual(gpu_lib, dims):
    import cism_b200 as cg
    P = system(dims, "all")
    x = problems.random_x0(P, 5)
    want = oracle.matvec(P, *x)
    if dims == 3:
        got = cg.matvec_multiply_structured_3d(P.nx, P.ny, P.nz, P.par, asm.indxA_3d(), P.active_vertex, P.Auu, P.Auv, P.Avu,
                                               P.Avv, *x)
    else:
        got = cg.matvec_multiply_structured_2d(P.nx, P.ny, P.par, asm.indxA_2d(), P.active_vertex, P.Auu, P.Auv, P.Avu,
                                               P.Avv, *x)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    s = cg.DeviceSolver(P, x0=x)
    ru, rv, *norms = s.residual_vector()
    s.close()
    wu, wv, *wnorms = oracle.residual_vector(P, *x, summode=oracle.SUM_DDTREE)
    np.testing.assert_array_equal(ru, wu)
    np.testing.assert_array_equal(rv, wv)
    assert tuple(norms) == tuple(wnorms)


@pytest.mark.gpu
@pytest.mark.parametrize("edges", ["all", "ilo", "jhi"])
@pytest.mark.parametrize("dims,precond", [(2, 1), (3, 1), (3, 2)])
def test_mixed_full_layout(gpu_lib, dims, precond, edges):
    """err is the FP64 residual; x within cond(A) times it of the FP64 solution.  Gershgorin: the eigenvalues lie in
    12 +- sum |couplings|, about 12 +- 6, so cond(A) < 10."""
    import cism_b200 as cg
    P = system(dims, edges)
    s = cg.DeviceSolver(P)
    err, nit = s.solve(cg.ALG_MIXED_CHRONGEAR, precond, 5, 1e-10, 200)
    assert not s.mixed_symmetric_half()
    xu, xv = s.x()
    s.close()
    st, ou, ov, oerr, onit = oracle.pcg("chrongear", P, precond, maxiters=200, tol=1e-12)
    assert st == 0 and err < 1e-10
    num = np.sqrt(np.sum((xu - ou) ** 2) + np.sum((xv - ov) ** 2))
    assert num < 10 * 2e-10 * np.sqrt(np.sum(ou ** 2) + np.sum(ov ** 2))

"""Chronopoulos-Gear with the line preconditioners where the staggered halo update of r reaches owned
vertices: under no_ice it zeroes the last owned row and column, which the lines run through, and the
reference updates r before its first preconditioner (glissade_velo_higher_pcg.F90:3118-3121) and after
every check.  The systems were not halo-updated by their caller, so r = b - A x is not zero
there beforehand.  Bit for bit against the oracle, in every order of the global sums."""
import contextlib

import numpy as np
import pytest

import oracle
from cism_b200 import assembly as asm
from tests import problems


def system(dims, seed):
    """Ice up to the last owned vertices, no_ice, A and b as assembled."""
    rng = np.random.default_rng(seed)
    nx, ny, dx = 14, 13, 2000.0
    thck = 800.0 + 400.0 * rng.random((ny, nx))
    ice = np.zeros((ny, nx), dtype=bool)
    ice[3:ny - 1, 3:nx - 1] = True
    thck = np.where(ice, thck, 0.0)
    beta = asm.lognormal_beta((ny - 1, nx - 1), seed + 100)
    if dims == 2:
        P = asm.assemble_ssa_2d(thck, thck.copy(), dx, dx, beta, bc="no_ice", name="noice2")
    else:
        usrf = 2000.0 - 20.0 * np.arange(nx)[None, :] + 30.0 * rng.random((ny, nx))
        P = asm.assemble_bp_3d(thck, np.where(ice, usrf, usrf - 900.0), dx, dx, 5, beta=beta, bc="no_ice", name="noice3")
    p = P.par
    halo = np.ones(P.active_vertex.shape, dtype=bool)
    halo[p["staggered_jlo"] - 1:p["staggered_jhi"], p["staggered_ilo"] - 1:p["staggered_ihi"]] = False
    P.active_vertex = np.where(halo, 0, P.active_vertex).astype(np.int32)  # a halo column has no matrix
    return P


CASES = [(dims, precond, start) for dims in (2, 3) for precond in (3, 4) for start in ("zero", "random")]


def start_of(P, start):
    return problems.random_x0(P, seed=11, scale=10.0) if start == "random" else (np.zeros_like(P.bu), np.zeros_like(P.bv))


@pytest.mark.parametrize("dims,precond,start", CASES)
def test_halo_of_r_matters(dims, precond, start):
    """The inputs: the oracle solves them, past a check, and r is not zero where the update zeroes it."""
    P = system(dims, 4)
    x0 = start_of(P, start)
    yu, yv = oracle.matvec(P, *(oracle.halo(P.nx, P.ny, P.nz, P.par, a) for a in x0))
    i, j = P.par["staggered_ihi"] - 1, P.par["staggered_jhi"] - 1
    r = np.abs(P.bu - yu) + np.abs(P.bv - yv)
    assert r[:, i].max() > 0 and r[j, :].max() > 0
    assert np.array_equal(oracle.halo(P.nx, P.ny, P.nz, P.par, r)[:, i], np.zeros_like(r[:, i]))
    st, *_ = oracle.pcg("chrongear", P, precond, tol=1e-30, maxiters=12, x0=x0)
    assert st == 0


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["tree", "sequential", "reprosum"])
@pytest.mark.parametrize("dims,precond,start", CASES)
def test_lines_after_the_halo_of_r(gpu_lib, dims, precond, start, order):
    import cism_b200 as cg
    P = system(dims, 4)
    if order == "reprosum":
        P.par["reprosum"] = 1
    x0 = start_of(P, start)
    mode = {"tree": oracle.SUM_DDTREE, "sequential": oracle.SUM_SEQ, "reprosum": oracle.SUM_REPRO}[order]
    with cg.sum_order(cg.SUM_SEQUENTIAL) if order == "sequential" else contextlib.nullcontext():
        s = cg.DeviceSolver(P, x0=x0)
        err, nit = s.solve(cg.ALG_CHRONGEAR, precond, 5, 1e-30, 12)
        xu, xv = s.x()
        s.close()
    st, ou, ov, oerr, onit = oracle.pcg("chrongear", P, precond, tol=1e-30, maxiters=12, x0=x0, summode=mode)
    assert st == 0 and (nit, err) == (onit, oerr)
    np.testing.assert_array_equal(xu, ou)
    np.testing.assert_array_equal(xv, ov)

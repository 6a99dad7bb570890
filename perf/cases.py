"""The work that users of this library have it do, as cases that can be timed.

Each case is one pass through the public entry points (cism_b200): the reference-signature calls on
host arrays, solves on device-resident handles in FP64 and in mixed precision, a batch captured in a
CUDA graph, a burst of served requests, and the assembly and residual steps of a Picard iteration.
Sizes are those of the library's configurations and tests, with ragged ones beside them.

The systems are built here with torch: first-Picard Blatter-Pattyn (27-point) and SSA (9-point)
blocks of synthetic ice, in the caller's layout.  exact() solves the same systems in 64 bits
with torch alone.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

# Tile heights from the library's rule instead of its timing tuner and the tuner's cache file: a
# system then has one tiling, and one rounding, in every process.
os.environ["CISMGPU_TILE_TUNING"] = "0"
os.environ["CISMGPU_TILE_CACHE"] = os.devnull

import cism_b200 as cg
from cism_b200 import assembly as asm

DEV = "cuda"
TOL = 1.0e-8
NCHECK = 5
MAXITERS = 20000
HALO = asm.NHALO
F64 = torch.float64
NONE, DIAG, SIA, LINES = 0, 1, 2, 3
ALGORITHMS = {"standard": cg.ALG_STANDARD, "chrongear": cg.ALG_CHRONGEAR, "mixed": cg.ALG_MIXED_CHRONGEAR}


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
# geometry: "dome" (no-slip parabolic dome), "stream" (no-slip ice stream), "slide" (ice stream
# sliding on its own log-normal friction), "ssa" (2D, log-normal friction)
def listed():
    return [
        # the reference's own CPU configuration through the drop-in call: host arrays in, host
        # arrays out, standard PCG and the diagonal preconditioner
        dict(name="dome_call_standard", do="call", geometry="dome", ni=31, nj=31, nz=11, algorithm="standard",
             precond=DIAG),
        # the smallest solves, bound by latency: the dome on a handle, FP64 and mixed
        dict(name="dome_fp64", do="solve", geometry="dome", ni=31, nj=31, nz=11, algorithm="chrongear", precond=SIA),
        dict(name="dome_mixed", do="solve", geometry="dome", ni=31, nj=31, nz=11, algorithm="mixed", precond=SIA),
        # the 880k-unknown ice stream, FP64 (the drop-in arithmetic) and mixed
        dict(name="stream_fp64", do="solve", geometry="stream", ni=201, nj=201, nz=11, algorithm="chrongear",
             precond=SIA),
        dict(name="stream_mixed", do="solve", geometry="stream", ni=201, nj=201, nz=11, algorithm="mixed",
             precond=SIA),
        # more levels than the 16-level kernels take, ragged sizes
        dict(name="stream21_mixed", do="solve", geometry="stream", ni=131, nj=97, nz=21, algorithm="mixed",
             precond=SIA),
        # a sliding system with the tridiagonal line preconditioner, FP64, ragged
        dict(name="slide_lines_fp64", do="solve", geometry="slide", ni=150, nj=101, nz=11, algorithm="chrongear",
             precond=LINES),
        # 2D SSA: thousands of short iterations, FP64 and mixed, the latter ragged
        dict(name="ssa_fp64", do="solve", geometry="ssa", ni=401, nj=401, nz=1, algorithm="chrongear", precond=DIAG),
        dict(name="ssa_mixed", do="solve", geometry="ssa", ni=321, nj=257, nz=1, algorithm="mixed", precond=DIAG),
        # an ensemble of uneven sliding systems replayed as one CUDA graph
        dict(name="batch_mixed", do="batch", geometry="slide", members=6, lo=64, hi=256, nz=11, algorithm="mixed",
             precond=SIA),
        # one Picard iteration's assembly, symmetry check and residual on a handle
        dict(name="picard_system", do="picard", geometry="slide", ni=201, nj=161, nz=11),
        # a burst of mixed 2D and 3D requests through the serving loop (uploads included)
        dict(name="served_burst", do="serve", requests=6, lo=48, hi=256, algorithm="mixed"),
    ]


def draw(rng):
    """One more case over the ranges of the listed ones."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["call", "solve3", "solve3", "solve3", "solve2", "solve2", "batch", "picard", "serve"])
    if do == "call":
        if rng.random() < 0.5:
            return dict(do="call", geometry=rng.choice(["dome", "stream"]), ni=size(24, 128), nj=size(24, 128),
                        nz=rng.randint(5, 16), algorithm=rng.choice(["standard", "chrongear"]),
                        precond=rng.choice([DIAG, SIA]))
        return dict(do="call", geometry="ssa", ni=size(32, 256), nj=size(32, 256), nz=1,
                    algorithm=rng.choice(["standard", "chrongear"]), precond=DIAG)
    if do == "solve3":
        geometry = rng.choice(["dome", "stream", "stream", "slide"])
        return dict(do="solve", geometry=geometry, ni=size(28, 128 if geometry == "slide" else 224),
                    nj=size(28, 128 if geometry == "slide" else 224), nz=rng.randint(5, 21),
                    algorithm=rng.choice(["chrongear", "mixed", "mixed"]), precond=rng.choice([SIA, SIA, LINES]))
    if do == "solve2":
        return dict(do="solve", geometry="ssa", ni=size(48, 400), nj=size(48, 400), nz=1,
                    algorithm=rng.choice(["chrongear", "mixed", "standard"]), precond=DIAG)
    if do == "batch":
        return dict(do="batch", geometry="slide", members=rng.randint(2, 6), lo=rng.randint(40, 64),
                    hi=rng.randint(96, 200), nz=rng.randint(6, 14), algorithm="mixed",
                    precond=rng.choice([SIA, LINES]))
    if do == "picard":
        return dict(do="picard", geometry="slide", ni=size(32, 200), nj=size(32, 200), nz=rng.randint(5, 16))
    return dict(do="serve", requests=rng.randint(3, 6), lo=rng.randint(40, 64), hi=rng.randint(96, 224),
                algorithm="mixed")


# ---------------------------------------------------------------------------------------------
# synthetic systems (torch, FP64)
# ---------------------------------------------------------------------------------------------
R3 = 1.0 / math.sqrt(3.0)
SX = (-1, 1, 1, -1, -1, 1, 1, -1)
SY = (-1, -1, 1, 1, -1, -1, 1, 1)
SZ = (-1, -1, -1, -1, 1, 1, 1, 1)
BI, BJ = (0, 1, 1, 0) * 2, (0, 0, 1, 1) * 2          # a node's vertex within its cell's 2 x 2
BK = (1, 1, 1, 1, 0, 0, 0, 0)                        # a node's level below its layer's upper one


def _rng(seed):
    return torch.Generator().manual_seed(seed & 0x7FFFFFFF)


def _randn(shape, seed):
    return torch.randn(shape, generator=_rng(seed), dtype=F64).to(DEV)


def _smooth(shape, cells, seed):
    """A random field of unit variance, smooth over about `cells` cells."""
    f = torch.fft.fft2(_randn(shape, seed))
    ky = torch.fft.fftfreq(shape[0], dtype=F64, device=DEV)[:, None]
    kx = torch.fft.fftfreq(shape[1], dtype=F64, device=DEV)[None, :]
    f = torch.fft.ifft2(f * torch.exp(-2.0 * (math.pi * cells) ** 2 * (kx * kx + ky * ky))).real
    f = f - f.mean()
    return f / f.std().clamp_min(1e-30)


def _corners(f):
    """The four vertices of every interior cell, or the four cells around every vertex."""
    return f[:-1, :-1], f[:-1, 1:], f[1:, 1:], f[1:, :-1]


def _geometry(case, seed):
    """Cell fields and masks of a case's ice, halo included."""
    kind, ni, nj = case["geometry"], case["ni"], case["nj"]
    nx, ny = ni + 2 * HALO, nj + 2 * HALO
    dx = 1000.0 if kind == "ssa" else 2000.0
    inside = torch.zeros((ny, nx), dtype=torch.bool, device=DEV)
    inside[HALO + 1:ny - HALO - 1, HALO + 1:nx - HALO - 1] = True
    x = ((torch.arange(nx, device=DEV, dtype=F64) + 0.5) * dx)[None, :].expand(ny, nx)
    y = ((torch.arange(ny, device=DEV, dtype=F64) + 0.5) * dx)[:, None].expand(ny, nx)
    slope = 0.0
    if kind == "dome":  # H = H0 sqrt(1 - r^2/R^2) on a flat bed, R scaled with the domain
        ri, rj = 0.5 * ni * dx * 0.81, 0.5 * nj * dx * 0.81
        r2 = ((x - 0.5 * nx * dx) / ri) ** 2 + ((y - 0.5 * ny * dx) / rj) ** 2
        thck = 1000.0 * (1.0 + 0.02 * _smooth((ny, nx), 4.0, seed + 1)) * torch.sqrt((1.0 - r2).clamp_min(0.0))
        thck = torch.where(inside & (r2 < 1.0), thck, 0.0)
        usrf = thck.clone()
    elif kind == "ssa":
        f = _smooth((ny, nx), 20.0, seed + 1)
        thck = torch.where(inside, 500.0 + 1500.0 * (f - f.min()) / (f.max() - f.min()), 0.0)
        usrf = thck.clone()
    else:
        slope = math.tan(math.radians(0.5))
        top = 3000.0 - x * slope
        bed = top - 1500.0 + (0.05 * 1500.0 * _smooth((ny, nx), 4.0, seed + 1) if kind == "stream" else 0.0)
        if kind == "slide":  # a plane bed under a rough surface
            top = top + 0.02 * 1500.0 * _smooth((ny, nx), 6.0, seed + 1)
        thck = torch.where(inside, top - bed, 0.0)
        usrf = torch.where(inside, top, bed)
    ice = thck > 1.0
    cell = torch.zeros_like(ice)
    cell[HALO:ny - HALO + 1, HALO:nx - HALO + 1] = ice[HALO:ny - HALO + 1, HALO:nx - HALO + 1]
    a, b, c, d = _corners(cell)
    vertex = a | b | c | d
    n = sum(f.to(F64) for f in _corners(ice))

    def stagger(f):
        return sum(torch.where(ice, f, 0.0)[s] for s in CORNERS) / n.clamp_min(1.0)

    f00, f01, f11, f10 = _corners(usrf)
    sx, sy = ((f01 + f11) - (f00 + f10)) / (2.0 * dx), ((f10 + f11) - (f00 + f01)) / (2.0 * dx)
    beta = torch.exp(math.log(1.0e3) + _randn((ny - 1, nx - 1), seed + 2))
    return dict(nx=nx, ny=ny, dx=dx, cell=cell, vertex=vertex, thck=stagger(thck), usrf=stagger(usrf), sx=sx, sy=sy,
                beta=beta, slope=slope, lsrf=usrf - thck)


CORNERS = ((slice(None, -1), slice(None, -1)), (slice(None, -1), slice(1, None)), (slice(1, None), slice(1, None)),
           (slice(1, None), slice(None, -1)))
FLWA = 1.0e-16
FLWAFACT = 0.5 * FLWA ** (-1.0 / 3.0)
EFVS0 = FLWAFACT * (1.0e-8 ** 2) ** (-1.0 / 3.0)


def _loads(g, nz):
    sigma = _sigma(nz)
    w = torch.cat([torch.zeros(1, dtype=F64, device=DEV), 0.5 * (sigma[:-1] + sigma[1:]),
                   torch.ones(1, dtype=F64, device=DEV)])
    f = -asm.RHOI * asm.GRAV * g["dx"] ** 2 / asm.VOL0 * g["thck"][..., None] * (w[1:] - w[:-1])
    on = g["vertex"][..., None]
    return [torch.where(on, f * s[..., None], 0.0).contiguous() for s in (g["sx"], g["sy"])]


def _sigma(nz):
    return torch.from_numpy(asm.glide_sigma(nz)).to(DEV)


def _layer(g, nz, k):
    """The basis functions' derivatives (8 points, 8 nodes, cells) and detJ (8 points, cells) of layer k."""
    sigma, h = _sigma(nz), 0.5 * g["dx"]
    z = [(g["usrf"] - sigma[k + BK[n]] * g["thck"])[CORNERS[n % 4]] for n in range(8)]
    on = g["cell"][1:-1, 1:-1]
    dx, dy, dz, det = [], [], [], []
    for p in range(8):
        xq, yq, zq = SX[p] * R3, SY[p] * R3, SZ[p] * R3
        dr = [[SX[n] * (1 + SY[n] * yq) * (1 + SZ[n] * zq) / 8 for n in range(8)],
              [SY[n] * (1 + SX[n] * xq) * (1 + SZ[n] * zq) / 8 for n in range(8)],
              [SZ[n] * (1 + SX[n] * xq) * (1 + SY[n] * yq) / 8 for n in range(8)]]
        zx, zy, zz = (sum(dr[a][n] * z[n] for n in range(8)) for a in range(3))
        zz = torch.where(on, zz, 1.0)
        dx.append(torch.stack([(dr[0][n] - zx / zz * dr[2][n]) / h for n in range(8)]))
        dy.append(torch.stack([(dr[1][n] - zy / zz * dr[2][n]) / h for n in range(8)]))
        dz.append(torch.stack([dr[2][n] / zz for n in range(8)]))
        det.append(h * h * zz)
    return torch.stack(dx), torch.stack(dy), torch.stack(dz), torch.stack(det)


def _viscosity(g, nz, k, grads, u, v):
    """Glen's viscosity (8 points, cells) of layer k for the velocity u, v (NY, NX, nz)."""
    un = torch.stack([u[..., k + BK[n]][CORNERS[n % 4]] for n in range(8)])
    vn = torch.stack([v[..., k + BK[n]][CORNERS[n % 4]] for n in range(8)])
    ux, uy, uz = ((d * un).sum(1) for d in grads)
    vx, vy, vz = ((d * vn).sum(1) for d in grads)
    sq = 1.0e-8 ** 2 + ux * ux + vy * vy + ux * vy + 0.25 * ((vx + uy) ** 2 + uz * uz + vz * vz)
    return FLWAFACT * sq ** (-1.0 / 3.0)


def _lower_from_upper(A):
    """Lower couplings from their transpose partners: the symmetric matrix that the reference's check leaves."""
    A[2, ..., 13] = A[1, ..., 13]
    NY, NX, nz = A.shape[1:4]
    for c in range(13):
        i, j, k = c % 3 - 1, c // 3 % 3 - 1, c // 9 - 1
        to = (slice(max(0, -j), NY - max(0, j)), slice(max(0, -i), NX - max(0, i)), slice(max(0, -k), nz - max(0, k)))
        at = tuple(slice(s.start + d, s.stop + d) for s, d in zip(to, (j, i, k)))
        for b, p in ((0, 0), (1, 2), (2, 1), (3, 3)):
            A[(b, *to, c)] = A[(p, *at, 26 - c)]


def _blocks_3d(g, nz, velocity=None):
    """The Blatter-Pattyn stiffness blocks (uu, uv, vu, vv) as (4, ny-1, nx-1, nz, 27), and the viscosity."""
    NY, NX = g["vertex"].shape
    A = torch.zeros((4, NY, NX, nz, 27), dtype=F64, device=DEV)
    on = g["cell"][1:-1, 1:-1]
    efvs = torch.zeros((g["ny"], g["nx"], nz - 1), dtype=F64, device=DEV)
    for k in range(nz - 1):
        dx, dy, dz, det = _layer(g, nz, k)
        mu = EFVS0 if velocity is None else _viscosity(g, nz, k, (dx, dy, dz), *velocity)
        f = torch.where(on, mu * det / asm.VOL0, 0.0)
        if velocity is not None:
            efvs[1:-1, 1:-1, k] = torch.where(on, mu.mean(0), 0.0)
        for r in range(8):
            for s in range(8):
                c = (BI[s] - BI[r] + 1) + 3 * (BJ[s] - BJ[r] + 1) + 9 * (BK[s] - BK[r] + 1)
                if c < 13:
                    continue
                xx, yy, zz = ((f * (d[:, r] * d[:, s])).sum(0) for d in (dx, dy, dz))
                xy, yx = (f * (dx[:, r] * dy[:, s])).sum(0), (f * (dy[:, r] * dx[:, s])).sum(0)
                at = (*CORNERS[r % 4], k + BK[r], c)
                for b, t in enumerate((4 * xx + yy + zz, 2 * xy + yx, 2 * yx + xy, 4 * yy + xx + zz)):
                    A[(b, *at)] += t
    return A, efvs


def _system_3d(case, seed):
    """One first-Picard system: A (4, ny-1, nx-1, nz, 27) and bu, bv on the GPU, and its geometry."""
    g, nz = _geometry(case, seed), case["nz"]
    A, _ = _blocks_3d(g, nz)
    bu, bv = _loads(g, nz)
    if case["geometry"] == "slide":
        drag = _drag(g)
        A[0, ..., nz - 1, 13] += drag
        A[3, ..., nz - 1, 13] += drag
    else:  # no-slip: identity rows at the bed
        bed = g["vertex"]
        for c in range(18, 27):  # couplings down to the bed
            i, j = c % 3 - 1, c // 3 % 3 - 1
            A[:, :, :, nz - 2, c] *= ~torch.roll(bed, (-j, -i), (0, 1))
        A[:, :, :, nz - 1][:, bed] = 0.0
        for b in (0, 3):
            A[b, :, :, nz - 1, 13] += bed.to(F64)
        for v in (bu, bv):
            v[..., nz - 1] *= ~bed
    _lower_from_upper(A)
    return A, bu, bv, g


def _drag(g):
    return torch.where(g["vertex"], g["dx"] ** 2 / asm.VOL0 * g["beta"] * math.sqrt(1.0 + g["slope"] ** 2), 0.0)


def _system_2d(case, seed):
    """One SSA system: A (4, 9, ny-1, nx-1) and bu, bv on the GPU, and its geometry."""
    g = _geometry(case, seed)
    NY, NX = g["vertex"].shape
    A = torch.zeros((4, 9, NY, NX), dtype=F64, device=DEV)
    on, h = g["cell"][1:-1, 1:-1], 0.5 * g["dx"]
    H = [g["thck"][s] for s in CORNERS]
    for p in range(4):
        xq, yq = SX[p] * R3, SY[p] * R3
        hq = sum((1 + SX[n] * xq) * (1 + SY[n] * yq) / 4 * H[n] for n in range(4))
        f = torch.where(on, hq * EFVS0 * h * h / asm.VOL0, 0.0)
        dx = [SX[n] * (1 + SY[n] * yq) / 4 / h for n in range(4)]
        dy = [SY[n] * (1 + SX[n] * xq) / 4 / h for n in range(4)]
        for r in range(4):
            for s in range(4):
                c = (BI[s] - BI[r] + 1) + 3 * (BJ[s] - BJ[r] + 1)
                xx, yy, xy, yx = dx[r] * dx[s], dy[r] * dy[s], dx[r] * dy[s], dy[r] * dx[s]
                for b, t in enumerate((4 * xx + yy, 2 * xy + yx, 2 * yx + xy, 4 * yy + xx)):
                    A[(b, c, *CORNERS[r])] += f * t
    drag = _drag(g)
    A[0, 4] += drag
    A[3, 4] += drag
    f = torch.where(g["vertex"], -asm.RHOI * asm.GRAV * g["dx"] ** 2 / asm.VOL0 * g["thck"], 0.0)
    return A, f * g["sx"], f * g["sy"], g


def _is3d(case):
    return case["geometry"] != "ssa"


def _system(case, seed):
    return (_system_3d if _is3d(case) else _system_2d)(case, seed)


def _problem(case, seed):
    """The system as a host program holds it: numpy arrays in the caller's layout."""
    A, bu, bv, g = _system(case, seed)
    A, bu, bv = A.cpu().numpy(), bu.cpu().numpy(), bv.cpu().numpy()
    return asm.Problem("3d" if _is3d(case) else "2d", g["nx"], g["ny"], case["nz"], A[0], A[1], A[2], A[3], bu, bv,
                       g["vertex"].to(torch.int32).cpu().numpy(), asm.default_par(g["nx"], g["ny"]))


def _pinned(shape):
    return torch.zeros(shape, dtype=F64, pin_memory=True).numpy()


def _members(case):
    """The systems of a batch: uneven sizes from lo to hi, every other side shortened."""
    n = case["members"]
    out = []
    for k in range(n):
        side = int(round(case["lo"] + (case["hi"] - case["lo"]) * k / max(1, n - 1)))
        out.append(dict(geometry=case["geometry"], ni=side, nj=side - 7 * (k % 2), nz=case["nz"], algorithm="mixed",
                        precond=case["precond"]))
    return out


def _requests(case):
    """The systems of a served burst: 2D and 3D in turn, sizes and level counts from small to large."""
    n = case["requests"]
    out = []
    for k in range(n):
        side = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (k / max(1, n - 1))))
        if k % 2:
            out.append(dict(geometry="ssa", ni=side, nj=side - 5, nz=1, algorithm="mixed", precond=DIAG))
        else:
            out.append(dict(geometry="stream", ni=side // 2 + 16, nj=side // 2 + 11, nz=5 + 4 * (k % 5),
                            algorithm="mixed", precond=SIA))
    return out


# ---------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    do = case["do"]
    if do == "call":
        P = _problem(case, seed)
        return dict(case=case, problem=P, zero=np.zeros_like(P.bu))
    if do == "solve":
        P = _problem(case, seed)
        return dict(case=case, solver=cg.DeviceSolver(P), xu=_pinned(P.bu.shape), xv=_pinned(P.bv.shape))
    if do == "batch":
        solvers = [cg.DeviceSolver(_problem(m, seed + 1000 * k)) for k, m in enumerate(_members(case))]
        batch = cg.GraphBatch(solvers, precond=case["precond"], ncheck=NCHECK, tol=TOL, maxiters=MAXITERS)
        return dict(case=case, solvers=solvers, batch=batch,
                    x=[(_pinned(s.problem.bu.shape), _pinned(s.problem.bv.shape)) for s in solvers])
    if do == "serve":
        return dict(case=case, server=cg.Server(), requests=[(_problem(r, seed + 1000 * k), r["precond"])
                                                             for k, r in enumerate(_requests(case))])
    inputs, u, v, g = _picard_inputs(case, seed)
    nz = case["nz"]
    nodes = g["vertex"].shape + (nz,)
    zero = np.zeros(nodes + (27,))
    P = asm.Problem("3d", g["nx"], g["ny"], nz, zero, zero, zero, zero, np.zeros(nodes), np.zeros(nodes),
                    g["vertex"].to(torch.int32).cpu().numpy(), asm.default_par(g["nx"], g["ny"]))
    return dict(case=case, solver=cg.DeviceSolver(P, x0=(u.cpu().numpy(), v.cpu().numpy())), inputs=inputs)


def _picard_inputs(case, seed):
    """What the assembly of one Picard iteration takes, and the velocity it starts from."""
    g, nz = _geometry(case, seed), case["nz"]
    profile = 1.0 - 0.8 * _sigma(nz) ** 4
    on = g["vertex"][..., None]
    u, v = (torch.where(on, s * (1.0 + 0.1 * _smooth(g["vertex"].shape, 8.0, seed + 3 + i))[..., None] * profile, 0.0)
            for i, s in enumerate((60.0, 8.0)))
    loadu, loadv = (t.cpu().numpy() for t in _loads(g, nz))
    NY, NX = g["vertex"].shape
    xv, yv = np.meshgrid(np.arange(NX) * g["dx"], np.arange(NY) * g["dx"])
    host = {k: np.ascontiguousarray(g[k].cpu().numpy()) for k in ("thck", "usrf", "beta", "lsrf")}
    inputs = dict(nhalo=HALO, dx=g["dx"], dy=g["dx"], sigma=asm.glide_sigma(nz),
                  active_cell=g["cell"].to(torch.int32).cpu().numpy(),
                  active_vertex=g["vertex"].to(torch.int32).cpu().numpy(), xVertex=xv, yVertex=yv,
                  stagusrf=host["usrf"], stagthck=host["thck"],
                  flwafact=np.full((g["ny"], g["nx"], nz - 1), FLWAFACT), loadu=loadu, loadv=loadv, beta=host["beta"],
                  lsrf=host["lsrf"])
    return inputs, u.contiguous(), v.contiguous(), g


def _call(P, algorithm, precond, xu, xv):
    tail = (P.active_vertex, P.Auu, P.Auv, P.Avu, P.Avv, P.bu, P.bv, xu, xv, precond, NCHECK, TOL, MAXITERS)
    if P.kind == "3d":
        f = cg.pcg_solver_standard_3d if algorithm == "standard" else cg.pcg_solver_chrongear_3d
        return f(P.nx, P.ny, P.nz, P.par, asm.indxA_2d(), asm.indxA_3d(), *tail)
    f = cg.pcg_solver_standard_2d if algorithm == "standard" else cg.pcg_solver_chrongear_2d
    return f(P.nx, P.ny, P.par, asm.indxA_2d(), *tail)


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "call":
        xu, xv = state["zero"].copy(), state["zero"].copy()
        _, niters = _call(state["problem"], case["algorithm"], case["precond"], xu, xv)
        return {"xu": xu, "xv": xv, "niters": niters}
    if do == "solve":
        s = state["solver"]
        _, niters = s.solve(ALGORITHMS[case["algorithm"]], case["precond"], NCHECK, TOL, MAXITERS)
        s.x_into(state["xu"], state["xv"])
        out = {"xu": state["xu"], "xv": state["xv"]}
        if case["algorithm"] != "mixed":  # FP64: the reference's own iteration count
            out["niters"] = niters
        return out
    if do == "batch":
        state["batch"].run()
        state["batch"].wait()
        for s, x in zip(state["solvers"], state["x"]):
            s.x_into(*x)
        return {"x": state["x"]}
    if do == "serve":
        server = state["server"]
        ids = [server.submit(P, precond=pc, ncheck=NCHECK, tol=TOL, maxiters=MAXITERS) for P, pc in state["requests"]]
        server.drain()
        return {"x": [server.result(i)[:2] for i in ids]}
    s = state["solver"]
    efvs = s.assemble_system(**state["inputs"])
    s.check_symmetry()
    ru, rv, norm, _ = s.residual_vector()
    return {"efvs": efvs, "resid_u": ru, "resid_v": rv, "norm": norm}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _iterations(case):
    """About how many iterations a system of this kind takes to 1e-8 (measured: the dome 180 with the
    diagonal and 25 with the SIA preconditioner, ice streams 25, sliding ones ten a vertex of their longer
    side, half that with lines, SSA nine)."""
    side = max(case["ni"], case["nj"])
    if case["geometry"] == "ssa":
        return 9 * side
    if case["geometry"] == "slide":
        return (10 if case["precond"] == SIA else 5) * side
    return 25 if case["precond"] != DIAG else 180


def _solve_work(case):
    """One solve: per iteration the matrix (its symmetric half in 3D) and the vectors once, in FP64 or, in
    mixed precision, in FP32 with an FP64 matrix every NCHECK iterations."""
    nodes = (case["ni"] - 1) * (case["nj"] - 1) * case["nz"]
    stored, couplings = (14, 27) if _is3d(case) else (9, 9)
    word = 4 if case["algorithm"] == "mixed" else 8
    vectors = 2 * 12 * word + (6 * word if case["precond"] == SIA else 2 * word)
    n = _iterations(case)
    check = 4 * stored * 8 + 40
    nbytes = nodes * (n * (4 * stored * word + vectors) + n / NCHECK * check)
    flops = nodes * (n * (8 * couplings + 40) + n / NCHECK * 8 * couplings)
    return nbytes, flops


def work(case):
    do = case["do"]
    if do in ("call", "solve"):
        nbytes, flops = _solve_work(case)
        if do == "call":  # the blocks and vectors cross PCIe as well
            nodes = (case["ni"] + 3) * (case["nj"] + 3) * case["nz"]
            nbytes += nodes * 8 * (4 * (27 if _is3d(case) else 9) + 6)
        return {"bytes": nbytes, "flops": flops}
    if do in ("batch", "serve"):
        each = [_solve_work(m) for m in (_members(case) if do == "batch" else _requests(case))]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    # the blocks written, checked and multiplied once; each element's 8 points of 64 entries in 5 sums
    nodes = (case["ni"] + 3) * (case["nj"] + 3) * case["nz"]
    return {"bytes": nodes * (3 * 4 * 27 * 8 + 100), "flops": nodes * (8 * 64 * 5 * 3 + 216)}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits, by torch
# ---------------------------------------------------------------------------------------------
def _planes(case, A):
    """Coefficient planes (4, couplings, NY, NX[, nz]) and the offsets of the couplings."""
    if _is3d(case):
        return A.permute(0, 4, 1, 2, 3).contiguous(), [(c // 3 % 3, c % 3, c // 9) for c in range(27)]
    return A, [(c // 3, c % 3) for c in range(9)]


def _product(P, offsets, x):
    """A x; x (2, NY, NX[, nz])."""
    p = torch.zeros((2, *(n + 2 for n in x.shape[1:])), dtype=F64, device=DEV)
    p[(slice(None), *(slice(1, -1),) * (x.ndim - 1))] = x
    y = torch.zeros_like(x)
    for c, off in enumerate(offsets):
        q = p[(slice(None), *(slice(o, o + n) for o, n in zip(off, x.shape[1:])))]
        y[0].addcmul_(P[0, c], q[0]).addcmul_(P[1, c], q[1])
        y[1].addcmul_(P[2, c], q[0]).addcmul_(P[3, c], q[1])
    return y


def _column_factors(case, P):
    """The Thomas factors of every column's tridiagonal (3D): levels first."""
    lo, di, up = (torch.stack([P[0, c], P[3, c]]).movedim(-1, 0) for c in (4, 13, 22))
    di = torch.where(di == 0, 1.0, di)
    inv, gam = [1.0 / di[0]], []
    for k in range(1, case["nz"]):
        gam.append(up[k - 1] * inv[k - 1])
        inv.append(1.0 / (di[k] - lo[k] * gam[-1]))
    return lo, inv, gam


def _columns(f, r):
    lo, inv, gam = f
    y = [r[..., 0] * inv[0]]
    for k in range(1, r.shape[-1]):
        y.append((r[..., k] - lo[k] * y[-1]) * inv[k])
    for k in range(r.shape[-1] - 2, -1, -1):
        y[k] = y[k] - gam[k] * y[k + 1]
    return torch.stack(y, -1)


def _solution(case, seed):
    """x of A x = b, to a relative residual of 1e-13 or as near as 64 bits go."""
    A, bu, bv, _ = _system(case, seed)
    P, offsets = _planes(case, A)
    b = torch.stack([bu, bv])
    if _is3d(case):
        f = _column_factors(case, P)
        precond = lambda r: _columns(f, r)  # noqa: E731
    else:
        d = torch.stack([P[0, 4], P[3, 4]])
        inv = torch.where(d != 0, 1.0 / d, 0.0)
        precond = lambda r: r * inv  # noqa: E731
    x = torch.zeros_like(b)
    r, z = b.clone(), precond(b)
    d, rz, norm = z.clone(), (b * z).sum(), float(b.norm())
    for it in range(1, 12000):
        q = _product(P, offsets, d)
        alpha = rz / (d * q).sum()
        x += alpha * d
        r -= alpha * q
        if it % 50 == 0 and float(r.norm()) < 1e-13 * norm:
            break
        z = precond(r)
        new = (r * z).sum()
        d = z + (new / rz) * d
        rz = new
    return x[0].cpu().numpy(), x[1].cpu().numpy()


def exact(case, seed):
    do = case["do"]
    if do in ("call", "solve"):
        if _iterations(case) > 4000:
            return None  # minutes in plain torch
        if case["precond"] == LINES and case["algorithm"] != "mixed":
            return None  # the line solves leave values at ice-free vertices that the system does not determine
        xu, xv = _solution(case, seed)
        out = {"xu": xu, "xv": xv}
        if do == "call" or case["algorithm"] != "mixed":
            out["niters"] = None
        return out
    if do == "batch":
        return {"x": [_solution(m, seed + 1000 * k) if max(m["ni"], m["nj"]) <= 150 else (None, None)
                      for k, m in enumerate(_members(case))]}
    if do == "serve":
        return {"x": [_solution(r, seed + 1000 * k) for k, r in enumerate(_requests(case))]}
    _, u, v, g = _picard_inputs(case, seed)
    nz = case["nz"]
    A, efvs = _blocks_3d(g, nz, (u, v))
    drag = _drag(g)
    A[0, ..., nz - 1, 13] += drag
    A[3, ..., nz - 1, 13] += drag
    _lower_from_upper(A)
    y = _product(*_planes(case, A), torch.stack([u, v])) - torch.stack(_loads(g, nz))
    y = torch.where(g["vertex"][..., None], y, 0.0)
    return {"efvs": efvs.cpu().numpy(), "resid_u": y[0].cpu().numpy(), "resid_v": y[1].cpu().numpy(),
            "norm": float(y.norm())}

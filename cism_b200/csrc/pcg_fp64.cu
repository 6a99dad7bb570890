// pcg_fp64.cu -- plain FP64 structured PCG on B200 (sm_100a), reference-faithful.
//
// Each kernel restates one or more consecutive whole-array statements of
// libglissade/glissade_velo_higher_pcg.F90 with the same floating-point operation
// order (the library is compiled with --fmad=false, so a*b+c is never contracted),
// and global sums go through the fixed double-double tree of common.cuh.  The
// kernels never read the CPU; scalars (alpha, beta, ...) live in SolveState in HBM
// and are produced by the last CTA of the reducing kernel.
#include "common.cuh"
#include "../../include/cismgpu.h"

namespace cismgpu {

// ---------------------------------------------------------------------------
// launches of an iteration
// ---------------------------------------------------------------------------
// The kernels of an FP64 iteration depend on each other and many last a few microseconds, so the
// gap between them counts.  They are launched with programmatic dependence: a kernel's blocks are
// set up while the one before still runs, and wait here for its end (and so for everything before
// it) before they read anything.  Every kernel launched by launch_dep starts with after_previous.
// A product of the 31x31x11 dome behind another one: 6.2 -> 4.8 us, SSA 401x401 8.2 -> 6.2.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
inline void launch_dep(void (*k)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, A... a) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, P(a)...);
}

// ---------------------------------------------------------------------------
// reduction: per-CTA dd partials -> last CTA finishes with the fixed tree and
// runs the scalar epilogue
// ---------------------------------------------------------------------------
struct RedCtx {
    DD *partials;        // [gridDim.x][2]
    SolveState *st;
    int epi;
    int iter;
};

__device__ void epilogue(SolveState *st, int epi, int iter, double S0, double S1) {
    switch (epi) {
    case EPI_L2RHS:
        st->L2_rhs = sqrt(S0);
        break;
    case EPI_STD_ETA1: {  // :1325-1337
        st->eta1 = S0;
        if (S0 != S0) { st->status = CISMGPU_EBREAKDOWN_ETA1; st->done = 1; st->niters = iter; break; }
        st->beta = st->eta1 / st->eta0;
        break;
    }
    case EPI_STD_ETA2: {  // :1371-1394
        st->eta0 = st->eta1;
        st->eta2 = S0;
        st->alpha = st->eta1 / st->eta2;
        if (st->alpha != st->alpha) { st->status = CISMGPU_EBREAKDOWN_ALPHA; st->done = 1; st->niters = iter; }
        break;
    }
    case EPI_CHECK: {     // :1466-1513, :3516-3563
        st->err = sqrt(S0) / st->L2_rhs;
        st->checks += 1;
        if (st->err < st->tol) { st->niters = iter; st->done = 1; }
        break;
    }
    case EPI_CG_RHO0:     // (r,z) of the first pass, kept until (d,q) is known (:3215, :3258)
        st->rho_old = S0;
        break;
    case EPI_CG_FIRST: {  // :3258-3266
        st->sigma = S0;
        st->alpha = st->rho_old / st->sigma;
        if (st->alpha != st->alpha) { st->status = CISMGPU_EBREAKDOWN_ALPHA; st->done = 1; st->niters = iter; }
        break;
    }
    case EPI_CG_ITER: {   // :3426-3437
        st->rho = S0;
        st->delta = S1;
        st->beta = st->rho / st->rho_old;
        st->sigma = st->delta - st->beta * st->rho / st->alpha;
        st->alpha = st->rho / st->sigma;
        st->rho_old = st->rho;
        if (st->alpha != st->alpha) { st->status = CISMGPU_EBREAKDOWN_ALPHA; st->done = 1; st->niters = iter; }
        break;
    }
    case EPI_RESID_VEC:   // glissade_velo_higher.F90:9858-9859, :9883-9884
        st->err = sqrt(S0);
        st->L2_rhs = sqrt(S1);
        break;
    case EPI_SUM:
        st->rho = S0;
        break;
    default:
        break;
    }
}

// The fixed tree over the values of a block's first 256 threads (a block of any size; the other
// threads pass through the barriers): shuffle-down over the 32 lanes, then over the 8 warp sums.
// Result in thread 0.  The NF trees run side by side: each is a chain of dependent additions, and
// one after the other they would cost twice the latency.
template <int NF>
__device__ __forceinline__ void block_tree_first(DD &v0, DD &v1, DD (*sm)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < kBlock / 32) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const DD o0 = dd_shfl_down(v0, off), o1 = (NF > 1) ? dd_shfl_down(v1, off) : DD{0.0, 0.0};
            if (lane + off < 32) {
                v0 = dd_add(v0, o0);
                if (NF > 1) v1 = dd_add(v1, o1);
            }
        }
    }
    __syncthreads();  // protect 'sm' reuse across consecutive calls
    if (warp < kBlock / 32 && lane == 0) {
        sm[0][warp] = v0;
        if (NF > 1) sm[1][warp] = v1;
    }
    __syncthreads();
    if (warp == 0) {
        v0 = (lane < 8) ? sm[0][lane] : DD{0.0, 0.0};
        if (NF > 1) v1 = (lane < 8) ? sm[1][lane] : DD{0.0, 0.0};
#pragma unroll
        for (int off = 4; off >= 1; off >>= 1) {
            const DD o0 = dd_shfl_down(v0, off), o1 = (NF > 1) ? dd_shfl_down(v1, off) : DD{0.0, 0.0};
            if (lane + off < 32) {
                v0 = dd_add(v0, o0);
                if (NF > 1) v1 = dd_add(v1, o1);
            }
        }
    }
}

// Called by all threads of every CTA; the first kBlock threads hold their columns' sums.
template <int NF>
__device__ void reduce_and_finish(const RedCtx &rc, DD v0, DD v1) {
    __shared__ DD sm[NF][8];
    __shared__ bool last;
    block_tree_first<NF>(v0, v1, sm);
    if (threadIdx.x == 0) {
        rc.partials[2 * blockIdx.x + 0] = v0;
        rc.partials[2 * blockIdx.x + 1] = v1;
        __threadfence();
        unsigned int t = atomicAdd(&rc.st->ticket[0], 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    DD a0{0.0, 0.0}, a1{0.0, 0.0};
    if (threadIdx.x < kBlock)
        for (unsigned int c = threadIdx.x; c < gridDim.x; c += kBlock) {
            DD p0, p1;
            p0.hi = __ldcg(&rc.partials[2 * c].hi);
            p0.lo = __ldcg(&rc.partials[2 * c].lo);
            if (NF > 1) {
                p1.hi = __ldcg(&rc.partials[2 * c + 1].hi);
                p1.lo = __ldcg(&rc.partials[2 * c + 1].lo);
            }
            a0 = dd_add(a0, p0);
            if (NF > 1) a1 = dd_add(a1, p1);
        }
    block_tree_first<NF>(a0, a1, sm);
    if (threadIdx.x == 0) {
        rc.st->ticket[0] = 0u;
        epilogue(rc.st, rc.epi, rc.iter, a0.hi + a0.lo, a1.hi + a1.lo);
    }
}

__device__ __forceinline__ void col_of(const Geom &g, long long q, int &i, int &j) {
    j = (int)(q / g.NX);
    i = (int)(q - (long long)j * g.NX);
}

// ---------------------------------------------------------------------------
// structured matvec row (matvec_multiply_structured_3d :5612-5650, _2d :5739-5771)
// ---------------------------------------------------------------------------
// The matrix as a matvec reads it.
//   MV_BOUNDS: the coefficient planes, every coupling tested against the array (any geometry);
//   MV_INNER: the same planes, no owned vertex on the edge of the array, so that only the levels
//     are tested, which is uniform over a block: all loads of a row are issued without branches;
//   MV_HALF: MV_INNER of an exactly symmetric 3D matrix (as the reference's check leaves it): its
//     symmetric half of k_half3d, one 32-byte load per coupling and node.  A lower coupling c is
//     its partner's coupling 26 - c with uv and vu swapped, the same number, so the sums are too.
// 3D product on 201x201x11: 72.7 us with tests, 59.7 without, 37.0 from the half (5.6 TB/s; it
// streams 448 bytes a node instead of 864, and the partners' couplings come from L2).
enum MvLayout { MV_BOUNDS = 0, MV_INNER, MV_HALF };

struct MvMatrix {
    const double *A;   // [4][NC][nz][NQ]
    const double *H;   // MV_HALF: [14][nz][NQ][4], couplings 13..26 as (uu, uv, vu, vv)
    int layout;
};

struct __align__(32) Dbl4 { double x, y, z, w; };
__device__ __forceinline__ Dbl4 ldg256(const double *p) {  // 32-byte aligned, read-only in the launch
    Dbl4 v;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

template <int NC, int LAY>
__device__ __forceinline__ void mv_row(const Geom &g, const MvMatrix &M, const double *__restrict__ xu,
                                       const double *__restrict__ xv, int i, int j, long long q, int k,
                                       double &yu, double &yv) {
    const long long plane = (long long)g.nz * g.NQ, e = (long long)k * g.NQ + q;
    const double *__restrict__ Auu = M.A, *__restrict__ Auv = M.A + NC * plane, *__restrict__ Avu = M.A + 2 * NC * plane,
                              *__restrict__ Avv = M.A + 3 * NC * plane;
    constexpr int K0 = (NC == 27) ? -1 : 0, K1 = (NC == 27) ? 1 : 0;
    double su = 0.0, sv = 0.0;
#pragma unroll
    for (int kA = K0; kA <= K1; ++kA) {
        if (k + kA < 0 || k + kA >= g.nz) continue;
#pragma unroll
        for (int c9 = 0; c9 < 9; ++c9) {
            const int iA = c9 % 3 - 1, jA = c9 / 3 - 1, c = (kA - K0) * 9 + c9;
            if (LAY == MV_BOUNDS && (i + iA < 0 || i + iA >= g.NX || j + jA < 0 || j + jA >= g.NY)) continue;
            const long long n = e + (long long)kA * g.NQ + (long long)jA * g.NX + iA;
            const double x1 = xu[n], x2 = xv[n];
            Dbl4 a;
            if (LAY == MV_HALF) {
                if (c >= 13) {
                    a = ldg256(M.H + 4 * ((c - 13) * plane + e));
                } else {
                    const Dbl4 p = ldg256(M.H + 4 * ((13 - c) * plane + n));
                    a = Dbl4{p.x, p.z, p.y, p.w};
                }
            } else {
                const long long f = c * plane + e;
                a = Dbl4{__ldg(Auu + f), __ldg(Auv + f), __ldg(Avu + f), __ldg(Avv + f)};
            }
            su = __dadd_rn(__dadd_rn(su, __dmul_rn(a.x, x1)), __dmul_rn(a.y, x2));
            sv = __dadd_rn(__dadd_rn(sv, __dmul_rn(a.z, x1)), __dmul_rn(a.w, x2));
        }
    }
    yu = su;
    yv = sv;
}

// The symmetric half of a 3D matrix, [14][nz][NQ][4]: couplings c = 13..26 (the diagonal and the
// upper offsets) of every node as (uu, uv, vu, vv), couplings leaving the array as zero.  *flag is
// set if a lower coupling of an owned active row differs from its transpose partner (Auu with
// Auu, Auv with Avu, Avv with Avv, bit for bit), which check_symmetry_assembled_matrix_3d averages
// to equality before every 3D solve (glissade_velo_higher.F90:2923-2931).  No owned vertex may lie
// on the edge of the array (a partner is then always inside).  a32 (may be null): the same half
// as FP32.  One thread per node and stored coupling; every plane is read once, coalesced (201x201x11: 98 us
// for the test and the FP64 half).  Once a difference is known the copy is of no use, and the blocks
// that have not started yet end at once; a block may still read an old flag, and then does its part in vain.
__global__ void __launch_bounds__(kBlock) k_half3d(Geom g, const int32_t *__restrict__ act, const double *__restrict__ A,
                                                   double *__restrict__ H, float4 *__restrict__ a32, int *flag) {
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    const int k = blockIdx.y, h = blockIdx.z, c = 13 + h;
    if (*flag != 0) return;
    bool bad = false;
    if (q < g.NQ) {
        const int i = (int)(q % g.NX), j = (int)(q / g.NX);
        const int iA = c % 3 - 1, jA = (c / 3) % 3 - 1, kA = c / 9 - 1;
        const int in = i + iA, jn = j + jA;
        const bool inside = in >= 0 && in < g.NX && jn >= 0 && jn < g.NY && k + kA < g.nz;
        const long long plane = (long long)g.nz * g.NQ, bs = 27 * plane, e = (long long)k * g.NQ + q, f = c * plane + e;
        Dbl4 a{0.0, 0.0, 0.0, 0.0};
        if (inside) {
            a = Dbl4{A[f], A[bs + f], A[2 * bs + f], A[3 * bs + f]};
            const long long qn = (long long)jn * g.NX + in;
            if (h > 0 && owned(g, in, jn) && act[qn] != 0) {
                const long long l = (26 - c) * plane + (long long)(k + kA) * g.NQ + qn;
                bad = A[l] != a.x || A[bs + l] != a.z || A[2 * bs + l] != a.y || A[3 * bs + l] != a.w;
            }
        }
        reinterpret_cast<Dbl4 *>(H)[h * plane + e] = a;
        if (a32) a32[h * plane + e] = make_float4((float)a.x, (float)a.y, (float)a.z, (float)a.w);
    }
    if (bad) *flag = 1;
}

enum MvMode { MV_PLAIN = 0, MV_RESID, MV_DQ, MV_CG_AZ };

constexpr int kDotChunk = 8;  // levels whose loads a column's dot terms issue together

// y = A x over owned active columns, 0 elsewhere; optional fused statements:
//   MV_RESID : r = b - y (whole array); S0 = (r,r)             [:1454-1466, :3504-3516]
//   MV_DQ    : S0 = (x,y) with x = d, y = q                    [:1376-1381, :3241-3248]
//   MV_CG_AZ : S0 = (r,z), S1 = (y,z) with x = z, y = Az       [:3401-3413]
// One thread per node (column q, level k = blockIdx.y): a launch has nz * NQ/256 CTAs and enough
// loads in flight to stream the coefficients.  Dot products in 3D: every node writes its
// term(s) to T ([2][nz][NQ]); the last level block of each column block to finish has one thread
// per column add them over k in level order, then the block tree of the 256 columns and the
// last-CTA tree: the order the reduction has always had, without a launch of its own, and with the
// sums of the early column blocks overlapping the rest of the matvec.  The per-column-block
// counters sit after the partials and return to zero here.  In 2D a column has one level, so
// every block reduces its own terms.
// 2D: five blocks an SM (48 registers).  Microseconds an iteration with 3, 4, 5 and 6: 201x201 16.4, 16.1,
// 17.5, 18.0; 301x301 19.3, 20.0, 19.2, 20.8; 401x401 25.7, 25.8, 23.0, 23.5; 601x601 56.4, 53.8, 50.2, 52.0;
// 801x801 90.2, 86.4, 85.2, 85.1; equal up to 121x121.
template <int NC, int MODE, int LAY>
__global__ void __launch_bounds__(kBlock, NC == 9 ? 5 : 3) k_mv_nodes(Geom g, MvMatrix M, const int32_t *__restrict__ act,
                                                        const double *__restrict__ xu, const double *__restrict__ xv,
                                                        double *__restrict__ yu, double *__restrict__ yv,
                                                        const double *__restrict__ bu, const double *__restrict__ bv,
                                                        double *__restrict__ ru, double *__restrict__ rv,
                                                        double *__restrict__ T, RedCtx rc) {
    constexpr int NF = (MODE == MV_CG_AZ) ? 2 : 1;
    after_previous();
    if (rc.st && rc.st->done) return;
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    const int k = blockIdx.y;
    const long long plane = (long long)g.nz * g.NQ;
    bool own = false;
    double t0 = 0.0, t1 = 0.0;
    if (q < g.NQ) {
        int i, j;
        col_of(g, q, i, j);
        own = owned(g, i, j);
        const long long e = (long long)k * g.NQ + q;
        double a = 0.0, b = 0.0;
        if (own && act[q] != 0) mv_row<NC, LAY>(g, M, xu, xv, i, j, q, k, a, b);
        yu[e] = a;
        yv[e] = b;
        if (MODE == MV_RESID) {
            const double r1 = __dsub_rn(bu[e], a), r2 = __dsub_rn(bv[e], b);
            ru[e] = r1;
            rv[e] = r2;
            t0 = __dadd_rn(__dmul_rn(r1, r1), __dmul_rn(r2, r2));
        } else if (MODE == MV_DQ && own) {
            t0 = __dadd_rn(__dmul_rn(xu[e], a), __dmul_rn(xv[e], b));
        } else if (MODE == MV_CG_AZ && own) {
            const double z1 = xu[e], z2 = xv[e];
            t0 = __dadd_rn(__dmul_rn(ru[e], z1), __dmul_rn(rv[e], z2));
            t1 = __dadd_rn(__dmul_rn(a, z1), __dmul_rn(b, z2));
        }
        if (NC == 27 && MODE != MV_PLAIN && own) {
            T[e] = t0;
            if (NF > 1) T[plane + e] = t1;
        }
    }
    if (MODE == MV_PLAIN) return;
    DD s0{0.0, 0.0}, s1{0.0, 0.0};
    if (NC == 9) {
        if (own) {
            s0 = dd_add_d(s0, t0);
            if (NF > 1) s1 = dd_add_d(s1, t1);
        }
    } else {
        __shared__ bool lastk;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned *cnt = reinterpret_cast<unsigned *>(rc.partials + 2 * gridDim.x) + blockIdx.x;
            __threadfence();  // this block's terms before its count
            const unsigned t = atomicAdd(cnt, 1u);
            lastk = t == gridDim.y - 1;
            if (lastk) *cnt = 0u;
        }
        __syncthreads();
        if (!lastk) return;
        __threadfence();
        if (own)
            for (int k0 = 0; k0 < g.nz; k0 += kDotChunk) {  // through L2: other CTAs of the launch wrote them
                double v0[kDotChunk], v1[kDotChunk];
#pragma unroll
                for (int u = 0; u < kDotChunk; ++u) {
                    const long long e = (long long)(k0 + u) * g.NQ + q;
                    v0[u] = (k0 + u < g.nz) ? __ldcg(T + e) : 0.0;
                    v1[u] = (NF > 1 && k0 + u < g.nz) ? __ldcg(T + plane + e) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kDotChunk; ++u)
                    if (k0 + u < g.nz) {
                        s0 = dd_add_d(s0, v0[u]);
                        if (NF > 1) s1 = dd_add_d(s1, v1[u]);
                    }
            }
    }
    reduce_and_finish<NF>(rc, s0, s1);
}

// y = A x (+ the statement MODE fuses with it, see MvMode) on stream s.  T: the dot terms ([2][nz][NQ]).
template <int NC, int MODE>
inline void launch_mv(cudaStream_t s, const Geom &g, const MvMatrix &M, const int32_t *act, const double *xu,
                      const double *xv, double *yu, double *yv, const double *bu, const double *bv, double *ru,
                      double *rv, double *T, const RedCtx &rc) {
    const dim3 grid((unsigned)((g.NQ + kBlock - 1) / kBlock), (unsigned)g.nz);
    if (NC == 27 && M.layout == MV_HALF)
        launch_dep(k_mv_nodes<27, MODE, MV_HALF>, grid, kBlock, 0, s, g, M, act, xu, xv, yu, yv, bu, bv, ru, rv, T, rc);
    else if (M.layout == MV_INNER)
        launch_dep(k_mv_nodes<NC, MODE, MV_INNER>, grid, kBlock, 0, s, g, M, act, xu, xv, yu, yv, bu, bv, ru, rv, T, rc);
    else
        launch_dep(k_mv_nodes<NC, MODE, MV_BOUNDS>, grid, kBlock, 0, s, g, M, act, xu, xv, yu, yv, bu, bv, ru, rv, T, rc);
}

// ---------------------------------------------------------------------------
// vector statements and preconditioners over the whole array (halo included)
// ---------------------------------------------------------------------------
// The statements between two matvecs are pointwise in a node or in a column, so they share
// launches: an iteration is bound by HBM/L2 traffic on large grids and by its launches and memory
// round trips on small ones.  The staggered halo (k_halo) of the vectors they read or write is
// taken at the same time: a halo position reads its source (halo_src), or the source's thread
// writes its images (put_haloed).  Both give the values the reference's separate update leaves.
// With one launch per statement group and one thread per column walking its levels, an iteration
// of the 201x201x11 ice stream spent 90 us of 190 here.  Joining them took its solve from 5.42 to 3.88 ms
// (SIA), the 31x31x11 dome from 2.16 to 1.08 and SSA 401x401 (diagonal) from 161 to 113; with the half,
// the dependent launches and the 2D product's blocks these are 2.58, 0.78 and 84 ms.

// Positions of the staggered halo that hold zero (outflow, no_ice).
__device__ __forceinline__ bool zero_pos(const Geom &g, int i, int j) {
    if (g.outflow) return i == 0 || i == g.NX - 1 || j == 0 || j == g.NY - 1;
    if (g.no_ice) return i <= 1 || i >= g.NX - 2 || j <= 1 || j >= g.NY - 2;
    return false;
}

// Source coordinate of a periodic halo coordinate (identity elsewhere).
__device__ __forceinline__ int pmap(int i, int N) {
    if (i == 0) return N - 3;
    if (i == 1) return N - 2;
    if (i == N - 1) return 2;
    return i;
}

__device__ __forceinline__ bool periodic_halo(const Geom &g, int i, int j) {
    return g.periodic && (i <= 1 || i == g.NX - 1 || j <= 1 || j == g.NY - 1);
}

// Column whose value (i, j) holds after the staggered halo update; -1: it holds zero.
__device__ __forceinline__ long long halo_src(const Geom &g, int i, int j, long long q) {
    if (zero_pos(g, i, j)) return -1;
    if (periodic_halo(g, i, j)) return (long long)pmap(j, g.NY) * g.NX + pmap(i, g.NX);
    return q;
}

// The staggered halo update writes owned positions (no_ice: the last owned row and column in the
// reference's geometry).
inline bool halo_reaches_owned(const Geom &g) {
    auto in = [&](int lo, int hi, int N) {
        if (g.outflow ? (lo <= 0 || hi >= N - 1) : (g.no_ice && (lo <= 1 || hi >= N - 2))) return true;
        return g.periodic && (lo <= 1 || hi >= N - 1);
    };
    return in(g.ilo, g.ihi, g.NX) || in(g.jlo, g.jhi, g.NY);
}

// a(i, j) = v followed by the staggered halo update of a, by the thread of (i, j) alone: a zero
// position stores zero, a periodic halo position nothing, any other its value and its images.
__device__ __forceinline__ void put_haloed(const Geom &g, int i, int j, double *__restrict__ a, double v) {
    const int NX = g.NX, NY = g.NY;
    const long long q = (long long)j * NX + i;
    if (zero_pos(g, i, j)) {
        a[q] = 0.0;
        return;
    }
    if (!g.periodic) {
        a[q] = v;
        return;
    }
    if (periodic_halo(g, i, j)) return;
    a[q] = v;
    if (i != 2 && i < NX - 3 && j != 2 && j < NY - 3) return;  // no images
    for (int b = 0; b < 4; ++b) {
        const int jj = (b == 0) ? j : (b == 1 ? 0 : (b == 2 ? 1 : NY - 1));
        if (b > 0 && pmap(jj, NY) != j) continue;
        for (int c = 0; c < 4; ++c) {
            const int ii = (c == 0) ? i : (c == 1 ? 0 : (c == 2 ? 1 : NX - 1));
            if (c > 0 && pmap(ii, NX) != i) continue;
            if ((b > 0 || c > 0) && !zero_pos(g, ii, jj)) a[(long long)jj * NX + ii] = v;
        }
    }
}

// The statements before the preconditioner (or alone).
enum Upd {
    U_NONE = 0,
    U_RHALO,      // halo of r                                            [:1478-1480, :3118-3121]
    U_XR,         // x = x + alpha*d; r = r - alpha*q                     [:1399-1403]
    U_XR_X,       // U_XR, then the halo of x                             [:1399-1403, :1440-1450]
    U_XR_Q,       // the halo of q, then U_XR                             [:3268-3276]
    U_CG,         // the halo of Az, then d = z + beta*d; q = Az + beta*q; x += alpha*d; r -= alpha*q [:3444-3459]
    U_DIR,        // d = z + beta*d, then the halo of d                   [:1340-1350]
    U_STD_INIT,   // r = b - z; d = 0; z = 0                              [:1190-1206]
    U_CG_INIT,    // r = b - z                                            [:3115-3116]
};

// What follows in the same thread: nothing, z = r, or z = r / diagonal.  The column solves are
// in k_col.
enum Pre { P_KEEP = 0, P_NONE, P_DIAG, P_SIA };

struct VecArgs {
    const double *bu, *bv;
    double *xu, *xv, *ru, *rv, *du, *dv, *qu, *qv, *zu, *zv;
    const double *Azu, *Azv;
};

// One thread per node (column, level = blockIdx.y): every load of a statement group is issued at
// once and nz * NQ/256 CTAs stream the planes (a thread per column took one round trip per level:
// the update alone 41 us on 201x201x11, 1.9 TB/s).
template <int UPD, int PRE>
__global__ void __launch_bounds__(kBlock) k_node(Geom g, VecArgs v, const SolveState *st,
                                                 const double *__restrict__ dgu, const double *__restrict__ dgv) {
    after_previous();
    if (st->done) return;
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    if (q >= g.NQ) return;
    const double alpha = st->alpha, beta = st->beta;
    const long long kq = (long long)blockIdx.y * g.NQ, e = kq + q;
    int i, j;
    col_of(g, q, i, j);
    double r1 = 0.0, r2 = 0.0;
    if (UPD == U_STD_INIT) {
        r1 = __dsub_rn(v.bu[e], v.zu[e]);
        r2 = __dsub_rn(v.bv[e], v.zv[e]);
        v.ru[e] = r1; v.rv[e] = r2;
        v.du[e] = 0.0; v.dv[e] = 0.0;
        v.zu[e] = 0.0; v.zv[e] = 0.0;
        return;
    }
    if (UPD == U_CG_INIT) {
        v.ru[e] = __dsub_rn(v.bu[e], v.zu[e]);
        v.rv[e] = __dsub_rn(v.bv[e], v.zv[e]);
        return;
    }
    if (UPD == U_DIR) {
        put_haloed(g, i, j, v.du + kq, __dadd_rn(v.zu[e], __dmul_rn(beta, v.du[e])));
        put_haloed(g, i, j, v.dv + kq, __dadd_rn(v.zv[e], __dmul_rn(beta, v.dv[e])));
        return;
    }
    const double a1 = (PRE == P_DIAG) ? dgu[e] : 1.0, a2 = (PRE == P_DIAG) ? dgv[e] : 1.0;
    const long long s = (UPD == U_RHALO || UPD == U_XR_Q || UPD == U_CG) ? halo_src(g, i, j, q) : q;
    if (UPD == U_NONE) {
        r1 = v.ru[e];
        r2 = v.rv[e];
    } else if (UPD == U_RHALO) {
        r1 = s >= 0 ? v.ru[kq + s] : 0.0;
        r2 = s >= 0 ? v.rv[kq + s] : 0.0;
        if (s != q) { v.ru[e] = r1; v.rv[e] = r2; }
    } else if (UPD == U_CG) {
        const double d1 = __dadd_rn(v.zu[e], __dmul_rn(beta, v.du[e]));
        const double d2 = __dadd_rn(v.zv[e], __dmul_rn(beta, v.dv[e]));
        const double q1 = __dadd_rn(s >= 0 ? v.Azu[kq + s] : 0.0, __dmul_rn(beta, v.qu[e]));
        const double q2 = __dadd_rn(s >= 0 ? v.Azv[kq + s] : 0.0, __dmul_rn(beta, v.qv[e]));
        const double x1 = __dadd_rn(v.xu[e], __dmul_rn(alpha, d1));
        const double x2 = __dadd_rn(v.xv[e], __dmul_rn(alpha, d2));
        r1 = __dsub_rn(v.ru[e], __dmul_rn(alpha, q1));
        r2 = __dsub_rn(v.rv[e], __dmul_rn(alpha, q2));
        v.du[e] = d1; v.dv[e] = d2;
        v.qu[e] = q1; v.qv[e] = q2;
        v.xu[e] = x1; v.xv[e] = x2;
        v.ru[e] = r1; v.rv[e] = r2;
    } else {  // U_XR, U_XR_X, U_XR_Q
        const double q1 = s >= 0 ? v.qu[kq + s] : 0.0, q2 = s >= 0 ? v.qv[kq + s] : 0.0;
        const double x1 = __dadd_rn(v.xu[e], __dmul_rn(alpha, v.du[e]));
        const double x2 = __dadd_rn(v.xv[e], __dmul_rn(alpha, v.dv[e]));
        r1 = __dsub_rn(v.ru[e], __dmul_rn(alpha, q1));
        r2 = __dsub_rn(v.rv[e], __dmul_rn(alpha, q2));
        if (UPD == U_XR_Q && s != q) { v.qu[e] = q1; v.qv[e] = q2; }
        if (UPD == U_XR_X) {
            put_haloed(g, i, j, v.xu + kq, x1);
            put_haloed(g, i, j, v.xv + kq, x2);
        } else {
            v.xu[e] = x1; v.xv[e] = x2;
        }
        v.ru[e] = r1; v.rv[e] = r2;
    }
    if (PRE == P_NONE) {
        v.zu[e] = r1; v.zv[e] = r2;
    } else if (PRE == P_DIAG) {  // :1238-1253 (3D), :467-480 (2D)
        v.zu[e] = (a1 != 0.0) ? r1 / a1 : 0.0;
        v.zv[e] = (a2 != 0.0) ? r2 / a2 : 0.0;
    }
}

constexpr int kMaxNz = 64;

// The pivots of tridiag_solver (:5870-5922) on the columns of the SIA matrix (easy_sia_solver
// :5777-5866): beta_k and gamma_k = spdiag_{k-1} / beta_{k-1} depend on the matrix alone, so a
// solve takes them once, with the operations of the reference's recurrence, and its column solves
// keep one division per level instead of two.  fac: [u, v][beta, gamma][nz][NQ]; one thread per
// active column and component, loads of kColChunk levels at a time.
constexpr int kColChunk = 4;
__global__ void k_sia_factor(Geom g, const double *__restrict__ A, const int32_t *__restrict__ act,
                             double *__restrict__ fac) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.NQ || act[q] == 0) return;
    const int nz = g.nz;
    const long long NQ = g.NQ, plane = (long long)nz * NQ;
    const double *B = A + (blockIdx.y ? 3LL : 0LL) * 27 * plane;
    const double *Mlo = B + 4 * plane, *Mdi = B + 13 * plane, *Mup = B + 22 * plane;
    double *fb = fac + (blockIdx.y ? 2 : 0) * plane, *fg = fb + plane;
    double beta = Mdi[q];
    fb[q] = beta;
    fg[q] = 0.0;
    for (int k0 = 1; k0 < nz; k0 += 8) {
        double sp[8], sb[8], dg[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long e = (long long)(k0 + u) * NQ + q;
            const bool in = k0 + u < nz;
            sp[u] = in ? Mup[e - NQ] : 0.0;
            sb[u] = in ? Mlo[e] : 0.0;
            dg[u] = in ? Mdi[e] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (k0 + u < nz) {
                const long long e = (long long)(k0 + u) * NQ + q;
                const double gam = sp[u] / beta;
                beta = __dsub_rn(dg[u], __dmul_rn(sb[u], gam));
                fb[e] = beta;
                fg[e] = gam;
            }
    }
}

struct ColArgs {
    int upd;                    // Upd: U_NONE, U_RHALO, U_XR or U_CG
    int setd;                   // d = z (first pass of Chronopoulos-Gear, :3215-3223)
    const double *lo[2];        // P_SIA: the sub-diagonal planes of u and v
    const double *fac;          // P_SIA: k_sia_factor
    const double *dg[2];        // P_DIAG: the diagonal planes
    const double *zs;           // line preconditioners (3D): [2][NQ] line solution, added on every level
    const int32_t *act;
};

// One thread per (column, component): a block holds CW columns' u components, then their v
// components.  UPD as k_node, then the preconditioner: P_SIA, the column solves of
// tridiag_solver (:5870-5922) (+ the line solution, tridiag_solver_{local,global}_3d :4617-4655 /
// :4876-4911), or with DOT also P_NONE, P_DIAG and P_KEEP.  Loads of kColChunk levels are issued
// together; NZM > 0: a column of up to NZM levels stays in registers between the two sweeps, else
// it goes through z.  DOT: S0 = (r,z) over the owned columns, per column in level order
// (:1320-1326): the v threads hand their products to the u threads through shared memory.
// Bound by HBM on large grids (224 bytes a node with U_CG); 64-column blocks without DOT, so that
// 84k threads of a 201x201 grid spread over all SMs (256 are the reduction's chunk with DOT).
template <int PRE, bool DOT, int NZM>
__global__ void __launch_bounds__(DOT ? 2 * kBlock : 128) k_col(Geom g, VecArgs v, ColArgs c, RedCtx rc) {
    after_previous();
    if (rc.st->done) return;
    constexpr int CW = DOT ? kBlock : 64;
    constexpr int C = kColChunk;
    __shared__ double sprod[DOT ? C : 1][DOT ? kBlock : 1];
    const int comp = threadIdx.x >= CW ? 1 : 0, cl = threadIdx.x - comp * CW;
    const long long q = (long long)blockIdx.x * CW + cl;
    const int nz = g.nz;
    const long long NQ = g.NQ, plane = (long long)nz * NQ;
    const bool in = q < NQ;
    const double alpha = rc.st->alpha, beta = rc.st->beta;
    double *__restrict__ R = comp ? v.rv : v.ru;
    double *__restrict__ Z = comp ? v.zv : v.zu;
    double *__restrict__ D = comp ? v.dv : v.du;
    double *__restrict__ Q = comp ? v.qv : v.qu;
    double *__restrict__ X = comp ? v.xv : v.xu;
    const double *__restrict__ Az = comp ? v.Azv : v.Azu;
    const double *__restrict__ fb = c.fac + (comp ? 2 : 0) * plane, *__restrict__ fg = fb + plane;
    const double *__restrict__ lo = comp ? c.lo[1] : c.lo[0], *__restrict__ dg = comp ? c.dg[1] : c.dg[0];
    bool own = false, solve = false;
    if (in) {
        int i, j;
        col_of(g, q, i, j);
        own = owned(g, i, j);
        solve = (PRE == P_SIA) && c.act[q] != 0;
        const long long s = (c.upd == U_RHALO || c.upd == U_CG) ? halo_src(g, i, j, q) : q;
        double y[NZM > 0 ? NZM : 1];
        double prev = 0.0;
        // r of C levels from k0 (the update's statements included)
        auto chunk = [&](int k0, double (&r)[C]) {
            if (c.upd == U_CG) {
                double dd[C], qq[C], xx[C], zz[C], az[C];
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    const long long e = (long long)(k0 + u) * NQ + q;
                    const bool on = k0 + u < nz;
                    r[u] = on ? R[e] : 0.0;
                    dd[u] = on ? D[e] : 0.0;
                    qq[u] = on ? Q[e] : 0.0;
                    xx[u] = on ? X[e] : 0.0;
                    zz[u] = on ? Z[e] : 0.0;
                    az[u] = (on && s >= 0) ? Az[e - q + s] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    if (k0 + u >= nz) continue;
                    const long long e = (long long)(k0 + u) * NQ + q;
                    const double dn = __dadd_rn(zz[u], __dmul_rn(beta, dd[u]));
                    const double qn = __dadd_rn(az[u], __dmul_rn(beta, qq[u]));
                    r[u] = __dsub_rn(r[u], __dmul_rn(alpha, qn));
                    D[e] = dn;
                    Q[e] = qn;
                    X[e] = __dadd_rn(xx[u], __dmul_rn(alpha, dn));
                    R[e] = r[u];
                }
            } else if (c.upd == U_XR) {
                double dd[C], qq[C], xx[C];
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    const long long e = (long long)(k0 + u) * NQ + q;
                    const bool on = k0 + u < nz;
                    r[u] = on ? R[e] : 0.0;
                    dd[u] = on ? D[e] : 0.0;
                    qq[u] = on ? Q[e] : 0.0;
                    xx[u] = on ? X[e] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    if (k0 + u >= nz) continue;
                    const long long e = (long long)(k0 + u) * NQ + q;
                    r[u] = __dsub_rn(r[u], __dmul_rn(alpha, qq[u]));
                    X[e] = __dadd_rn(xx[u], __dmul_rn(alpha, dd[u]));
                    R[e] = r[u];
                }
            } else {
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    const long long e = (long long)(k0 + u) * NQ + q;
                    r[u] = (k0 + u < nz && s >= 0) ? R[e - q + s] : 0.0;
                }
                if (s != q) {
#pragma unroll
                    for (int u = 0; u < C; ++u)
                        if (k0 + u < nz) R[(long long)(k0 + u) * NQ + q] = r[u];
                }
            }
        };
        // forward sweep: sol_1 = r_1 / beta_1; sol_k = (r_k - sbdiag_k sol_{k-1}) / beta_k
        auto forward = [&](int k0, double *yk) {
            double r[C], sb[C], be[C];
            if (PRE == P_SIA && solve) {
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    const long long e = (long long)(k0 + u) * NQ + q;
                    const bool on = k0 + u < nz;
                    sb[u] = on ? lo[e] : 0.0;
                    be[u] = on ? fb[e] : 1.0;
                }
            } else if (PRE == P_DIAG) {
#pragma unroll
                for (int u = 0; u < C; ++u) be[u] = (k0 + u < nz) ? dg[(long long)(k0 + u) * NQ + q] : 0.0;
            }
            chunk(k0, r);
#pragma unroll
            for (int u = 0; u < C; ++u) {
                if (k0 + u >= nz) continue;
                const long long e = (long long)(k0 + u) * NQ + q;
                if (PRE == P_SIA) {
                    if (!solve) continue;
                    prev = (k0 + u == 0) ? r[u] / be[u] : __dsub_rn(r[u], __dmul_rn(sb[u], prev)) / be[u];
                    if (NZM > 0) yk[u] = prev;
                    else Z[e] = prev;
                } else if (PRE == P_NONE) {
                    Z[e] = r[u];
                } else if (PRE == P_DIAG) {
                    Z[e] = (be[u] != 0.0) ? r[u] / be[u] : 0.0;
                }
            }
        };
        if (NZM > 0) {
#pragma unroll
            for (int k0 = 0; k0 < NZM; k0 += C)
                if (k0 < nz) forward(k0, &y[k0]);
        } else {
            for (int k0 = 0; k0 < nz; k0 += C) forward(k0, y);
        }
        // back substitution: sol_k = sol_k - gamma_{k+1} sol_{k+1}
        if (PRE == P_SIA && solve) {
            if (NZM > 0) {
#pragma unroll
                for (int k0 = (NZM - 1) / C * C; k0 >= 0; k0 -= C) {
                    if (k0 >= nz) continue;
                    double ga[C];
#pragma unroll
                    for (int u = 0; u < C; ++u) ga[u] = (k0 + u < nz - 1) ? fg[(long long)(k0 + u + 1) * NQ + q] : 0.0;
#pragma unroll
                    for (int u = C - 1; u >= 0; --u) {
                        if (k0 + u < nz - 1) y[k0 + u] = prev = __dsub_rn(y[k0 + u], __dmul_rn(ga[u], prev));
                        if (k0 + u < nz) Z[(long long)(k0 + u) * NQ + q] = y[k0 + u];
                    }
                }
            } else {
                for (int k1 = nz - 2; k1 >= 0; k1 -= C) {
                    double ga[C], yy[C];
#pragma unroll
                    for (int u = 0; u < C; ++u) {
                        ga[u] = (k1 - u >= 0) ? fg[(long long)(k1 - u + 1) * NQ + q] : 0.0;
                        yy[u] = (k1 - u >= 0) ? Z[(long long)(k1 - u) * NQ + q] : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < C; ++u)
                        if (k1 - u >= 0)
                            Z[(long long)(k1 - u) * NQ + q] = prev = __dsub_rn(yy[u], __dmul_rn(ga[u], prev));
                }
            }
        }
        if (PRE == P_SIA && c.zs) {  // + the line solution, its halo update taken on the way
            const long long sz = halo_src(g, i, j, q);
            const double zl = sz >= 0 ? c.zs[(comp ? NQ : 0) + sz] : 0.0;
            for (int k0 = 0; k0 < nz; k0 += C) {
                double zz[C];
#pragma unroll
                for (int u = 0; u < C; ++u) zz[u] = (k0 + u < nz) ? Z[(long long)(k0 + u) * NQ + q] : 0.0;
#pragma unroll
                for (int u = 0; u < C; ++u)
                    if (k0 + u < nz) Z[(long long)(k0 + u) * NQ + q] = __dadd_rn(zz[u], zl);
            }
        }
    }
    if (DOT) {  // the products again from r and z (this thread's own stores), C levels at a time
        DD s0{0.0, 0.0};
        for (int k0 = 0; k0 < nz; k0 += C) {
            double p[C];
#pragma unroll
            for (int u = 0; u < C; ++u) {
                p[u] = 0.0;
                if (in && k0 + u < nz) {
                    const long long e = (long long)(k0 + u) * NQ + q;
                    const double z = Z[e];
                    p[u] = __dmul_rn(R[e], z);
                    if (c.setd) D[e] = z;
                }
                if (comp) sprod[u][cl] = p[u];
            }
            __syncthreads();
            if (!comp && own) {
#pragma unroll
                for (int u = 0; u < C; ++u)
                    if (k0 + u < nz) s0 = dd_add_d(s0, __dadd_rn(p[u], sprod[u][cl]));
            }
            __syncthreads();
        }
        reduce_and_finish<1>(rc, s0, s0);
    }
}

// S0 = (b,b) over the owned columns, per column in level order (:1208-1216, :3067-3074).
__global__ void __launch_bounds__(kBlock) k_dot_bb(Geom g, const double *__restrict__ bu, const double *__restrict__ bv,
                                                   RedCtx rc) {
    if (rc.st->done) return;
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    DD s0{0.0, 0.0};
    int i = -1, j = -1;
    if (q < g.NQ) col_of(g, q, i, j);
    if (q < g.NQ && owned(g, i, j))
        for (int k0 = 0; k0 < g.nz; k0 += 8) {
            double t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const long long e = (long long)(k0 + u) * g.NQ + q;
                t[u] = (k0 + u < g.nz) ? __dadd_rn(__dmul_rn(bu[e], bu[e]), __dmul_rn(bv[e], bv[e])) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (k0 + u < g.nz) s0 = dd_add_d(s0, t[u]);
        }
    reduce_and_finish<1>(rc, s0, s0);
}

// ---------------------------------------------------------------------------
// nonlinear-iteration diagnostics (glissade_velo_higher.F90)
// ---------------------------------------------------------------------------
// compute_residual_vector_{2d,3d} (:9502-9689 / :9693-9894), after y = A u (k_mv MV_PLAIN,
// the same statements and order): resid = y - b on owned active vertices, 0 elsewhere;
// S0 = sum of resid_u^2 + resid_v^2, S1 = sum of bu^2 + bv^2 over owned active vertices (the
// global sums' fixed tree).
__global__ void __launch_bounds__(kBlock) k_resid_vec(Geom g, const int32_t *__restrict__ act,
                                                      const double *__restrict__ yu, const double *__restrict__ yv,
                                                      const double *__restrict__ bu, const double *__restrict__ bv,
                                                      double *__restrict__ ru, double *__restrict__ rv, RedCtx rc) {
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    DD s0{0.0, 0.0}, s1{0.0, 0.0};
    if (q < g.NQ) {
        int i, j;
        col_of(g, q, i, j);
        const bool on = owned(g, i, j) && act[q] != 0;
        for (int k0 = 0; k0 < g.nz; k0 += kDotChunk) {  // a chunk's loads together, then its terms in order
            double y1[kDotChunk], y2[kDotChunk], b1[kDotChunk], b2[kDotChunk];
#pragma unroll
            for (int u = 0; u < kDotChunk; ++u) {
                const long long e = (long long)(k0 + u) * g.NQ + q;
                const bool in = on && k0 + u < g.nz;
                y1[u] = in ? yu[e] : 0.0;
                y2[u] = in ? yv[e] : 0.0;
                b1[u] = in ? bu[e] : 0.0;
                b2[u] = in ? bv[e] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kDotChunk; ++u) {
                if (k0 + u >= g.nz) continue;
                const long long e = (long long)(k0 + u) * g.NQ + q;
                const double r1 = on ? __dsub_rn(y1[u], b1[u]) : 0.0, r2 = on ? __dsub_rn(y2[u], b2[u]) : 0.0;
                ru[e] = r1;
                rv[e] = r2;
                if (on) {
                    s0 = dd_add_d(s0, __dadd_rn(__dmul_rn(r1, r1), __dmul_rn(r2, r2)));
                    s1 = dd_add_d(s1, __dadd_rn(__dmul_rn(b1[u], b1[u]), __dmul_rn(b2[u], b2[u])));
                }
            }
        }
    }
    reduce_and_finish<2>(rc, s0, s1);
}

// compute_residual_velocity_{2d,3d} (:10188-10310 / :10314-10446) over owned vertices and
// levels k < kmax: speed = sqrt(u**2 + v**2); where speed /= 0, d = abs((oldspeed-speed)/speed).
// Max modes: the largest d, as atomicMax on the bits of a non-negative double (a NaN d never
// wins, as "d > resid_velo" is false for it; the state's maxbits starts at +0).  Mean mode: the
// count and the sum of d (the global sums' fixed tree; EPI_SUM).
__global__ void __launch_bounds__(kBlock) k_resid_velo(Geom g, int kmax, int mean, const double *__restrict__ u,
                                                       const double *__restrict__ v, const double *__restrict__ us,
                                                       const double *__restrict__ vs, RedCtx rc) {
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    DD s0{0.0, 0.0};
    unsigned long long cnt = 0;
    if (q < g.NQ) {
        int i, j;
        col_of(g, q, i, j);
        if (owned(g, i, j))
            for (int k = 0; k < kmax; ++k) {
                const long long e = (long long)k * g.NQ + q;
                const double speed = __dsqrt_rn(__dadd_rn(__dmul_rn(u[e], u[e]), __dmul_rn(v[e], v[e])));
                if (speed != 0.0) {
                    const double old = __dsqrt_rn(__dadd_rn(__dmul_rn(us[e], us[e]), __dmul_rn(vs[e], vs[e])));
                    const double d = fabs(__ddiv_rn(__dsub_rn(old, speed), speed));
                    if (mean) {
                        ++cnt;
                        s0 = dd_add_d(s0, d);
                    } else if (d > 0.0) {
                        atomicMax(&rc.st->maxbits, (unsigned long long)__double_as_longlong(d));
                    }
                }
            }
    }
    if (mean) {
        if (cnt) atomicAdd(&rc.st->count, cnt);
        reduce_and_finish<1>(rc, s0, s0);
    }
}

// ---------------------------------------------------------------------------
// check_symmetry_assembled_matrix_{3d,2d} (glissade_velo_higher.F90:10854-11117 and
// :10648-10850) pair by pair
// ---------------------------------------------------------------------------
// The reference visits every owned active row R and compares each coefficient of offset d
// with its transpose partner at row R+d, offset -d: Auu with Auu, Auv with Avu (Auu's
// diagonal in the tolerance), then Avv with Avv, Avu with Auv (Avv's diagonal).  A visit
// whose values differ raises maxdiff to |val2 - val1| and, when that is below
// eps11 * |diag of the visited row|, the 3D check averages the pair in place; otherwise it
// warns.  Every coefficient has exactly one partner, so the in-place loop is a function of
// each pair alone: a pair is seen from R (if R is owned and active) and from R+d (likewise),
// it is averaged when either visit's test passes on the original values, the earlier visit
// warns when its test fails, and the later one when its own fails and the earlier one did not
// average.  "Earlier" is the reference's loop order: rows j, i, k, then the Auu/Auv loop
// before the Avv/Avu loop.  One thread owns each pair (the Auv member of an Auv-Avu pair; of
// an Auu or Avv pair the member with the smaller offset index c < 26 - c), reads both values
// and writes both, and only the owners write; the diagonals that the tolerance reads are
// their own partners and are never written, so no thread reads what another writes.
constexpr double kEps11 = 1.0e-11;  // eps11, libglimmer/glimmer_paramets.F90:77

// Element offsets of coefficient c (canonical offset index (iA+1) + 3(jA+1) + 9(kA+1)) at
// level k of column q: the canonical planes (map = identity) or the caller's Fortran blocks,
// (27, nz, NX, NY) in 3D (raw3) or (NX, NY, 9) in 2D, through the caller's indxA map.
struct SymIdx {
    int32_t map[27];
    long long n;  // nz * NQ
    long long NQ;
    int nz;
    int raw3;
    __device__ __forceinline__ long long at(int c, int k, long long q) const {
        const long long m = map[c] - 1;
        return raw3 ? m + 27LL * (k + (long long)nz * q) : m * n + (long long)k * NQ + q;
    }
};

// blockIdx.z: the pairs' kind and the coefficient c of their first member (Auu-Auu and Avv-Avv: c <=
// NC/2, Auv-Avu: all), blockIdx.y its level, x its column, so that a block reads two runs of
// columns.  (One flat index over all coefficients, divided by 64-bit sizes per thread and half its
// threads without a pair, took 276 us on 201x161x11; now 170.)
// out[0]: maxdiff as the bits of a non-negative double
// (a NaN difference never wins: "abs(val2 - val1) > maxdiff" is false for it), out[1]: warnings.
template <int NC>
__host__ __device__ constexpr int sym_pairs() { return 2 * (NC / 2 + 1) + NC; }

template <int NC, bool FIX>
__global__ void __launch_bounds__(kBlock) k_sym_check(Geom g, SymIdx L, const int32_t *__restrict__ act,
                                                      double *Auu, double *Auv, double *Avu, double *Avv,
                                                      unsigned long long *out) {
    constexpr int NH = NC / 2 + 1;
    const int w = blockIdx.z, k = blockIdx.y;
    const int kind = w < NH ? 0 : (w < NH + NC ? 1 : 2), c = w - (kind == 0 ? 0 : (kind == 1 ? NH : NH + NC));
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    unsigned long long dbits = 0ull, nw = 0ull;
    if (q < g.NQ) {
        const int j = (int)q / g.NX, i = (int)q - j * g.NX;
        const int iA = c % 3 - 1, jA = (c / 3) % 3 - 1, kA = (NC == 27) ? c / 9 - 1 : 0;
        const int cc = NC - 1 - c, cd = NC / 2;
        const int kp = k + kA, ip = i + iA, jp = j + jA;
        // a partner outside the arrays (owned rows at the array edge) is not compared
        const bool inside = kp >= 0 && kp < g.nz && ip >= 0 && ip < g.NX && jp >= 0 && jp < g.NY;
        if (inside) {
            const long long qp = (long long)jp * g.NX + ip;
            const bool self = kind != 1 && c == cc;  // a diagonal is its own partner
            const bool visA = owned(g, i, j) && act[q] != 0;
            const bool visB = !self && owned(g, ip, jp) && act[qp] != 0;
            double *X = kind == 0 ? Auu : (kind == 1 ? Auv : Avv);
            double *Y = kind == 0 ? Auu : (kind == 1 ? Avu : Avv);
            const long long ea = L.at(c, k, q), eb = L.at(cc, kp, qp);
            const double x = (visA || visB) ? X[ea] : 0.0, y = (visA || visB) ? Y[eb] : 0.0;
            if (y != x) {  // val2 /= val1, true for a NaN
                const double d = fabs(__dsub_rn(y, x));
                if (d > 0.0) dbits = (unsigned long long)__double_as_longlong(d);
                // visit A from R: Auu's diagonal for the Auu and Auv checks, Avv's for Avv;
                // visit B from R+d: Auu's for Auu, Avv's for the Avv and Avu checks
                const double *DA = kind == 2 ? Avv : Auu, *DB = kind == 0 ? Auu : Avv;
                const bool passA = visA && d < __dmul_rn(kEps11, fabs(DA[L.at(cd, k, q)]));
                const bool passB = visB && d < __dmul_rn(kEps11, fabs(DB[L.at(cd, kp, qp)]));
                if (FIX) {
                    const long long rowA = k + (long long)g.nz * q, rowB = kp + (long long)g.nz * qp;
                    const bool aFirst = rowA <= rowB;  // equal rows: the Auv check (A) precedes Avu's (B)
                    const bool v1 = aFirst ? visA : visB, p1 = aFirst ? passA : passB;
                    const bool v2 = aFirst ? visB : visA, p2 = aFirst ? passB : passA;
                    nw = (unsigned long long)(v1 && !p1) + (unsigned long long)(v2 && !p2 && !p1);
                    if (passA || passB) {
                        const double avg = __dmul_rn(0.5, __dadd_rn(x, y));
                        X[ea] = avg;
                        Y[eb] = avg;
                    }
                } else {
                    nw = (unsigned long long)(visA && !passA) + (unsigned long long)(visB && !passB);
                }
            }
        }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        dbits = max(dbits, __shfl_down_sync(0xffffffffu, dbits, off));
        nw += __shfl_down_sync(0xffffffffu, nw, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (dbits) atomicMax(&out[0], dbits);
        if (nw) atomicAdd(&out[1], nw);
    }
}

// ---------------------------------------------------------------------------
// tridiagonal line preconditioners (precond 3 local, 4 global) on one task
// ---------------------------------------------------------------------------
// On one task the global form's solution is its particular solution (tasks_rc = 1,
// tridiag_solver_global_2d :5495-5497), which is the local form's arithmetic on the owned
// block; the forms differ in the global setup's extra zero-pivot check (:4472-4488), in
// 3D inactive columns (local zeroes all nine summed couplings, :3823-3833; global only sets
// the centre, :4025-4032) and in the local back substitution continuing below the owned
// range (:4999-5001, gamma = omega = 0 there).  Lines: u along rows j (i varies), v along
// columns i (j varies), one thread per line.  Work planes of NQ doubles:
enum TriPlane {
    TU_SUB = 0, TU_DG, TU_SP, TU_ADR, TU_OM, TU_DEN,  // u lines: sub, diag, super, 1/diag, omega, 1/denom
    TV_SUB, TV_DG, TV_SP, TV_ADR, TV_OM, TV_DEN,      // v lines
    TZS_U, TZS_V,                                     // 3D: line solution of the summed problem
    NTRI
};

// Coefficient planes of the line systems: [u/v][sub, diag, super] -> the device planes of the
// caller's raw indices m (2D: plane c[..][0]) or m, m+9, m+18 (3D vertical sums), with m the
// raw index (1..9) indxA_2d gives the coupling.
struct TriMap {
    int c[2][3][3];
    int m[2][3];
};

// setup_preconditioner_tridiag_{local,global}_{2d,3d}: the line coefficients, zero-diagonal
// fix (:4306-4313) and 1/diag (:4347), omega = 1/denom = 0 until k_tri_factor.  3D: sums
// over levels of the three vertical offsets, ((s + A(m)) + A(m+9)) + A(m+18) (:3813-3819).
template <int NC>
__global__ void k_tri_coef(Geom g, const double *__restrict__ A, const int32_t *__restrict__ act, TriMap tm,
                           int global, double *__restrict__ T) {
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    if (q >= g.NQ) return;
    const long long plane = (long long)g.nz * g.NQ;
    // 3D, global: the staggered halo update of the nine summed planes (:4055-4058) is taken on the way: the
    // column s whose sums q holds after it, or zero.  With no_ice it reaches the last owned row and
    // column, otherwise owned positions only where these lie in the halo.
    const long long s = (NC == 27 && global) ? halo_src(g, (int)(q % g.NX), (int)(q / g.NX), q) : q;
    for (int comp = 0; comp < 2; ++comp) {
        const double *B = A + (comp ? 3LL : 0LL) * NC * plane;  // Auu or Avv
        double v[3] = {0.0, 0.0, 0.0};
        for (int e = 0; e < 3 && s >= 0; ++e) {
            if (NC == 9) {
                v[e] = B[(long long)tm.c[comp][e][0] * g.NQ + q];
            } else {
                double sum = 0.0;
                for (int k = 0; k < g.nz; ++k) {
                    const long long o = (long long)k * g.NQ + s;
                    sum = __dadd_rn(__dadd_rn(__dadd_rn(sum, B[tm.c[comp][e][0] * plane + o]),
                                              B[tm.c[comp][e][1] * plane + o]),
                                    B[tm.c[comp][e][2] * plane + o]);
                }
                if (act[s] == 0) {
                    if (tm.m[comp][e] == 5) sum = 1.0;
                    else if (!global) sum = 0.0;
                }
                v[e] = sum;
            }
        }
        if (v[1] == 0.0) { v[1] = 1.0; v[0] = 0.0; v[2] = 0.0; }
        double *P = T + (comp ? TV_SUB : TU_SUB) * g.NQ;
        P[0 * g.NQ + q] = v[0];
        P[1 * g.NQ + q] = v[1];
        P[2 * g.NQ + q] = v[2];
        P[3 * g.NQ + q] = __ddiv_rn(1.0, v[1]);
        P[4 * g.NQ + q] = 0.0;
        P[5 * g.NQ + q] = 0.0;
    }
}

__device__ __forceinline__ void tri_line(const Geom &g, int t, bool &along_i, int &l, int &s0, int &s1) {
    const int nu = g.jhi - g.jlo + 1;
    along_i = t < nu;
    l = along_i ? g.jlo + t : g.ilo + (t - nu);
    s0 = along_i ? g.ilo : g.jlo;
    s1 = along_i ? g.ihi : g.jhi;
}
__device__ __forceinline__ long long tri_at(const Geom &g, bool along_i, int l, int s) {
    return along_i ? (long long)l * g.NX + s : (long long)s * g.NX + l;
}
__host__ __device__ inline int tri_lines(const Geom &g) { return (g.jhi - g.jlo + 1) + (g.ihi - g.ilo + 1); }

// Forward elimination per owned line (:4324-4342 / :4361-4379; global :4441-4452), and for the
// global form the reverse recurrence it checks for zero pivots (:4464-4488).  A zero pivot
// is GM_FATAL in the reference: the solve ends with CISMGPU_EDIVZERO before it starts.
__global__ void k_tri_factor(Geom g, int global, double *__restrict__ T, SolveState *st) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    if (t >= tri_lines(g)) return;
    bool along_i;
    int l, s0, s1;
    tri_line(g, t, along_i, l, s0, s1);
    double *P = T + (along_i ? TU_SUB : TV_SUB) * g.NQ;
    const double *sub = P, *dg = P + g.NQ, *sp = P + 2 * g.NQ;
    double *om = P + 4 * g.NQ, *den = P + 5 * g.NQ;
    long long e = tri_at(g, along_i, l, s0);
    double omp = __ddiv_rn(sp[e], dg[e]);
    om[e] = omp;
    for (int s = s0 + 1; s <= s1; ++s) {
        e = tri_at(g, along_i, l, s);
        const double d = __dsub_rn(dg[e], __dmul_rn(sub[e], omp));
        if (d == 0.0) {
            st->status = CISMGPU_EDIVZERO;
            st->done = 1;
            return;
        }
        const double dn = __ddiv_rn(1.0, d);
        den[e] = dn;
        omp = __dmul_rn(sp[e], dn);
        om[e] = omp;
    }
    if (global) {
        e = tri_at(g, along_i, l, s1);
        double o = __ddiv_rn(sub[e], dg[e]);
        for (int s = s1 - 1; s >= s0; --s) {
            e = tri_at(g, along_i, l, s);
            const double d = __dsub_rn(dg[e], __dmul_rn(sp[e], o));
            if (d == 0.0) {
                st->status = CISMGPU_EDIVZERO;
                st->done = 1;
                return;
            }
            o = __ddiv_rn(sub[e], d);
        }
    }
}

// Line solves of tridiag_solver_local_2d (:4985-5013 u, :5041-5069 v) from planes bu, bv into
// xu, xv, which hold zeros outside the lines: gamma forward, then back substitution.  SUM (3D): the
// right-hand side is the sum of r over the levels, in level order (tridiag_solver_local_3d :4585-4590).
// PENDING: the halo update of b is still to come (U_RHALO, by the kernel that follows) and reaches owned
// positions (halo_reaches_owned), so the lines read what it will leave.  A variant of its own: the test
// in every staged element cost a 150x101x11 solve 6 % where no update reaches an owned position.
// A line is a chain of dependent FP64 operations (three a position forward, two backward; 66 ns a
// position, 10 of the 22 us below), so everything else is taken off the chain: a block stages kTriLines lines,
// kTriChunk positions at a time, in shared memory with all its threads (coalesced for the u lines,
// whole 32-byte sectors for the v lines, kTriLines adjacent columns), one thread per line runs the
// recurrences there, and all threads store.  The operations and their order are the reference's.
// 150x101x11: 22 us for the lines and the level sums; with a thread per line on global memory, all
// lines in one block, and the sums as a launch of their own, 55 + 6.5.
constexpr int kTriLines = 4, kTriChunk = 376, kTriThreads = 128;
static_assert(4 * kTriLines * (kTriChunk + 1) * sizeof(double) <= 48 * 1024, "no opt-in shared memory");

template <bool SUM, bool PENDING>
__global__ void __launch_bounds__(kTriThreads) k_tri_lines(Geom g, int global, const double *__restrict__ bu,
                                                           const double *__restrict__ bv, double *__restrict__ xu,
                                                           double *__restrict__ xv, const double *__restrict__ T,
                                                           const SolveState *st) {
    after_previous();
    if (st->done) return;
    extern __shared__ double stri[];  // [b / gamma, sub, 1/denom, omega][line][pitch]
    const int nu = g.jhi - g.jlo + 1, nug = (nu + kTriLines - 1) / kTriLines;
    const bool along_i = (int)blockIdx.x < nug;
    const int l0 = along_i ? g.jlo + (int)blockIdx.x * kTriLines : g.ilo + ((int)blockIdx.x - nug) * kTriLines;
    const int nl = min(kTriLines, (along_i ? g.jhi : g.ihi) - l0 + 1);
    const int s0 = along_i ? g.ilo : g.jlo, s1 = along_i ? g.ihi : g.jhi, len = s1 - s0 + 1;
    const int nch = (len + kTriChunk - 1) / kTriChunk, pitch = min(len, kTriChunk) + 1;
    const double *P = T + (along_i ? TU_SUB : TV_SUB) * g.NQ;
    const double *sub = P, *adr = P + 3 * g.NQ, *om = P + 4 * g.NQ, *den = P + 5 * g.NQ;
    const double *b = along_i ? bu : bv;
    double *x = along_i ? xu : xv;
    double *sb = stri, *ss = sb + kTriLines * pitch, *sd = ss + kTriLines * pitch, *so = sd + kTriLines * pitch;
    const int tid = threadIdx.x;
    // the elements (line, position) of a chunk: positions run fastest along u lines, lines along v lines
    auto each = [&](int c0, int n, auto &&f) {
        for (int w = tid; w < nl * n; w += kTriThreads) {
            const int ln = along_i ? w / n : w % nl, s = along_i ? w % n : w / nl;
            f(ln * pitch + s, tri_at(g, along_i, l0 + ln, s0 + c0 + s));
        }
    };
    double gp = 0.0;
    for (int c = 0; c < nch; ++c) {
        const int c0 = c * kTriChunk, n = min(kTriChunk, len - c0);
        each(c0, n, [&](int w, long long e) {
            long long f = e;
            if (PENDING) {
                const int j = (int)e / g.NX, i = (int)e - j * g.NX;
                f = halo_src(g, i, j, e);
            }
            double v = 0.0;
            if (SUM && (!PENDING || f >= 0)) {
                for (int k0 = 0; k0 < g.nz; k0 += 8) {
                    double r[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) r[u] = (k0 + u < g.nz) ? b[(long long)(k0 + u) * g.NQ + f] : 0.0;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k0 + u < g.nz) v = __dadd_rn(v, r[u]);
                }
            } else if (!PENDING || f >= 0) {
                v = b[f];
            }
            sb[w] = v;
            ss[w] = sub[e];
            sd[w] = den[e];
            if (nch == 1) so[w] = om[e];
        });
        __syncthreads();
        if (tid < nl) {
            double *vb = sb + tid * pitch;
            const double *vs = ss + tid * pitch, *vd = sd + tid * pitch;
            int s = 0;
            if (c == 0) {
                gp = __dmul_rn(vb[0], adr[tri_at(g, along_i, l0 + tid, s0)]);
                vb[0] = gp;
                s = 1;
            }
            for (; s < n; s += 8) {
                double r[8], p[8], d[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int w = min(s + u, n - 1);
                    r[u] = vb[w];
                    p[u] = vs[w];
                    d[u] = vd[w];
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (s + u < n) {
                        gp = __dmul_rn(__dsub_rn(r[u], __dmul_rn(p[u], gp)), d[u]);
                        vb[s + u] = gp;
                    }
            }
        }
        __syncthreads();
        if (nch > 1) {
            each(c0, n, [&](int w, long long e) { x[e] = sb[w]; });
            __syncthreads();
        }
    }
    double xn = gp;
    for (int c = nch - 1; c >= 0; --c) {
        const int c0 = c * kTriChunk, n = min(kTriChunk, len - c0);
        if (nch > 1) {
            each(c0, n, [&](int w, long long e) {
                sb[w] = x[e];  // gamma, as this block stored it
                so[w] = om[e];
            });
            __syncthreads();
        }
        if (tid < nl) {
            double *vb = sb + tid * pitch;
            const double *vo = so + tid * pitch;
            for (int s = (c == nch - 1) ? n - 2 : n - 1; s >= 0; s -= 8) {
                double r[8], o[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int w = max(s - u, 0);
                    r[u] = vb[w];
                    o[u] = vo[w];
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (s - u >= 0) {
                        xn = __dsub_rn(r[u], __dmul_rn(o[u], xn));
                        vb[s - u] = xn;
                    }
            }
        }
        __syncthreads();
        each(c0, n, [&](int w, long long e) { x[e] = sb[w]; });
        __syncthreads();
    }
    // the local back substitution runs on below the owned range (:4999-5001; gamma is zero there)
    if (!global && tid < nl)
        for (int s = s0 - 1; s >= 0; --s) {
            const long long e = tri_at(g, along_i, l0 + tid, s);
            xn = __dsub_rn(0.0, __dmul_rn(om[e], xn));
            x[e] = xn;
        }
}

// Blocks and shared memory of k_tri_lines.
inline unsigned tri_blocks(const Geom &g) {
    return (unsigned)((g.jhi - g.jlo + kTriLines) / kTriLines + (g.ihi - g.ilo + kTriLines) / kTriLines);
}
inline size_t tri_smem(const Geom &g) {
    const int len = g.ihi - g.ilo > g.jhi - g.jlo ? g.ihi - g.ilo + 1 : g.jhi - g.jlo + 1;
    return (size_t)4 * kTriLines * ((len < kTriChunk ? len : kTriChunk) + 1) * sizeof(double);
}

// ---------------------------------------------------------------------------
// staggered halo on one rank (parallel_mpi.F90:10772-10936)
// ---------------------------------------------------------------------------
// Threads enumerate the ring columns: rows j in {0,1,NY-2,NY-1} (all i), then
// columns i in {0,1,NX-2,NX-1} for 2 <= j <= NY-3.  A periodic halo position
// (i in {0,1,NX-1} or j in {0,1,NY-1}) takes the value at (pi(i), pj(j)) with
// pi(0)=NX-3, pi(1)=NX-2, pi(NX-1)=2 (identity otherwise): the composite of the
// east-west exchange on owned rows followed by the north-south exchange on all
// columns.  Sources are never halo positions, so one pass is race free.  Outflow
// then zeroes i,j in {0, N-1}; no_ice zeroes i,j in {0,1,N-2,N-1}.  Levels k run over
// blockIdx.y, blockIdx.y + gridDim.y, ... (many planes, such as the 27 nz coefficient planes of
// a block, take a grid with several rows of blocks).
__global__ void __launch_bounds__(kBlock) k_halo(Geom g, double *__restrict__ au, double *__restrict__ av,
                                                 const SolveState *st) {
    if (st && st->done) return;
    const int NX = g.NX, NY = g.NY;
    const long long nring = 4LL * NX + 4LL * (NY - 4);
    const long long t = (long long)blockIdx.x * kBlock + threadIdx.x;
    if (t >= nring) return;
    int i, j;
    if (t < 4LL * NX) {
        const int r = (int)(t / NX);
        i = (int)(t - (long long)r * NX);
        j = (r < 2) ? r : NY - 4 + r;  // 0,1,NY-2,NY-1
    } else {
        const long long u = t - 4LL * NX;
        const int r = (int)(u / (NY - 4));
        j = 2 + (int)(u - (long long)r * (NY - 4));
        i = (r < 2) ? r : NX - 4 + r;
    }
    const long long q = (long long)j * NX + i;
    if (zero_pos(g, i, j)) {
        for (int k = blockIdx.y; k < g.nz; k += gridDim.y) {
            au[(long long)k * g.NQ + q] = 0.0;
            av[(long long)k * g.NQ + q] = 0.0;
        }
        return;
    }
    if (g.periodic) {
        if (!periodic_halo(g, i, j)) return;
        const long long s = (long long)pmap(j, NY) * NX + pmap(i, NX);
        for (int k = blockIdx.y; k < g.nz; k += gridDim.y) {
            au[(long long)k * g.NQ + q] = au[(long long)k * g.NQ + s];
            av[(long long)k * g.NQ + q] = av[(long long)k * g.NQ + s];
        }
    }
}

// ---------------------------------------------------------------------------
// owned-vertex global sum of arr1 + arr2 (parallel_global_sum_stagger on one rank)
// ---------------------------------------------------------------------------
// FORTRAN_LAYOUT: element (k, q) at k + nz*q (the caller's arrays); otherwise k*NQ + q.
// Same tree as every solver reduction: column dd sums over k, block tree per chunk of
// 256 columns, chunk partials, fixed final tree by the last CTA (which also resets the
// ticket for the next use).
template <bool FORTRAN_LAYOUT>
__global__ void __launch_bounds__(kBlock) k_gsum(Geom g, const double *__restrict__ a1, const double *__restrict__ a2,
                                                 DD *partials, unsigned int *ticket, double *out) {
    __shared__ DD sm[8];
    __shared__ bool last;
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    DD acc{0.0, 0.0};
    if (q < g.NQ) {
        int i, j;
        j = (int)(q / g.NX);
        i = (int)(q - (long long)j * g.NX);
        if (owned(g, i, j))
            for (int k = 0; k < g.nz; ++k) {
                const long long e = FORTRAN_LAYOUT ? (long long)k + (long long)g.nz * q : (long long)k * g.NQ + q;
                acc = dd_add_d(acc, __dadd_rn(a1[e], a2[e]));
            }
    }
    DD b = block_tree(acc, sm);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = b;
        __threadfence();
        const unsigned int t = atomicAdd(ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    DD a{0.0, 0.0};
    for (unsigned int c = threadIdx.x; c < gridDim.x; c += kBlock) {
        DD p;
        p.hi = __ldcg(&partials[c].hi);
        p.lo = __ldcg(&partials[c].lo);
        a = dd_add(a, p);
    }
    DD r = block_tree(a, sm);
    if (threadIdx.x == 0) {
        *ticket = 0u;
        *out = r.hi + r.lo;
    }
}

// ---------------------------------------------------------------------------
// layout conversion between the caller's Fortran arrays and device planes
// ---------------------------------------------------------------------------
// 3D block A(27,nz,NX,NY) raw -> planes [c][k][q]; canonical c reads m = indxA(c)
__global__ void k_perm_block3(Geom g, const double *__restrict__ raw, double *__restrict__ dst,
                              const int32_t *__restrict__ map27) {
    const long long node = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // Fortran order k + nz*q
    const long long n = (long long)g.nz * g.NQ;
    if (node >= n) return;
    const long long q = node / g.nz;
    const int k = (int)(node - q * g.nz);
    const double *src = raw + 27LL * node;
    for (int c = 0; c < 27; ++c) dst[(long long)c * n + (long long)k * g.NQ + q] = src[map27[c] - 1];
}

// 2D block A(NX,NY,9) raw (already planes) -> canonical planes
__global__ void k_perm_block2(Geom g, const double *__restrict__ raw, double *__restrict__ dst,
                              const int32_t *__restrict__ map9) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.NQ) return;
    for (int c = 0; c < 9; ++c) dst[(long long)c * g.NQ + q] = raw[(long long)(map9[c] - 1) * g.NQ + q];
}

// vector (nz,NX,NY) Fortran <-> level-major planes
__global__ void k_vec_in(Geom g, const double *__restrict__ raw, double *__restrict__ dst) {
    const long long node = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)g.nz * g.NQ;
    if (node >= n) return;
    const long long q = node / g.nz;
    const int k = (int)(node - q * g.nz);
    dst[(long long)k * g.NQ + q] = raw[node];
}

__global__ void k_vec_out(Geom g, const double *__restrict__ src, double *__restrict__ raw) {
    const long long node = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)g.nz * g.NQ;
    if (node >= n) return;
    const long long q = node / g.nz;
    const int k = (int)(node - q * g.nz);
    raw[node] = src[(long long)k * g.NQ + q];
}

// Reproducible-sum solves (parallel%reprosum): the two product fields work2u = au*bu and
// work2v = av*bv of one parallel_global_sum_stagger call, written in the caller's layout
// (node k + nz*q) that the reproducible sum reads.  An owned node whose au*bu + av*bv is not
// finite is recorded in *flag (1 NaN, 2 +Inf, 4 -Inf) and its products are written as zero,
// so the integer expansion only ever sees finite summands; the host then returns the IEEE
// sum of the non-finite values instead.
__global__ void __launch_bounds__(kBlock) k_repro_products(Geom g, const double *__restrict__ au,
                                                           const double *__restrict__ bu,
                                                           const double *__restrict__ av,
                                                           const double *__restrict__ bv, double *__restrict__ o1,
                                                           double *__restrict__ o2, int *flag) {
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    if (q >= g.NQ) return;
    int i, j;
    col_of(g, q, i, j);
    const bool own = owned(g, i, j);
    int f = 0;
    for (int k = 0; k < g.nz; ++k) {
        const long long e = (long long)k * g.NQ + q;
        double p1 = __dmul_rn(au[e], bu[e]);
        double p2 = __dmul_rn(av[e], bv[e]);
        if (own) {
            const double v = __dadd_rn(p1, p2);
            if (v != v) f |= 1;
            else if (v == __longlong_as_double(0x7ff0000000000000LL)) f |= 2;
            else if (v == __longlong_as_double(0xfff0000000000000LL)) f |= 4;
            if (!(v - v == 0.0)) { p1 = 0.0; p2 = 0.0; }
        }
        o1[(long long)k + (long long)g.nz * q] = p1;
        o2[(long long)k + (long long)g.nz * q] = p2;
    }
    if (f) atomicOr(flag, f);
}

// The scalar epilogue of a sum computed on the host side of the stream (the reproducible sum).
__global__ void k_epilogue_value(SolveState *st, int epi, int iter, double S0, double S1) {
    if (st->done) return;
    epilogue(st, epi, iter, S0, S1);
}

// ---------------------------------------------------------------------------
// Global sums in the reference's own order (parallel_global_sum_stagger without reprosum,
// parallel_mpi.F90:6770 (3D), :6637 (2D), nflds forms :7042 (3D), :6904 (2D)):
//   local_sum = local_sum + arr1(k,i,j) + arr2(k,i,j)
// over owned vertices, j outer, then i, then k, every addition rounded in turn, and the
// work arrays products rounded first (worku = ru*zu, ...).  A chain of dependent additions
// has no parallelism, so one thread adds while the other warps of the CTA stage the next
// chunk of summands in shared memory (two buffers).  With two fields (Chronopoulos-Gear's
// nflds = 2 calls) the two chains are independent and run interleaved in the same thread.
// ---------------------------------------------------------------------------
constexpr int kSeqChunk = 512;  // summands per term per chunk

struct SeqArgs {
    const double *a[2][2];  // field f: u term a[f][0], v term a[f][1]
    const double *b[2][2];  // and their second factors (null: the term is a itself)
};

// FLAYOUT: element (k, q) at k + nz*q (the caller's arrays); otherwise planes k*NQ + q.
// epi2 != EPI_NONE: the two sums finish two epilogues, epi with S0 then epi2 with S1 (the
// first pass of Chronopoulos-Gear); otherwise one epilogue epi(S0, S1).  out (optional)
// receives S0.  One CTA of kBlock threads.
template <int NF, bool FLAYOUT>
__global__ void __launch_bounds__(kBlock) k_seq_sum(Geom g, SeqArgs s, SolveState *st, int epi, int epi2, int iter,
                                                    double *out) {
    __shared__ double sm[2][NF][2][kSeqChunk];
    if (st && st->done) return;
    const long long W = (long long)(g.ihi - g.ilo + 1) * g.nz;  // summands of one owned row j
    const long long n = (long long)(g.jhi - g.jlo + 1) * W;
    const long long nchunk = (n + kSeqChunk - 1) / kSeqChunk;
    // stage chunk c into buffer buf with threads [t0, kBlock)
    auto stage = [&](long long c, int buf, int t0) {
        for (int t = threadIdx.x - t0; t < kSeqChunk; t += kBlock - t0) {
            const long long e = c * kSeqChunk + t;
            if (e >= n) break;
            const long long r = e / W, rem = e - r * W;
            const int i = g.ilo + (int)(rem / g.nz), k = (int)(rem % g.nz), j = g.jlo + (int)r;
            const long long q = (long long)j * g.NX + i;
            const long long x = FLAYOUT ? (long long)k + (long long)g.nz * q : (long long)k * g.NQ + q;
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    sm[buf][f][h][t] = s.b[f][h] ? __dmul_rn(s.a[f][h][x], s.b[f][h][x]) : s.a[f][h][x];
        }
    };
    double s0 = 0.0, s1 = 0.0;
    if (nchunk > 0) stage(0, 0, 0);
    __syncthreads();
    for (long long c = 0; c < nchunk; ++c) {
        const int buf = (int)(c & 1);
        if (threadIdx.x >= 32) {
            if (c + 1 < nchunk) stage(c + 1, buf ^ 1, 32);
        } else if (threadIdx.x == 0) {
            const int cnt = (int)min((long long)kSeqChunk, n - c * kSeqChunk);
            const double *u0 = sm[buf][0][0], *v0 = sm[buf][0][1];
            const double *u1 = sm[buf][NF - 1][0], *v1 = sm[buf][NF - 1][1];
#pragma unroll 8
            for (int t = 0; t < cnt; ++t) {
                s0 = __dadd_rn(__dadd_rn(s0, u0[t]), v0[t]);
                if (NF > 1) s1 = __dadd_rn(__dadd_rn(s1, u1[t]), v1[t]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (out) *out = s0;
        if (st) {
            if (epi2 != EPI_NONE) {
                epilogue(st, epi, iter, s0, 0.0);
                if (!st->done) epilogue(st, epi2, iter, s1, 0.0);
            } else {
                epilogue(st, epi, iter, s0, s1);
            }
        }
    }
}

__global__ void k_init_state(SolveState *st, double tol, int maxiters) {
    st->eta0 = 1.0; st->eta1 = 0.0; st->eta2 = 0.0; st->alpha = 0.0; st->beta = 0.0;
    st->rho_old = 0.0; st->sigma = 0.0; st->rho = 0.0; st->delta = 0.0;
    st->L2_rhs = 0.0;
    st->err = __longlong_as_double(0x7ff8000000000000LL);  // NaN until the first check
    st->tol = tol;
    st->done = 0; st->status = 0; st->niters = maxiters; st->checks = 0;
    for (int t = 0; t < 4; ++t) st->ticket[t] = 0u;
}

}  // namespace cismgpu

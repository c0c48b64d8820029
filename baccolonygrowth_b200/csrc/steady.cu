/*
 * steady.cu -- steady glucose field of a colony and its adjoint (VJP).
 * No counterpart in the reference: an extension for gradients of a
 * nutrient-profile loss with respect to the diffusivities, the Monod
 * constants and per-cell uptake weights.
 *
 * Problem (2-D x-z grid, nx x nz vertices, spacing h; rows k < nz_agar
 * are agar, the rest the colony region):
 *   F_p(C) = sum_faces Df (C_nb - C_p) / h^2 - q_p vmax C_p / (km + C_p) = 0
 * for k >= 1, C = c0 on row 0 (the agar reservoir), no flux through the
 * other sides.  A point's diffusivity is d_agar or d_colony by its row,
 * a face takes the harmonic mean of its two points.  The uptake density
 * q_p = sum over cells whose centre rounds to p of w_c L_c R_c / h^2 (the
 * deposition GetDensity makes, Compute.cpp:120-253, with a weight per
 * cell: its growth rate).
 *
 * Solve: Newton, each step A delta = F with A = -dF/dC (symmetric positive
 * definite: the diffusion operator plus diag(q vmax km / (km + C)^2)),
 * by conjugate gradients preconditioned with one symmetric V-cycle
 * (red-black Gauss-Seidel, bilinear prolongation, its transpose / 4 as
 * restriction, coarse operators rediscretised at 2h).
 * Adjoint: for a loss L(C), A lambda = -dL/dC at the converged C (A is
 * symmetric), then dL/dtheta = -lambda . dF/dtheta.  This is the exact
 * gradient of the converged solution (implicit function theorem): the
 * V-cycles and Newton steps are not replayed, only the converged state is
 * kept, so memory does not grow with the iteration count.
 * All arithmetic FP64; every reduction runs in a fixed order.
 */
#include "ctx.cuh"
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

#define ST_MAX_LEVELS 12
#define ST_RED_BLOCKS 256
/* points of the levels the one-block tail of the V-cycle holds in shared
 * memory (32 B each: x, b, the reciprocal diagonal, neighbour sums) */
#define ST_TAIL_POINTS 6400
/* points a half-sweep updates on the levels one warp of the tail runs alone */
#define ST_WARP_POINTS 96
#define ST_TAIL_THREADS 512
/* unknowns of the coarsest level up to which its sweeps run as one matrix */
#define ST_OP_MAX 32
#define ST_CHUNK 4               /* CG iterations a captured graph holds (even: buffers alternate) */
#define ST_FIRST 12              /* iterations queued before the host first looks */

struct StLevel {
    int nx, nz;
    double h;
    double* x;     /* correction after pre-smoothing */
    double* xo;    /* ... after post-smoothing (the tiles read their neighbours' x) */
    double* b;     /* right-hand side */
    double* sig;   /* diagonal term */
    double* diag;  /* sig + the face coefficients */
    double* id;    /* 1 / diag, 0 on the Dirichlet row */
    double* cs;    /* per row: coefficient of the faces to the sides, D_k / h^2 */
    double* cd;    /* per row: of the face to the row below; cd[nz] = 0 */
};

struct bcg_steady {
    bcg_steady_params P;
    cudaStream_t stream;
    int nlev;
    StLevel L[ST_MAX_LEVELS];
    int n;                       /* nx * nz */
    int tail;                    /* first level of the one-block tail; nlev: no level fits it */
    int nt0, ntd;                /* blocks of the level-0 tile kernels and of the direction kernel */
    double *C, *q, *F, *g;
    double *cg_x, *cg_r[2], *cg_p[2], *cg_ap;
    double *part_rn, *part_rz[2], *part_pap;   /* per-block partial results, reduced in order by their readers */
    double* scal;                /* [0] tolerance, [1] max |rhs| */
    int* ctl;                    /* [0] done, [1] iterations, [2] their limit */
    double* op;                  /* coarsest level's sweeps as a matrix (column-major) */
    double* image;               /* the tail's coefficients as it keeps them */
    double* pin;                 /* pinned host staging */
    cudaGraphExec_t graph;       /* ST_CHUNK iterations */
    bool graph_off;
    int ncell;
    int* start;                  /* first of each point's cells in that order (n + 1) */
    int* order;                  /* cell of each entry */
    double* cell;                /* x, z, L, R per cell */
    int* cell_pt;                /* grid point of each cell, -1 outside the colony rows */
    double* w;
    double* gw;
    double* gpart;               /* per-block partial sums of the 4 parameter gradients */
    double theta[4];             /* parameters of the last solve */
    bool solved;
};

static int st_err(cudaError_t e) { if (e != cudaSuccess) { bcg_set_cuda_error(e); return BCG_E_CUDA; } return BCG_OK; }
#define ST_TRY(x) do { int r_ = st_err(x); if (r_) return r_; } while (0)

__device__ __forceinline__ double face_d(double a, double b) { return a == b ? a : 2.0 * a * b / (a + b); }

/* ---- the preconditioned CG iteration ------------------------------------- */
/* A x = diag x - sum_f c_f x_nb on rows k >= 1; row 0 is the Dirichlet row
 * (x = 0 there).  A row's diffusivity is constant, so the face coefficients
 * are one value a row (cs, cd).
 *
 * What bounds it: a V-cycle of these grids (8 thousand to 264 thousand
 * points, everything in L2) moves a few MB, a microsecond or two of traffic.
 * One kernel per half-sweep made it 215 to 260 launches, 160 of them for the
 * ten unknowns of the coarsest level: 1.0 ms a cycle at any grid size.
 * Here a level's whole descent (four half-sweeps, residual, restriction) is one
 * launch, and its ascent (prolongation, four half-sweeps) another, on tiles
 * that carry a halo as wide as the sweeps reach and recompute it; the levels
 * that fit one block's shared memory run as one launch; and the vector
 * updates and dot products of CG ride along in the level-0 launches.
 * Measured, device time of one CG iteration with its V-cycle: 129 x 65 points
 * 38 us (tail 22, descent 6.5, ascent 5.1, direction 4.2), 513 x 257 points
 * 68 us, each 1000 us before.  What bounds it now is the chain of dependent
 * phases: the tail's 50 (5 levels), about 0.35 us each. */

/* sum (MAX: largest) of `np` per-block partials, the same value in every
 * thread, in a fixed order */
template <bool MAX, int THREADS>
__device__ double st_total(const double* __restrict__ part, int np, double* sh)
{
    double s = 0.0;
    for (int j = threadIdx.x; j < np; j += THREADS) s = MAX ? fmax(s, part[j]) : s + part[j];
    for (int o = 16; o >= 1; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, s, o);
        s = MAX ? fmax(s, v) : s + v;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    s = sh[0];
    for (int w = 1; w < THREADS / 32; w++) s = MAX ? fmax(s, sh[w]) : s + sh[w];
    return s;
}
/* two sums at once */
template <int THREADS>
__device__ void st_total2(const double* __restrict__ pa, int na, const double* __restrict__ pb, int nb, double* sh,
                          double& ta, double& tb)
{
    double a = 0.0, b = 0.0;
    for (int j = threadIdx.x; j < na || j < nb; j += THREADS) {
        const double va = j < na ? pa[j] : 0.0, vb = j < nb ? pb[j] : 0.0;
        a += va; b += vb;
    }
    for (int o = 16; o >= 1; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) { sh[threadIdx.x >> 5] = a; sh[32 + (threadIdx.x >> 5)] = b; }
    __syncthreads();
    ta = sh[0]; tb = sh[32];
    for (int w = 1; w < THREADS / 32; w++) { ta += sh[w]; tb += sh[32 + w]; }
}
/* the block's own contribution, into part[blockIdx] */
template <bool MAX, int THREADS>
__device__ void st_partial(double s, double* part, int block, double* sh)
{
    for (int o = 16; o >= 1; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, s, o);
        s = MAX ? fmax(s, v) : s + v;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = sh[0];
        for (int w = 1; w < THREADS / 32; w++) s = MAX ? fmax(s, sh[w]) : s + sh[w];
        part[block] = s;
    }
}

/* the CG vectors of one iteration as the level-0 kernels see them */
struct StCg {
    const int* ctl;
    const double* rin;           /* residual before the step (first: the right-hand side) */
    double* rout;                /* ... after it */
    const double* ap;
    const double* p;
    double* x;
    const double* part_rz;       /* r.z of the step's start */
    const double* part_pap;
    double* part_rn;             /* max |r| after the step */
    int n_rz, n_pap, first;
};

/* A tile is T x T points, kept with a halo as W x W in shared memory, the two
 * colours in separate halves (entry j of row lk of colour c is column
 * 2 j + ((lk + c) & 1)): a half-sweep then reads whole rows of entries side
 * by side, where one array would cost every access twice the bank cycles.
 * Points off the grid and the Dirichlet row carry a zero reciprocal diagonal,
 * so a sweep leaves them 0; the outermost ring is never updated, and what is
 * stale there moves in one point per half-sweep. */
template <int T> struct StTile { static constexpr int THREADS = T == 32 ? 512 : 256; };

/* neighbours' part of A x at one point, and the Gauss-Seidel update from it:
 * two short chains of multiply-adds */
__device__ __forceinline__ double st_off(double cs, double cd, double cu, double l, double r, double d, double u)
{
    return fma(cs, l + r, fma(cd, d, cu * u));
}
/* where column li, row lk of a W-wide tile is kept */
template <int W> __device__ __forceinline__ int st_at(int li, int lk) { return ((li + lk) & 1) * (W * W / 2) + lk * (W / 2) + (li >> 1); }
/* one half-sweep over a tile: colour (i + k) & 1, which is (li + lk) & 1 for
 * an even tile origin and halo.  KEEP: the point's neighbour sum takes the
 * place of its b (see the residual). */
template <int W, int THREADS, bool KEEP>
__device__ __forceinline__ void st_half_sweep(double* sx, double* sb, const double* si, const double* rcs,
                                              const double* rcd, int colour)
{
    constexpr int HW = W / 2;
    const double* other = sx + (1 - colour) * (W * HW);
    const int own = colour * (W * HW);
#pragma unroll
    for (int q = threadIdx.x; q < (W - 2) * HW; q += THREADS) {
        const int lk = 1 + q / HW, j = q % HW, par = (lk + colour) & 1, o = lk * HW + j;
        if (par ? j == HW - 1 : j == 0) continue;          /* the ring */
        const double off = st_off(rcs[lk], rcd[lk], rcd[lk + 1], other[o - 1 + par], other[o + par], other[o - HW], other[o + HW]);
        sx[own + o] = (sb[own + o] + off) * si[own + o];
        if (KEEP) sb[own + o] = off;
    }
}

/* Descent on level L: x = two red-black sweeps from zero on b, and the
 * restricted residual (the transpose of the bilinear prolongation, / 4) into
 * the coarser level's b.  CG: level 0, whose b is the CG residual, stepped
 * here (r -= alpha Ap, x += alpha p) with its max-norm.  SMOOTH = false (a
 * one-level hierarchy): the CG step alone. */
template <int T, bool CG, bool SMOOTH>
__global__ void __launch_bounds__(StTile<T>::THREADS) k_st_down(StLevel L, StLevel Lc, StCg cg, int row0)
{
    constexpr int THREADS = StTile<T>::THREADS, HALO = SMOOTH ? 6 : 0, W = T + 2 * HALO;
    constexpr int PER = (W * W + THREADS - 1) / THREADS;
    extern __shared__ __align__(16) unsigned char st_smem[];
    double* sx = reinterpret_cast<double*>(st_smem);
    double* sb = sx + W * W;
    double* si = sb + W * W;
    double* rcs = si + W * W;
    double* rcd = rcs + W;                   /* W + 1 */
    __shared__ double sh[64];
    const int kt = (T == 32 ? row0 : 0) + blockIdx.y, i0 = blockIdx.x * T, k0 = kt * T, nx = L.nx, nz = L.nz;
    const int done = cg.ctl[0];
    /* every load is under way before anything waits for one */
    double b[PER], a[PER], id[PER], pv[PER], xv[PER];
    const bool step = CG && !cg.first;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int q = threadIdx.x + j * THREADS, li = q % W, lk = q / W, i = i0 - HALO + li, k = k0 - HALO + lk;
        b[j] = a[j] = id[j] = pv[j] = xv[j] = 0.0;
        if (q < W * W && i >= 0 && i < nx && k >= 0 && k < nz) {
            const size_t p = (size_t)k * nx + i;
            b[j] = CG ? cg.rin[p] : L.b[p];
            if (SMOOTH) id[j] = L.id[p];
            if (step) {
                a[j] = cg.ap[p];
                if (li >= HALO && li < HALO + T && lk >= HALO && lk < HALO + T) { pv[j] = cg.p[p]; xv[j] = cg.x[p]; }
            }
        }
    }
    double c1 = 0.0, c2 = 0.0;
    if (SMOOTH && threadIdx.x <= W) {
        const int k = k0 - HALO + threadIdx.x;
        c1 = k >= 0 && k < nz ? L.cs[k] : 0.0;
        c2 = k >= 1 && k < nz ? L.cd[k] : 0.0;
    }
    if (done) return;
    if (SMOOTH && threadIdx.x <= W) {
        if (threadIdx.x < W) rcs[threadIdx.x] = c1;
        rcd[threadIdx.x] = c2;
    }
    double alpha = 0.0;
    if (step) {
        double rz, pap;
        st_total2<THREADS>(cg.part_rz, cg.n_rz, cg.part_pap, cg.n_pap, sh, rz, pap);
        alpha = pap != 0.0 ? rz / pap : 0.0;
    }
    double rn = 0.0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int q = threadIdx.x + j * THREADS, li = q % W, lk = q / W, i = i0 - HALO + li, k = k0 - HALO + lk;
        if (q >= W * W) continue;
        if (step) b[j] += -alpha * a[j];
        if (CG && li >= HALO && li < HALO + T && lk >= HALO && lk < HALO + T && i < nx && k < nz) {
            const size_t p = (size_t)k * nx + i;
            rn = fmax(rn, fabs(b[j]));
            cg.rout[p] = b[j];
            cg.x[p] = step ? xv[j] + alpha * pv[j] : 0.0;
        }
        if (SMOOTH) { const int o = st_at<W>(li, lk); sx[o] = 0.0; sb[o] = b[j]; si[o] = id[j]; }
    }
    if (CG) st_partial<true, THREADS>(rn, cg.part_rn, kt * gridDim.x + blockIdx.x, sh);
    if constexpr (SMOOTH) {
        __syncthreads();
        st_half_sweep<W, THREADS, false>(sx, sb, si, rcs, rcd, 0);
        __syncthreads();
        st_half_sweep<W, THREADS, false>(sx, sb, si, rcs, rcd, 1);
        __syncthreads();
        st_half_sweep<W, THREADS, true>(sx, sb, si, rcs, rcd, 0);
        __syncthreads();
        st_half_sweep<W, THREADS, false>(sx, sb, si, rcs, rcd, 1);
        __syncthreads();
        /* The residual b + off - diag x.  A point of the colour updated last
         * has none; one of the other colour was left with diag x = b + off of
         * the neighbours it saw then, so its residual is the change of off
         * since.  In place of that sum, one point around the tile; 0 off the
         * grid and on the Dirichlet row. */
        for (int q = threadIdx.x; q < (T + 2) * (T / 2 + 1); q += THREADS) {
            const int lk = HALO - 1 + q / (T / 2 + 1), par = lk & 1, j = (HALO - 1 + 1 - par) / 2 + q % (T / 2 + 1), o = lk * (W / 2) + j;
            const double* other = sx + W * W / 2;
            const double off = st_off(rcs[lk], rcd[lk], rcd[lk + 1], other[o - 1 + par], other[o + par], other[o - W / 2], other[o + W / 2]);
            sb[o] = si[o] != 0.0 ? off - sb[o] : 0.0;
        }
        for (int q = threadIdx.x; q < T * T; q += THREADS) {
            const int li = q % T, lk = q / T, i = i0 + li, k = k0 + lk;
            if (i < nx && k < nz) L.x[(size_t)k * nx + i] = sx[st_at<W>(li + HALO, lk + HALO)];
        }
        __syncthreads();
        for (int q = threadIdx.x; q < (T / 2) * (T / 2); q += THREADS) {
            const int li = 2 * (q % (T / 2)), lk = 2 * (q / (T / 2)), i = i0 + li, k = k0 + lk;
            if (i >= nx || k >= nz) continue;
            double s = 0.0;
            if (k > 0) {
                const double* r = sb + (lk + HALO) * (W / 2) + (li + HALO) / 2;      /* colour 0, an even row */
                s = r[0] + 0.25 * ((r[-W / 2 - 1] + r[-W / 2]) + (r[W / 2 - 1] + r[W / 2]));
            }
            Lc.b[(size_t)(k / 2) * Lc.nx + i / 2] = 0.25 * s;
        }
    }
}

/* Ascent on level L: x += bilinear prolongation of the coarser level, then
 * two black-red sweeps, into xo.  CG: level 0, b = the CG residual, and the
 * tile's share of r.z.  SMOOTH = false: the dot product alone (xo is there). */
template <int T, bool CG, bool SMOOTH>
__global__ void __launch_bounds__(StTile<T>::THREADS) k_st_up(StLevel L, StLevel Lc, const int* __restrict__ ctl,
                                                              const double* __restrict__ r, double* part_rz, int row0)
{
    constexpr int THREADS = StTile<T>::THREADS, HALO = SMOOTH ? 4 : 0, W = T + 2 * HALO;
    constexpr int PER = (W * W + THREADS - 1) / THREADS;
    const int done = ctl[0];
    extern __shared__ __align__(16) unsigned char st_smem[];
    double* sx = reinterpret_cast<double*>(st_smem);
    double* sb = sx + W * W;
    double* si = sb + W * W;
    double* rcs = si + W * W;
    double* rcd = rcs + W;                   /* W + 1 */
    __shared__ double sh[32];
    const int kt = (T == 32 ? row0 : 0) + blockIdx.y, i0 = blockIdx.x * T, k0 = kt * T, nx = L.nx, nz = L.nz;
    const double* bsrc = CG ? r : L.b;
    if constexpr (SMOOTH) {
        /* only the colour the first half-sweep reads needs its value */
        double x[PER], b[PER], id[PER], c[PER][4];
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int q = threadIdx.x + j * THREADS, li = q % W, lk = q / W, i = i0 - HALO + li, k = k0 - HALO + lk;
            x[j] = b[j] = id[j] = c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0;
            if (q < W * W && i >= 0 && i < nx && k > 0 && k < nz) {
                const size_t p = (size_t)k * nx + i;
                if (((li + lk) & 1) == 0) {
                    const int I0 = i / 2, K0 = k / 2, I1 = (i & 1) ? I0 + 1 : I0, K1 = (k & 1) ? K0 + 1 : K0;
                    const double* c0 = Lc.xo + (size_t)K0 * Lc.nx;
                    const double* c1 = Lc.xo + (size_t)K1 * Lc.nx;
                    x[j] = L.x[p];
                    c[j][0] = c0[I0]; c[j][1] = c0[I1]; c[j][2] = c1[I0]; c[j][3] = c1[I1];
                }
                b[j] = bsrc[p];
                id[j] = L.id[p];
            }
        }
        double r1 = 0.0, r2 = 0.0;
        if (threadIdx.x <= W) {
            const int k = k0 - HALO + threadIdx.x;
            r1 = k >= 0 && k < nz ? L.cs[k] : 0.0;
            r2 = k >= 1 && k < nz ? L.cd[k] : 0.0;
        }
        if (done) return;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int q = threadIdx.x + j * THREADS, o = st_at<W>(q % W, q / W);
            if (q < W * W) { sx[o] = x[j] + 0.25 * ((c[j][0] + c[j][1]) + (c[j][2] + c[j][3])); sb[o] = b[j]; si[o] = id[j]; }
        }
        if (threadIdx.x <= W) {
            if (threadIdx.x < W) rcs[threadIdx.x] = r1;
            rcd[threadIdx.x] = r2;
        }
        __syncthreads();
        for (int s = 0; s < 4; s++) {
            st_half_sweep<W, THREADS, false>(sx, sb, si, rcs, rcd, 1 - (s & 1));
            __syncthreads();
        }
    }
    if (!SMOOTH && done) return;
    double rz = 0.0;
    for (int q = threadIdx.x; q < T * T; q += THREADS) {
        const int li = q % T, lk = q / T, i = i0 + li, k = k0 + lk;
        if (i >= nx || k >= nz) continue;
        const size_t p = (size_t)k * nx + i;
        const int o = SMOOTH ? st_at<W>(li + HALO, lk + HALO) : 0;
        const double x = SMOOTH ? sx[o] : L.xo[p];
        if (SMOOTH) L.xo[p] = x;
        if (CG) rz += (SMOOTH ? sb[o] : r[p]) * x;
    }
    if (CG) st_partial<false, THREADS>(rz, part_rz, kt * gridDim.x + blockIdx.x, sh);
}

/* p = z + beta p (into the other buffer: neighbours read the old one), Ap and
 * the block's share of p.Ap */
__global__ void __launch_bounds__(256) k_st_direction(StLevel L, const int* __restrict__ ctl, const double* __restrict__ z,
                                                      const double* __restrict__ pold, double* __restrict__ pnew,
                                                      double* __restrict__ ap, const double* part_rz,
                                                      const double* part_rz_old, int n_rz, int first_possible,
                                                      double* part_pap)
{
    __shared__ double sh[64];
    const int done = ctl[0];
    const bool first = first_possible && ctl[1] == 0;
    const int nx = L.nx, nz = L.nz, n = nx * nz;
    double beta = 0.0, s = 0.0;
    for (int p = blockIdx.x * 256 + threadIdx.x, turn = 0; p < n || turn == 0; p += gridDim.x * 256, turn++) {
        /* the loads of a thread's first point are under way while the dot
         * products are reduced; a missing neighbour reads the point itself
         * with a zero coefficient */
        const bool on = p < n;
        const int pc = on ? p : 0, i = pc % nx, k = pc / nx;
        const int pd = k > 1 ? pc - nx : pc, pu = k + 1 < nz ? pc + nx : pc, pl = i > 0 ? pc - 1 : pc, pr = i + 1 < nx ? pc + 1 : pc;
        const double zc = z[pc], zd = z[pd], zu = z[pu], zl = z[pl], zr = z[pr];
        const double oc = pold[pc], od = pold[pd], ou = pold[pu], ol = pold[pl], orr = pold[pr];
        const double cs = L.cs[k], cd = L.cd[k], cu = L.cd[k + 1], dg = L.diag[pc];
        if (turn == 0) {
            if (done) return;
            if (!first) {
                double rz, old;
                st_total2<256>(part_rz, n_rz, part_rz_old, n_rz, sh, rz, old);
                beta = old != 0.0 ? rz / old : 0.0;
            }
        }
        if (!on) break;
        auto dir = [&](double zz, double oo) { return first ? zz : zz + beta * oo; };
        const double c = dir(zc, oc);
        double y = 0.0;
        if (k > 0) {
            double off = 0.0;
            if (k > 1) off += cd * dir(zd, od);
            if (k + 1 < nz) off += cu * dir(zu, ou);
            if (i > 0) off += cs * dir(zl, ol);
            if (i + 1 < nx) off += cs * dir(zr, orr);
            y = dg * c - off;
        }
        pnew[p] = c;
        ap[p] = y;
        s += c * y;
    }
    st_partial<false, 256>(s, part_pap, blockIdx.x, sh);
}

/* the stopping rule on the residual the descent just left: max |r| <= tol
 * max |rhs|, or the iteration limit; a zero right-hand side is done at once */
template <int THREADS>
__device__ bool st_stop(int* ctl, double* scal, const double* part_rn, int np, int first, double* sh)
{
    const double rn = st_total<true, THREADS>(part_rn, np, sh);
    bool done;
    if (first) done = rn == 0.0;
    else done = rn <= scal[0] * scal[1] || ctl[1] + 1 >= ctl[2];
    __syncthreads();                         /* every thread has read ctl and scal */
    if (threadIdx.x == 0) {
        if (first) scal[1] = rn;
        else ctl[1] += 1;
        if (done) ctl[0] = 1;
    }
    return done;
}

struct StTail { StLevel L[ST_MAX_LEVELS]; int l0, nlev, use_op; };

/* A level in the tail's shared memory: each array as two colour halves (entry
 * j of row k of colour c is column 2 j + ((k + c) & 1)), rows of `hw` entries
 * and a zero, which stands for the missing neighbour of either side; x has a
 * zero row above the grid.  An entry past the last column has a zero
 * reciprocal diagonal and stays 0. */
struct StShared { int nx, nz, hw, ph, half, halfx; unsigned mag; int x, b, id, o, cs, cd; };

/* Offsets of the tail's levels.  What a linearisation fixes (id, cs, cd) comes
 * first, in one piece that k_st_coarse_rest lays out in device memory once and
 * the tail copies with loads that do not wait for each other; the working
 * arrays follow.  Returns the length of that piece (even); *all = the whole. */
__host__ __device__ inline int st_tail_layout(const StLevel* L, int l0, int nlev, StShared* S, int* all)
{
    int at = 0;
    for (int l = l0; l < nlev; l++) {
        StShared& v = S[l];
        v.nx = L[l].nx; v.nz = L[l].nz; v.hw = (v.nx + 1) / 2; v.ph = v.hw + 1;
        v.half = v.ph * v.nz; v.halfx = v.ph * (v.nz + 1);
        v.mag = 0xffffffffu / (unsigned)v.hw + 1u;
        v.id = at; v.cs = v.id + 2 * v.half; v.cd = v.cs + v.nz;
        at = v.cd + v.nz + 1;
    }
    at += at & 1;
    const int image = at;
    for (int l = l0; l < nlev; l++) {
        StShared& v = S[l];
        v.x = at; v.b = v.x + 2 * v.halfx; v.o = v.b + 2 * v.half;
        at = v.o + v.half;
    }
    *all = at;
    return image;
}
/* entry of column i, row k in an array whose colour halves are `half` apart */
__device__ __forceinline__ int st_entry(const StShared& L, int half, int i, int k) { return ((i + k) & 1) * half + k * L.ph + (i >> 1); }

__device__ __forceinline__ void st_sync(bool one) { if (one) __syncwarp(); else __syncthreads(); }

/* one half-sweep of a level by `nth` threads; KEEP: keep the neighbour sums */
template <bool KEEP>
__device__ __forceinline__ void st_shared_half(double* m, const StShared& L, int colour, int th, int nth)
{
    const int n = L.hw * (L.nz - 1);
    double* x = m + L.x + colour * L.halfx;
    const double* other = m + L.x + (1 - colour) * L.halfx;
    const double* b = m + L.b + colour * L.half;
    const double* id = m + L.id + colour * L.half;
    for (int q = th; q < n; q += nth) {
        const int kk = (int)__umulhi((unsigned)q, L.mag), k = kk + 1, par = (k + colour) & 1;
        const int p = k * L.ph + q - kk * L.hw;
        const double off = st_off(m[L.cs + k], m[L.cd + k], m[L.cd + k + 1], other[p - 1 + par], other[p + par],
                                  other[p - L.ph], other[p + L.ph]);
        x[p] = (b[p] + off) * id[p];
        if (KEEP) m[L.o + p] = off;
    }
}
__device__ __forceinline__ void st_shared_down(double* m, const StShared L, const StShared Lc, int th, int nth, bool one)
{
    st_shared_half<false>(m, L, 0, th, nth); st_sync(one);
    st_shared_half<false>(m, L, 1, th, nth); st_sync(one);
    st_shared_half<true>(m, L, 0, th, nth); st_sync(one);
    st_shared_half<false>(m, L, 1, th, nth); st_sync(one);
    /* residual of colour 0 and restriction, as in k_st_down */
    {
        const double* other = m + L.x + L.halfx;
        for (int q = th; q < L.hw * (L.nz - 1); q += nth) {
            const int kk = (int)__umulhi((unsigned)q, L.mag), k = kk + 1, par = k & 1;
            const int p = k * L.ph + q - kk * L.hw;
            const double off = st_off(m[L.cs + k], m[L.cd + k], m[L.cd + k + 1], other[p - 1 + par], other[p + par],
                                      other[p - L.ph], other[p + L.ph]);
            m[L.o + p] = m[L.id + p] != 0.0 ? off - m[L.o + p] : 0.0;
        }
    }
    st_sync(one);
    const unsigned magc = 0xffffffffu / (unsigned)Lc.nx + 1u;
    for (int q = th; q < Lc.nx * (Lc.nz - 1); q += nth) {
        const int kk = (int)__umulhi((unsigned)q, magc), K = kk + 1, I = q - kk * Lc.nx;
        const double* r = m + L.o + 2 * K * L.ph + I;
        double s = r[0], c = 0.0;
        c += r[-L.ph - 1] + r[-L.ph];                    /* column -1 reads the row's zero */
        if (K + 1 < Lc.nz) c += r[L.ph - 1] + r[L.ph];
        m[Lc.b + st_entry(Lc, Lc.half, I, K)] = 0.25 * (s + 0.25 * c);
    }
    st_sync(one);
}
__device__ __forceinline__ void st_shared_up(double* m, const StShared L, const StShared Lc, int th, int nth, bool one)
{
    const double* c = m + Lc.x;
    for (int q = th; q < L.hw * (L.nz - 1); q += nth) {
        const int kk = (int)__umulhi((unsigned)q, L.mag), k = kk + 1, j = q - kk * L.hw, K = k >> 1;
        if (k & 1) {
            if (j < L.hw - 1)
                m[L.x + k * L.ph + j] += 0.25 * ((c[st_entry(Lc, Lc.halfx, j, K)] + c[st_entry(Lc, Lc.halfx, j + 1, K)]) +
                                                 (c[st_entry(Lc, Lc.halfx, j, K + 1)] + c[st_entry(Lc, Lc.halfx, j + 1, K + 1)]));
        } else m[L.x + k * L.ph + j] += c[st_entry(Lc, Lc.halfx, j, K)];
    }
    st_sync(one);
    st_shared_half<false>(m, L, 1, th, nth); st_sync(one);
    st_shared_half<false>(m, L, 0, th, nth); st_sync(one);
    st_shared_half<false>(m, L, 1, th, nth); st_sync(one);
    st_shared_half<false>(m, L, 0, th, nth); st_sync(one);
}

/* Levels l0 .. nlev-1 of the V-cycle in one block's shared memory, and
 * before them the stopping rule.  b of level l0 comes from device memory and
 * its x goes back there.  The coarsest level's 40 + 40 symmetric sweeps are
 * a fixed linear map of b: one matrix-vector product where it is small (its
 * matrix is made once per linearisation by k_st_coarse_rest), sweeps otherwise.
 * What bounds it is the chain of some 50 phases, each a shared-memory round
 * trip, a few dependent FP64 operations and a barrier; the levels of a few
 * dozen points run on one warp, whose barrier costs next to nothing. */
__global__ void __launch_bounds__(ST_TAIL_THREADS) k_st_tail(const __grid_constant__ StTail t, int* ctl, double* scal,
                                                             const double* part_rn, int np, int first,
                                                             const double* __restrict__ b0, const double* __restrict__ op,
                                                             const double* __restrict__ image)
{
    constexpr int NT = ST_TAIL_THREADS;
    __shared__ double sh[32];
    __shared__ StShared lv[ST_MAX_LEVELS];
    __shared__ double sop[ST_OP_MAX * ST_OP_MAX];
    __shared__ int len[2];
    extern __shared__ __align__(16) unsigned char st_smem[];
    double* m = reinterpret_cast<double*>(st_smem);
    const int th = threadIdx.x, last = t.nlev - 1;
    const int done = ctl[0];
    if (th == 0) len[0] = st_tail_layout(t.L, t.l0, t.nlev, lv, &len[1]);
    const int nu = t.L[last].nx * (t.L[last].nz - 1);
    if (t.use_op) for (int q = th; q < nu * nu; q += NT) sop[q] = op[q];
    __syncthreads();
    {
        const int n16 = len[0] / 2;
        const double2* src = reinterpret_cast<const double2*>(image);
        double2* dst = reinterpret_cast<double2*>(m);
        for (int q0 = th; q0 < n16; q0 += 8 * NT) {
            double2 v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) if (q0 + j * NT < n16) v[j] = src[q0 + j * NT];
#pragma unroll
            for (int j = 0; j < 8; j++) if (q0 + j * NT < n16) dst[q0 + j * NT] = v[j];
        }
        for (int q = len[0] + th; q < len[1]; q += NT) m[q] = 0.0;
    }
    __syncthreads();
    {
        const StShared S = lv[t.l0];
        const int n = S.nx * S.nz;
        const unsigned mag = 0xffffffffu / (unsigned)S.nx + 1u;
#pragma unroll 4
        for (int p = S.nx + th; p < n; p += NT) {
            const int k = (int)__umulhi((unsigned)p, mag);
            m[S.b + st_entry(S, S.half, p - k * S.nx, k)] = b0[p];
        }
    }
    if (done) return;
    if (st_stop<NT>(ctl, scal, part_rn, np, first, sh)) return;
    __syncthreads();
    int lw = t.l0;                           /* first level one warp runs alone */
    while (lw < last && lv[lw].hw * (lv[lw].nz - 1) > ST_WARP_POINTS) lw++;
    for (int l = t.l0; l < lw; l++) st_shared_down(m, lv[l], lv[l + 1], th, NT, false);
    const StShared B = lv[last];
    if (!t.use_op && lw == last) {           /* a coarsest level of many unknowns: sweeps by the block */
        for (int j = 0; j < 160; j++) {
            st_shared_half<false>(m, B, j < 80 ? (j & 1) : 1 - (j & 1), th, NT);
            __syncthreads();
        }
    } else if (th < 32) {
        for (int l = lw; l < last; l++) st_shared_down(m, lv[l], lv[l + 1], th, 32, true);
        if (t.use_op) {
            if (th < nu) {
                double s = 0.0;
                for (int j = 0, k = 1, i = 0; j < nu; j++) {
                    s = fma(sop[j * nu + th], m[B.b + st_entry(B, B.half, i, k)], s);
                    if (++i == B.nx) { i = 0; k++; }
                }
                m[B.x + st_entry(B, B.halfx, th % B.nx, 1 + th / B.nx)] = s;
            }
            __syncwarp();
        } else {
            for (int j = 0; j < 160; j++) {
                st_shared_half<false>(m, B, j < 80 ? (j & 1) : 1 - (j & 1), th, 32);
                __syncwarp();
            }
        }
        for (int l = last - 1; l >= lw; l--) st_shared_up(m, lv[l], lv[l + 1], th, 32, true);
    }
    __syncthreads();
    for (int l = lw - 1; l >= t.l0; l--) st_shared_up(m, lv[l], lv[l + 1], th, NT, false);
    const StShared S = lv[t.l0];
    double* out = t.L[t.l0].xo;
    const unsigned mag = 0xffffffffu / (unsigned)S.nx + 1u;
#pragma unroll 4
    for (int p = th; p < S.nx * S.nz; p += NT) {
        const int k = (int)__umulhi((unsigned)p, mag);
        out[p] = m[S.x + st_entry(S, S.halfx, p - k * S.nx, k)];
    }
}

/* The same steps where no level fits one block (a level of 3 rows or columns
 * and thousands of the other): the stopping rule, then the coarsest level's
 * half-sweeps, one launch each. */
__global__ void __launch_bounds__(ST_TAIL_THREADS) k_st_check(int* ctl, double* scal, const double* part_rn, int np, int first)
{
    if (ctl[0]) return;
    __shared__ double sh[32];
    st_stop<ST_TAIL_THREADS>(ctl, scal, part_rn, np, first, sh);
}
__global__ void k_st_rbgs(StLevel L, const int* __restrict__ ctl, const double* __restrict__ b, int colour, int from_zero)
{
    const int p = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + colour;
    if (p >= L.nx * L.nz || ctl[0]) return;
    const int i = p % L.nx, k = p / L.nx;
    if (k == 0) return;
    double off = 0.0;
    if (!from_zero) {                        /* the first half-sweep finds the last cycle's values */
        if (k > 1) off += L.cd[k] * L.xo[p - L.nx];
        if (k + 1 < L.nz) off += L.cd[k + 1] * L.xo[p + L.nx];
        if (i > 0) off += L.cs[k] * L.xo[p - 1];
        if (i + 1 < L.nx) off += L.cs[k] * L.xo[p + 1];
    }
    L.xo[p] = (b[p] + off) / L.diag[p];
}

/* ---- coefficients -------------------------------------------------------- */
__global__ void k_st_begin(int* ctl, double* scal, double tol, int max_it) { ctl[0] = 0; ctl[1] = 0; ctl[2] = max_it; scal[0] = tol; }

/* a level's row coefficients: row k of level l has the diffusivity of row k 2^l */
__global__ void k_st_rows(StLevel L, int l, int nz_agar, double d_agar, double d_col)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > L.nz) return;
    const double ih2 = 1.0 / (L.h * L.h);
    const double d = ((long)k << l) < nz_agar ? d_agar : d_col, dm = ((long)(k - 1) << l) < nz_agar ? d_agar : d_col;
    if (k < L.nz) L.cs[k] = d * ih2;
    L.cd[k] = k >= 1 && k < L.nz ? face_d(d, dm) * ih2 : 0.0;
}
/* sig + the coefficients of the point's faces (below, above, sides) */
__device__ __forceinline__ double st_diag(const StLevel& L, int i, int k, double sig)
{
    double d = sig;
    d += L.cd[k];
    if (k + 1 < L.nz) d += L.cd[k + 1];
    if (i > 0) d += L.cs[k];
    if (i + 1 < L.nx) d += L.cs[k];
    return d;
}
/* coarse diagonal term: weighted average of the fine one over the
 * restriction stencil; and the diagonal */
__device__ void st_coarse_point(const StLevel& Lc, const StLevel& Lf, int p)
{
    const int I = p % Lc.nx, K = p / Lc.nx;
    double s = 0.0, ws = 0.0;
    for (int dk = -1; dk <= 1; dk++) {
        int k = 2 * K + dk;
        if (k < 0 || k >= Lf.nz) continue;
        double wk = dk == 0 ? 1.0 : 0.5;
        for (int di = -1; di <= 1; di++) {
            int i = 2 * I + di;
            if (i < 0 || i >= Lf.nx) continue;
            double wi = di == 0 ? 1.0 : 0.5;
            s += wi * wk * Lf.sig[(size_t)k * Lf.nx + i];
            ws += wi * wk;
        }
    }
    const double sig = s / ws;
    Lc.sig[p] = sig;
    const double diag = K > 0 ? st_diag(Lc, I, K, sig) : 1.0;
    Lc.diag[p] = diag;
    Lc.id[p] = K > 0 ? 1.0 / diag : 0.0;
}
__global__ void k_st_coarse_coeffs(StLevel Lc, StLevel Lf)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < Lc.nx * Lc.nz) st_coarse_point(Lc, Lf, p);
}
/* levels l0 .. nlev-1 one after another in one block; the tail's image of
 * them (st_tail_layout); then, where the
 * coarsest level has at most ST_OP_MAX unknowns, the matrix of its 40 + 40
 * sweeps: warp j runs them on the j-th unit vector */
__global__ void __launch_bounds__(1024) k_st_coarse_rest(const __grid_constant__ StTail t, int tail, double* op, double* image)
{
    __shared__ StShared lv[ST_MAX_LEVELS];
    __shared__ int all;
    if (threadIdx.x == 0) st_tail_layout(t.L, tail, t.nlev, lv, &all);
    for (int l = t.l0; l < t.nlev; l++) {
        for (int p = threadIdx.x; p < t.L[l].nx * t.L[l].nz; p += blockDim.x) st_coarse_point(t.L[l], t.L[l - 1], p);
        __syncthreads();
    }
    __syncthreads();
    for (int l = tail; l < t.nlev; l++) {
        const StShared S = lv[l];
        const StLevel& L = t.L[l];
        for (int p = threadIdx.x; p < 2 * S.half; p += blockDim.x) {
            const int c = p >= S.half, k = (p - c * S.half) / S.ph, j = p - c * S.half - k * S.ph, i = 2 * j + ((k + c) & 1);
            image[S.id + p] = j < S.hw && i < S.nx ? L.id[k * S.nx + i] : 0.0;
        }
        for (int k = threadIdx.x; k <= S.nz; k += blockDim.x) { if (k < S.nz) image[S.cs + k] = L.cs[k]; image[S.cd + k] = L.cd[k]; }
    }
    if (!t.use_op) return;
    const StLevel& L = t.L[t.nlev - 1];
    const int nx = L.nx, nu = nx * (L.nz - 1);
    const int j = threadIdx.x >> 5, u = threadIdx.x & 31;
    if (j >= nu) return;                     /* whole warp */
    const int p = nx + (u < nu ? u : 0), i = p % nx, k = p / nx;
    const bool on = u < nu;
    const double id = on ? L.id[p] : 0.0;
    const double cs = L.cs[k], cdn = k > 1 ? L.cd[k] : 0.0, cup = k + 1 < L.nz ? L.cd[k + 1] : 0.0;
    const double cl = i > 0 ? cs : 0.0, cr = i + 1 < nx ? cs : 0.0;
    const double b = u == j ? 1.0 : 0.0;
    const int colour = (nx + u) & 1;
    double x = 0.0;
    for (int s = 0; s < 160; s++) {
        /* 40 x (0, 1), then 40 x (1, 0) */
        const int c = s < 80 ? (s & 1) : 1 - (s & 1);
        double off = cdn * __shfl_sync(0xffffffffu, x, k > 1 ? u - nx : u);
        off += cup * __shfl_sync(0xffffffffu, x, (u + nx) & 31);
        off += cl * __shfl_sync(0xffffffffu, x, i > 0 ? u - 1 : u);
        off += cr * __shfl_sync(0xffffffffu, x, (u + 1) & 31);
        if (on && colour == c) x = (b + off) * id;
    }
    if (on) op[j * nu + u] = x;
}

/* ---- problem-specific kernels ------------------------------------------ */
/* C = c0, and the deposition of the cells' weighted L*R (one thread per grid
 * point; bcg_steady_set_cells sorted the cells by point, so the sum order is
 * fixed and a point's entries lie side by side) */
__global__ void k_st_deposit(int n, double h, double c0, const int* __restrict__ start, const int* __restrict__ order,
                             const double* __restrict__ cell, const double* __restrict__ w, double* __restrict__ q,
                             double* __restrict__ C)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    double s = 0.0;
    const int e = start[p + 1];
#pragma unroll 4
    for (int j = start[p]; j < e; j++) {
        const int c = order[j];
        const double2 lr = *reinterpret_cast<const double2*>(cell + 4 * (size_t)c + 2);
        s += w[c] * lr.x * lr.y;
    }
    q[p] = s / (h * h);
    C[p] = c0;
}

/* F(C) (the Newton right-hand side), the linearised diagonal, and the
 * block's max |F| */
__global__ void __launch_bounds__(256) k_st_newton_rhs(StLevel L, const double* __restrict__ C, const double* __restrict__ q,
                                                       double vmax, double km, double* __restrict__ F, double* part)
{
    __shared__ double sh[32];
    const int p = blockIdx.x * 256 + threadIdx.x;
    double f = 0.0;
    if (p < L.nx * L.nz) {
        const int i = p % L.nx, k = p / L.nx;
        double sig = 0.0, diag = 1.0;
        if (k > 0) {
            const double cs = L.cs[k], c = C[p];
            double flux = 0.0;
            flux += L.cd[k] * (C[p - L.nx] - c);
            if (k + 1 < L.nz) flux += L.cd[k + 1] * (C[p + L.nx] - c);
            if (i > 0) flux += cs * (C[p - 1] - c);
            if (i + 1 < L.nx) flux += cs * (C[p + 1] - c);
            f = flux - q[p] * vmax * c / (km + c);
            sig = q[p] * vmax * km / ((km + c) * (km + c));
            diag = st_diag(L, i, k, sig);
        }
        F[p] = f;
        L.sig[p] = sig;
        L.diag[p] = diag;
        L.id[p] = k > 0 ? 1.0 / diag : 0.0;
    }
    st_partial<true, 256>(fabs(f), part, blockIdx.x, sh);
}

/* dst = -src, zero on the Dirichlet row */
__global__ void k_st_neg(int n, int nx, const double* __restrict__ src, double* __restrict__ dst)
{ int p = blockIdx.x * blockDim.x + threadIdx.x; if (p < n) dst[p] = p < nx ? 0.0 : -src[p]; }
__global__ void k_st_add(int n, const double* __restrict__ x, double* __restrict__ y) { int p = blockIdx.x * blockDim.x + threadIdx.x; if (p < n) y[p] += x[p]; }

/* gradients: per point contributions to dL/d(d_agar, d_colony, vmax, km),
 * reduced per block in fixed order; and dL/dw per cell */
__global__ void k_st_grad_part(StLevel L, int nz_agar, double d_agar, double d_col, const double* __restrict__ C,
                               const double* __restrict__ q, const double* __restrict__ lam, double vmax, double km,
                               double* gpart)
{
    __shared__ double sh[4][256];
    double g[4] = {0, 0, 0, 0};
    const double ih2 = 1.0 / (L.h * L.h);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < L.nx * L.nz; p += gridDim.x * blockDim.x) {
        int i = p % L.nx, k = p / L.nx;
        if (k == 0) continue;
        const double lp = lam[p], c = C[p];
        /* dF_p/d(d) summed over p's faces */
        double dfa = 0.0, dfc = 0.0;
        auto face = [&](int pn, int kn) {
            const bool pa = k < nz_agar, na = kn < nz_agar;
            const double dc = C[pn] - c;
            if (pa && na) dfa += dc * ih2;
            else if (!pa && !na) dfc += dc * ih2;
            else {
                /* harmonic mean 2 a b / (a + b): d/da = 2 b^2 / (a + b)^2 */
                const double s = d_agar + d_col;
                dfa += 2.0 * d_col * d_col / (s * s) * dc * ih2;
                dfc += 2.0 * d_agar * d_agar / (s * s) * dc * ih2;
            }
        };
        face(p - L.nx, k - 1);
        if (k + 1 < L.nz) face(p + L.nx, k + 1);
        if (i > 0) face(p - 1, k);
        if (i + 1 < L.nx) face(p + 1, k);
        /* dL/dtheta = -lambda . dF/dtheta */
        g[0] -= lp * dfa;
        g[1] -= lp * dfc;
        g[2] += lp * q[p] * c / (km + c);
        g[3] -= lp * q[p] * vmax * c / ((km + c) * (km + c));
    }
    for (int j = 0; j < 4; j++) sh[j][threadIdx.x] = g[j];
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) for (int j = 0; j < 4; j++) sh[j][threadIdx.x] += sh[j][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) for (int j = 0; j < 4; j++) gpart[4 * blockIdx.x + j] = sh[j][0];
}

__global__ void k_st_grad_w(int ncell, double h, const double* __restrict__ cell, const int* __restrict__ cell_pt,
                            const double* __restrict__ C, const double* __restrict__ lam, double vmax, double km,
                            double* __restrict__ gw)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    int p = cell_pt[c];
    if (p < 0) { gw[c] = 0.0; return; }
    const double cc = C[p];
    /* dF_p/dw_c = -(L R / h^2) vmax C / (km + C) */
    gw[c] = lam[p] * cell[4 * c + 2] * cell[4 * c + 3] / (h * h) * vmax * cc / (km + cc);
}

/* ---- host side ---------------------------------------------------------- */
static unsigned nblk(int n) { return (unsigned)((n + 255) / 256); }

/* Tile side: 32 recomputes least (a 44 x 44 box for 1024 points), 16 keeps
 * four times the blocks busy.  32 from the size where its tiles still fill
 * half the SMs. */
static int st_tile(const StLevel& L)
{
    return ((L.nx + 31) / 32) * ((L.nz + 31) / 32) >= 74 ? 32 : 16;
}
/* the tiles' rows from row0 on that one launch takes: a grid has at most 65535
 * blocks in y, fewer than the tallest levels have rows of tiles (of 32, since a
 * level of tiles of 16 has at most 148) */
#define ST_GRID_ROWS 65535
static int st_tile_rows(const StLevel& L, int T) { return (L.nz + T - 1) / T; }
static dim3 st_tiles(const StLevel& L, int T, int row0)
{
    const int rows = st_tile_rows(L, T) - row0;
    return dim3((unsigned)((L.nx + T - 1) / T), (unsigned)(rows < ST_GRID_ROWS ? rows : ST_GRID_ROWS));
}
static size_t st_down_smem(int T) { const int W = T + 12; return sizeof(double) * (3 * W * W + 2 * W + 1); }
static size_t st_up_smem(int T) { const int W = T + 8; return sizeof(double) * (3 * W * W + 2 * W + 1); }
static size_t st_tail_smem(const bcg_steady* s)
{
    StShared S[ST_MAX_LEVELS];
    int all = 0;
    st_tail_layout(s->L, s->tail, s->nlev, S, &all);
    return sizeof(double) * (size_t)all;
}
static int st_coarsest(const bcg_steady* s) { const StLevel& L = s->L[s->nlev - 1]; return L.nx * (L.nz - 1); }

template <bool CG, bool SMOOTH>
static void st_down(bcg_steady* s, int l, const StCg& cg)
{
    const StLevel &L = s->L[l], &Lc = s->L[l + 1 < s->nlev ? l + 1 : l];
    const int T = st_tile(L);
    for (int r0 = 0; r0 < st_tile_rows(L, T); r0 += ST_GRID_ROWS) {
        if (T == 32) k_st_down<32, CG, SMOOTH><<<st_tiles(L, 32, r0), 512, SMOOTH ? st_down_smem(32) : 0, s->stream>>>(L, Lc, cg, r0);
        else k_st_down<16, CG, SMOOTH><<<st_tiles(L, 16, 0), 256, SMOOTH ? st_down_smem(16) : 0, s->stream>>>(L, Lc, cg, 0);
    }
}
template <bool CG, bool SMOOTH>
static void st_up(bcg_steady* s, int l, const double* r, double* part_rz)
{
    const StLevel &L = s->L[l], &Lc = s->L[l + 1 < s->nlev ? l + 1 : l];
    const int T = st_tile(L);
    for (int r0 = 0; r0 < st_tile_rows(L, T); r0 += ST_GRID_ROWS) {
        if (T == 32) k_st_up<32, CG, SMOOTH><<<st_tiles(L, 32, r0), 512, SMOOTH ? st_up_smem(32) : 0, s->stream>>>(L, Lc, s->ctl, r, part_rz, r0);
        else k_st_up<16, CG, SMOOTH><<<st_tiles(L, 16, 0), 256, SMOOTH ? st_up_smem(16) : 0, s->stream>>>(L, Lc, s->ctl, r, part_rz, 0);
    }
}

/* the CG step of iteration `it` (0: the start), the stopping rule and the
 * V-cycle on the new residual, up to z in L[0].xo and the shares of r.z */
static void st_cycle(bcg_steady* s, const double* rhs, int it)
{
    const int cur = it & 1;
    const bool first = it == 0;
    double* r = s->cg_r[cur];
    StCg cg = {s->ctl, first ? rhs : s->cg_r[cur ^ 1], r, s->cg_ap, s->cg_p[cur ^ 1], s->cg_x,
               s->part_rz[cur ^ 1], s->part_pap, s->part_rn, s->nt0, s->ntd, first ? 1 : 0};
    const bool one = s->nlev == 1;
    if (one) st_down<true, false>(s, 0, cg); else st_down<true, true>(s, 0, cg);
    const int down_to = s->tail < s->nlev ? s->tail : s->nlev - 1;
    for (int l = 1; l < down_to; l++) st_down<false, true>(s, l, cg);
    if (s->tail < s->nlev) {
        StTail t;
        memcpy(t.L, s->L, sizeof(t.L));
        t.l0 = s->tail; t.nlev = s->nlev; t.use_op = st_coarsest(s) <= ST_OP_MAX;
        k_st_tail<<<1, ST_TAIL_THREADS, st_tail_smem(s), s->stream>>>(t, s->ctl, s->scal, s->part_rn, s->nt0, first,
                                                                      s->tail == 0 ? r : s->L[s->tail].b, s->op, s->image);
    } else {
        StLevel& L = s->L[s->nlev - 1];
        const double* b = one ? r : L.b;
        const unsigned nb = nblk((L.nx * L.nz + 1) / 2);
        k_st_check<<<1, ST_TAIL_THREADS, 0, s->stream>>>(s->ctl, s->scal, s->part_rn, s->nt0, first);
        for (int j = 0; j < 160; j++)
            k_st_rbgs<<<nb, 256, 0, s->stream>>>(L, s->ctl, b, j < 80 ? (j & 1) : 1 - (j & 1), j == 0);
    }
    for (int l = down_to - 1; l >= 1; l--) st_up<false, true>(s, l, r, nullptr);
    if (one) st_up<true, false>(s, 0, r, s->part_rz[cur]); else st_up<true, true>(s, 0, r, s->part_rz[cur]);
}
/* iteration `it` >= 1: direction, step, stopping rule, next z.  Iterations
 * after the one that stopped do nothing. */
static void st_iteration(bcg_steady* s, int it)
{
    const int cur = it & 1;
    /* the buffers alternate: iteration it reads r, p and r.z of it - 1 */
    k_st_direction<<<s->ntd, 256, 0, s->stream>>>(s->L[0], s->ctl, s->L[0].xo, s->cg_p[cur], s->cg_p[cur ^ 1], s->cg_ap,
                                                  s->part_rz[cur ^ 1], s->part_rz[cur], s->nt0, 1, s->part_pap);
    st_cycle(s, nullptr, it);
}
/* ST_CHUNK iterations, the first of them odd, as one graph launch; plain
 * launches where no graph can be made */
static int st_chunk(bcg_steady* s)
{
    if (!s->graph && !s->graph_off) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            for (int j = 1; j <= ST_CHUNK; j++) st_iteration(s, j);
            e = cudaStreamEndCapture(s->stream, &g);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&s->graph, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) { cudaGetLastError(); s->graph = nullptr; s->graph_off = true; }
    }
    if (s->graph) return st_err(cudaGraphLaunch(s->graph, s->stream));
    for (int j = 1; j <= ST_CHUNK; j++) st_iteration(s, j);
    return st_err(cudaGetLastError());
}

/* solve A x = rhs (A from the current level-0 sig/diag) by PCG to
 * ||r||_inf <= tol * ||rhs||_inf; x in cg_x */
static int st_pcg(bcg_steady* s, const double* rhs, double tol, int max_it, int* iters)
{
    /* coarse diagonals for this linearisation: the large levels on their own,
     * the smaller ones one after another in one block */
    k_st_begin<<<1, 1, 0, s->stream>>>(s->ctl, s->scal, tol, max_it);
    int lr = 1;
    for (; lr < s->nlev && s->L[lr].nx * s->L[lr].nz > ST_TAIL_POINTS; lr++)
        k_st_coarse_coeffs<<<nblk(s->L[lr].nx * s->L[lr].nz), 256, 0, s->stream>>>(s->L[lr], s->L[lr - 1]);
    StTail t;
    memcpy(t.L, s->L, sizeof(t.L));
    t.l0 = lr; t.nlev = s->nlev; t.use_op = s->tail < s->nlev && st_coarsest(s) <= ST_OP_MAX;
    k_st_coarse_rest<<<1, 1024, 0, s->stream>>>(t, s->tail, s->op, s->image);
    st_cycle(s, rhs, 0);
    int rc = st_err(cudaGetLastError());
    volatile int* h = reinterpret_cast<volatile int*>(s->pin);
    for (int done = 0, queue = ST_FIRST; !rc && !done; queue = ST_CHUNK) {
        for (int j = 0; j < queue && !rc; j += ST_CHUNK) rc = st_chunk(s);
        if (rc) break;
        ST_TRY(cudaMemcpyAsync(s->pin, s->ctl, 2 * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
        ST_TRY(cudaStreamSynchronize(s->stream));
        done = h[0];
        *iters = h[1];
    }
    return rc;
}

/* max |F| at C, with F, sig and the diagonal left on the device */
static int st_newton_rhs(bcg_steady* s, double vmax, double km, double* fn)
{
    const int nb = (int)nblk(s->n);
    k_st_newton_rhs<<<nb, 256, 0, s->stream>>>(s->L[0], s->C, s->q, vmax, km, s->F, s->part_rn);
    ST_TRY(cudaGetLastError());
    if (!fn) return BCG_OK;
    ST_TRY(cudaMemcpyAsync(s->pin, s->part_rn, sizeof(double) * nb, cudaMemcpyDeviceToHost, s->stream));
    ST_TRY(cudaStreamSynchronize(s->stream));
    double m = 0.0;
    for (int b = 0; b < nb; b++) m = fmax(m, s->pin[b]);
    *fn = m;
    return BCG_OK;
}

static int st_attributes()
{
    /* set on every creation: attributes belong to the current device */
#define ST_SMEM(k, b) if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(b)) != cudaSuccess) return BCG_E_CUDA
    ST_SMEM((k_st_down<32, true, true>), st_down_smem(32));
    ST_SMEM((k_st_down<32, false, true>), st_down_smem(32));
    ST_SMEM(k_st_tail, 32 * ST_TAIL_POINTS);
#undef ST_SMEM
    return BCG_OK;
}

extern "C" int bcg_steady_create(const bcg_steady_params* p, bcg_steady** out)
{
    if (!p || !out) return BCG_E_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return BCG_E_NO_DEVICE;
    auto pow2p1 = [](int v) { return v >= 3 && (((v - 1) & (v - 2)) == 0); };
    if (!pow2p1(p->nx) || !pow2p1(p->nz) || p->nz_agar < 1 || p->nz_agar > p->nz || !(p->h > 0) || p->max_cells < 0)
        return BCG_E_ARG;
    bcg_steady* s = (bcg_steady*)calloc(1, sizeof(bcg_steady));
    if (!s) return BCG_E_ARG;
    s->P = *p;
    int rc = BCG_OK;
#define ST_ALLOC(ptr, bytes) do { if (!rc) rc = st_err(cudaMalloc((void**)&(ptr), (bytes))); } while (0)
    if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) { free(s); return BCG_E_CUDA; }
    int nx = p->nx, nz = p->nz;
    double h = p->h;
    s->nlev = 0;
    while (s->nlev < ST_MAX_LEVELS) {
        StLevel& L = s->L[s->nlev];
        L.nx = nx; L.nz = nz; L.h = h;
        size_t b = sizeof(double) * (size_t)nx * nz;
        ST_ALLOC(L.x, b); ST_ALLOC(L.xo, b); ST_ALLOC(L.b, b); ST_ALLOC(L.sig, b); ST_ALLOC(L.diag, b); ST_ALLOC(L.id, b);
        ST_ALLOC(L.cs, sizeof(double) * (nz + 1)); ST_ALLOC(L.cd, sizeof(double) * (nz + 1));
        /* the Dirichlet row, which no kernel writes everywhere, is 0 */
        if (!rc) rc = st_err(cudaMemsetAsync(L.xo, 0, b, s->stream));
        s->nlev++;
        if (nx <= 3 || nz <= 3) break;
        nx = (nx + 1) / 2; nz = (nz + 1) / 2; h *= 2;
    }
    s->n = p->nx * p->nz;
    size_t b = sizeof(double) * (size_t)s->n;
    /* the largest set of levels, from the coarsest up, that fits the tail */
    s->tail = s->nlev;
    for (int l = s->nlev - 1, pts = 0; l >= (s->nlev > 1 ? 1 : 0); l--) {
        pts += (s->L[l].nx + 3) * (s->L[l].nz + 1) + s->L[l].nz / 2 + 2;    /* over st_tail_smem / 32 B */
        if (pts > ST_TAIL_POINTS) break;
        s->tail = l;
    }
    {
        const int T = st_tile(s->L[0]);
        s->nt0 = ((p->nx + T - 1) / T) * st_tile_rows(s->L[0], T);
        s->ntd = (int)nblk(s->n) < 592 ? (int)nblk(s->n) : 592;     /* 4 blocks an SM */
    }
    const size_t np = (size_t)(s->nt0 > (int)nblk(s->n) ? s->nt0 : (int)nblk(s->n));
    ST_ALLOC(s->C, b); ST_ALLOC(s->q, b); ST_ALLOC(s->F, b); ST_ALLOC(s->g, b);
    ST_ALLOC(s->cg_x, b); ST_ALLOC(s->cg_ap, b);
    for (int j = 0; j < 2; j++) { ST_ALLOC(s->cg_r[j], b); ST_ALLOC(s->cg_p[j], b); ST_ALLOC(s->part_rz[j], sizeof(double) * np); }
    ST_ALLOC(s->part_rn, sizeof(double) * np);
    ST_ALLOC(s->part_pap, sizeof(double) * np);
    ST_ALLOC(s->scal, sizeof(double) * 16);
    ST_ALLOC(s->ctl, sizeof(int) * 16);
    ST_ALLOC(s->op, sizeof(double) * ST_OP_MAX * ST_OP_MAX);
    ST_ALLOC(s->image, 32 * ST_TAIL_POINTS);
    ST_ALLOC(s->gpart, sizeof(double) * 4 * ST_RED_BLOCKS);
    ST_ALLOC(s->start, sizeof(int) * ((size_t)s->n + 1));
    if (!rc) rc = st_err(cudaMemsetAsync(s->start, 0, sizeof(int) * ((size_t)s->n + 1), s->stream));
    if (!rc) rc = st_err(cudaMallocHost((void**)&s->pin, sizeof(double) * (np > 4 * ST_RED_BLOCKS ? np : 4 * ST_RED_BLOCKS)));
    int mc = p->max_cells > 0 ? p->max_cells : 1;
    ST_ALLOC(s->cell, sizeof(double) * 4 * mc);
    ST_ALLOC(s->cell_pt, sizeof(int) * mc);
    ST_ALLOC(s->w, sizeof(double) * mc);
    ST_ALLOC(s->gw, sizeof(double) * mc);
    ST_ALLOC(s->order, sizeof(int) * mc);
    if (!rc) rc = st_attributes();
#undef ST_ALLOC
    if (rc) { bcg_steady_destroy(s); return rc; }
    *out = s;
    return BCG_OK;
}

extern "C" int bcg_steady_destroy(bcg_steady* s)
{
    if (!s) return BCG_OK;
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (int l = 0; l < s->nlev; l++) { 
        StLevel& L = s->L[l];
        void* lv[] = {L.x, L.xo, L.b, L.sig, L.diag, L.id, L.cs, L.cd};
        for (void* q : lv) if (q) cudaFree(q);
    }
    void* ptrs[] = {s->C, s->q, s->F, s->g, s->cg_x, s->cg_r[0], s->cg_r[1], s->cg_p[0], s->cg_p[1], s->cg_ap, s->part_rn,
                    s->part_rz[0], s->part_rz[1], s->part_pap, s->scal, s->ctl, s->op, s->image, s->gpart,
                    s->cell, s->cell_pt, s->w, s->gw, s->start, s->order};
    for (void* q : ptrs) if (q) cudaFree(q);
    if (s->graph) cudaGraphExecDestroy(s->graph);
    if (s->pin) cudaFreeHost(s->pin);
    if (s->stream) cudaStreamDestroy(s->stream);
    free(s);
    return BCG_OK;
}

/* cell centres (x from the grid's left edge, z from the agar bottom),
 * lengths and radii: 4 doubles per cell */
extern "C" int bcg_steady_set_cells(bcg_steady* s, const double* xzlr, int ncell)
{
    if (!s || ncell < 0 || ncell > s->P.max_cells || (ncell > 0 && !xzlr)) return BCG_E_ARG;
    s->ncell = ncell;
    s->solved = false;
    /* the cells of each grid point, in the order given (a counting sort) */
    const int nx = s->P.nx, nz = s->P.nz, n = s->n;
    std::vector<int> pt(ncell), start((size_t)n + 1, 0), order(ncell);
    for (int c = 0; c < ncell; c++) {
        long i = lround(xzlr[4 * c] / s->P.h), k = lround(xzlr[4 * c + 1] / s->P.h);
        pt[c] = (i >= 0 && i < nx && k >= s->P.nz_agar && k < nz) ? (int)(k * nx + i) : -1;
        if (pt[c] >= 0) start[pt[c] + 1]++;
    }
    for (int p = 0; p < n; p++) start[p + 1] += start[p];
    std::vector<int> fill(start.begin(), start.end() - 1);
    for (int c = 0; c < ncell; c++) if (pt[c] >= 0) order[fill[pt[c]]++] = c;
    ST_TRY(cudaMemcpyAsync(s->start, start.data(), sizeof(int) * ((size_t)n + 1), cudaMemcpyHostToDevice, s->stream));
    if (ncell) {
        ST_TRY(cudaMemcpyAsync(s->order, order.data(), sizeof(int) * ncell, cudaMemcpyHostToDevice, s->stream));
        ST_TRY(cudaMemcpyAsync(s->cell_pt, pt.data(), sizeof(int) * ncell, cudaMemcpyHostToDevice, s->stream));
        ST_TRY(cudaMemcpyAsync(s->cell, xzlr, sizeof(double) * 4 * (size_t)ncell, cudaMemcpyHostToDevice, s->stream));
    }
    ST_TRY(cudaStreamSynchronize(s->stream));
    return BCG_OK;
}

extern "C" int bcg_steady_solve(bcg_steady* s, const double* theta, const double* w, double tol,
                                double* C_out, int* newton_iters, int* cg_iters)
{
    if (!s || !theta || (s->ncell > 0 && !w)) return BCG_E_ARG;
    const double d_agar = theta[0], d_col = theta[1], vmax = theta[2], km = theta[3];
    if (!(d_agar > 0) || !(d_col > 0) || !(km > 0) || !(tol > 0)) return BCG_E_ARG;
    const int n = s->n;
    for (int l = 0; l < s->nlev; l++)
        k_st_rows<<<nblk(s->L[l].nz + 1), 256, 0, s->stream>>>(s->L[l], l, s->P.nz_agar, d_agar, d_col);
    if (s->ncell) ST_TRY(cudaMemcpyAsync(s->w, w, sizeof(double) * s->ncell, cudaMemcpyHostToDevice, s->stream));
    k_st_deposit<<<nblk(n), 256, 0, s->stream>>>(n, s->P.h, s->P.c0, s->start, s->order, s->cell, s->w, s->q, s->C);
    int it = 0, cgt = 0, rc;
    double f0 = 0.0;
    for (; it < 50; it++) {                  /* a run to the end (it == 50) missed its bound */
        double fn;
        if ((rc = st_newton_rhs(s, vmax, km, &fn))) return rc;
        if (it == 0) f0 = fn > 0 ? fn : 1.0;
        if (fn <= tol * f0 || fn == 0.0) break;
        int ci = 0;
        const double cg_tol = tol < 1e-8 ? (tol > 1e-14 ? tol : 1e-14) : 1e-8;
        if ((rc = st_pcg(s, s->F, cg_tol, 200, &ci))) return rc;
        cgt += ci;
        k_st_add<<<nblk(n), 256, 0, s->stream>>>(n, s->cg_x, s->C);   /* C += delta */
    }
    /* keep the converged linearisation for the adjoint */
    if ((rc = st_newton_rhs(s, vmax, km, nullptr))) return rc;
    s->solved = true;
    memcpy(s->theta, theta, sizeof(s->theta));
    if (C_out) ST_TRY(cudaMemcpyAsync(C_out, s->C, sizeof(double) * n, cudaMemcpyDeviceToHost, s->stream));
    ST_TRY(cudaStreamSynchronize(s->stream));
    if (newton_iters) *newton_iters = it;
    if (cg_iters) *cg_iters = cgt;
    return BCG_OK;
}

extern "C" int bcg_steady_vjp(bcg_steady* s, const double* dL_dC, double* grad_theta, double* grad_w, double tol)
{
    if (!s || !dL_dC || !grad_theta || !s->solved || !(tol > 0)) return BCG_E_ARG;
    const int n = s->n;
    /* A lambda = -dL/dC (row 0 is fixed: no adjoint there) */
    ST_TRY(cudaMemcpyAsync(s->cg_ap, dL_dC, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream));
    k_st_neg<<<nblk(n), 256, 0, s->stream>>>(n, s->P.nx, s->cg_ap, s->g);   /* g = -dL/dC, 0 on row 0 */
    int ci = 0;
    int rc = st_pcg(s, s->g, tol, 500, &ci);
    if (rc) return rc;
    const double* th = s->theta;
    k_st_grad_part<<<ST_RED_BLOCKS, 256, 0, s->stream>>>(s->L[0], s->P.nz_agar, th[0], th[1], s->C, s->q, s->cg_x, th[2], th[3], s->gpart);
    ST_TRY(cudaMemcpyAsync(s->pin, s->gpart, sizeof(double) * 4 * ST_RED_BLOCKS, cudaMemcpyDeviceToHost, s->stream));
    if (grad_w && s->ncell > 0) {
        k_st_grad_w<<<nblk(s->ncell), 256, 0, s->stream>>>(s->ncell, s->P.h, s->cell, s->cell_pt, s->C, s->cg_x, th[2], th[3], s->gw);
        ST_TRY(cudaMemcpyAsync(grad_w, s->gw, sizeof(double) * s->ncell, cudaMemcpyDeviceToHost, s->stream));
    }
    ST_TRY(cudaStreamSynchronize(s->stream));
    for (int j = 0; j < 4; j++) {
        double t = 0.0;
        for (int b = 0; b < ST_RED_BLOCKS; b++) t += s->pin[4 * b + j];
        grad_theta[j] = t;
    }
    return BCG_OK;
}

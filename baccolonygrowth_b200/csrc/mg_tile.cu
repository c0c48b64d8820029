/*
 * mg_tile.cu -- the agar multigrid on the levels that are too small to keep
 * the chip busy row by row: the zebra smoother on blocks of rows in
 * registers (k_mg_tile), and the coarsest levels of a V-cycle in one launch
 * (k_mg_tail).  The relaxation is relaxationAgarAtLevel's
 * (Multigrid.cpp:135-249), the transfers are those of Multigrid.cpp:269-467.
 *
 * k_mg_tile: a half-sweep relaxes every column of one parity bottom to top,
 *     E_k = A_k E_{k-1} + B_k,
 * where B_k holds the right-hand side, the neighbouring columns and the value
 * above, none of which the half-sweep changes before it reads them, and A_k is
 * w = 1/2 / (cf + 2) < 1/4 on interior rows.  Walking the rows costs a chain
 * as long as the column: the staged and the TMA forms take 17 to 60 us a
 * launch on levels whose traffic is 0.1 to 15 us.  Here a thread owns 9 rows
 * of a column pair and runs the recurrence on them from zero; what flows in
 * from below then adds w^(j+1) Y to its row j, Y the value at the top of the
 * rows below, which are the tops of the four chunks below combined (a fifth
 * adds w^36 < 3e-22 of itself).  A half-sweep is one pass over registers and
 * one barrier, whatever the column's height.
 *
 * Both are FP64: the mixed-precision solve's FP32 cycles keep the other forms.
 * Their result stands between the tolerance and FP32 rounding, so that another
 * order of the FP32 operations moves the solution by 2e-9 of itself.
 */
#include "ctx.cuh"
#include "mg.cuh"
#include <string.h>

/* Rows of a chunk (a warp's rows), and chunks a block stacks at most: 144 rows
 * of 128 registers a thread, which also takes the 2^a + 1 rows of the usual
 * grids up to 129 in one piece.  At 128 registers a thread spills little (172
 * bytes stored, 388 loaded in all).  Chunks of 8 would need 17 warps, five on a
 * scheduler, for which 96 registers are left. */
#define MT_ROWS 9
#define MT_WARPS 16

struct MtPlan { int S, n0, n1, warm; };      /* sweeps; rows of the first and of the later segments; warm-up rows */

/* What a thread knows of its rows and, per parity, of its column.  The cases
 * of relax_val come down to these: a side column takes its inner neighbour on
 * both sides (weights 1/2 + 1/2 for its 1), row 0 the value above twice, row nz
 * the value below twice; and a point that keeps R or its old value finds that
 * value in its R register, where the others have c R.  The top chunk and warps
 * with a side column run variants of their own, because a launch is bound by
 * the instruction count of its slowest warp (a warp alone on a scheduler
 * issues about one in three cycles): 10.4 us at 897 x 129 points against 13.3 us
 * with one variant for both cases. */
struct MtRows {
    double w, p2, p3, p4, p9;     /* w and its powers */
    int slot, jt;            /* chunk; the top row's place in it (>= MT_ROWS: not here) */
    bool bottom;             /* the chunk holds row 0 */
    bool sides;              /* the warp holds a side column */
    bool top_levels;
};
struct MtCol { bool left, right, hold, row0; };    /* i = 0, i = nx; keeps a value above row 0, on row 0 */

/* Chunk exchange of a strip: [parity][4 + chunk] tops after the local
 * recurrence (slot 3 the row below the segment, 0 to 2 zero), [parity][chunk]
 * first rows. */
template <int N> struct MtShare { double L[2][N + 4][32], F[2][N + 1][32]; };

/* First part of a half-sweep of the columns of parity PAR: X this parity's
 * rows, O the other's; the recurrence from zero. */
template <int PAR, bool TOP, bool SIDES, class SH>
__device__ __forceinline__ void mt_pre(double (&X)[MT_ROWS], const double (&O)[MT_ROWS], const double (&R)[MT_ROWS], const MtRows& c,
                                       const MtCol& col, SH& sh)
{
    const int lane = threadIdx.x & 31;
    const double top = sh.F[PAR][c.slot + 1][lane];           /* the chunk above, before this half-sweep */
    double prev = 0.0;
#pragma unroll
    for (int j = 0; j < MT_ROWS; j++) {
        const double nb = PAR ? __shfl_down_sync(0xffffffffu, O[j], 1) : __shfl_up_sync(0xffffffffu, O[j], 1);
        double xm = PAR ? O[j] : nb, xp = PAR ? nb : O[j];
        if (SIDES) { if (col.left) xm = xp; if (col.right) xp = xm; }
        double up = j + 1 < MT_ROWS ? X[j + 1 < MT_ROWS ? j + 1 : j] : top;
        if (j == 0 && c.bottom) up += up;
        double dn = prev;
        if (TOP) { if (j >= c.jt) up = 0.0; if (j == c.jt) dn += dn; }
        prev = fma(c.w, dn, fma(c.w, (xm + xp) + up, R[j]));
        if (SIDES && col.hold) prev = R[j];
        if (j == 0 && c.bottom && col.row0) prev = R[0];
        if (TOP) { if (j > c.jt || (j == c.jt && !c.top_levels)) prev = X[j]; }
        X[j] = prev;
    }
    sh.L[PAR][c.slot + 4][lane] = prev;
}
/* Second part: what flows in from the chunks below. */
template <int PAR, bool TOP, bool SIDES, class SH>
__device__ __forceinline__ void mt_post(double (&X)[MT_ROWS], const MtRows& c, const MtCol& col, SH& sh)
{
    const int lane = threadIdx.x & 31;
    double y = sh.L[PAR][c.slot][lane];
#pragma unroll
    for (int d = 1; d <= 3; d++) y = fma(c.p9, y, sh.L[PAR][c.slot + d][lane]);
    if (SIDES && col.hold) y = 0.0;                     /* a held column takes nothing from below */
    const double y4 = c.p4 * y, y8 = c.p4 * y4;
    const double z[MT_ROWS] = {y, y, y, y, y4, y4, y4, y4, y8};
    const double p[4] = {c.w, c.p2, c.p3, c.p4};
#pragma unroll
    for (int j = 0; j < MT_ROWS; j++) {
        if (TOP) {
            double zz = z[j];
            if (j == c.jt) zz += zz;
            if (j < c.jt || (j == c.jt && c.top_levels)) X[j] = fma(p[j & 3], zz, X[j]);
        } else X[j] = fma(p[j & 3], z[j], X[j]);
    }
    sh.F[PAR][c.slot][lane] = X[0];
}
/* S sweeps on a strip's chunks.  A block's warps are in either variant, with
 * the same barriers.  Between a first part and its second the tops are
 * published; the first rows a half-sweep leaves are read two half-sweeps later,
 * with a barrier between. */
template <bool TOP, bool SIDES, class SH>
__device__ __forceinline__ void mt_sweeps(double (&Ee)[MT_ROWS], double (&Eo)[MT_ROWS], const double (&Re)[MT_ROWS], const double (&Ro)[MT_ROWS],
                                          const MtRows& c, const MtCol& ke, const MtCol& ko, SH& sh, int S)
{
    for (int s = 0; s < S; s++) {
        mt_pre<0, TOP, SIDES>(Ee, Eo, Re, c, ke, sh);
        asm volatile("bar.sync 0;" ::: "memory");
        mt_post<0, TOP, SIDES>(Ee, c, ke, sh);
        mt_pre<1, TOP, SIDES>(Eo, Ee, Ro, c, ko, sh);
        asm volatile("bar.sync 0;" ::: "memory");
        mt_post<1, TOP, SIDES>(Eo, c, ko, sh);
    }
}

/* One smoothing of a strip: rows k0 .. k0 + MT_ROWS - 1 of columns ce, ce + 1
 * (lane order) read through ld(array, k), S sweeps, and the results left in Ee
 * and Eo.  kw: first row of the segment. */
template <class SH, class Load, class Add>
__device__ __forceinline__ void mt_strip(double (&Ee)[MT_ROWS], double (&Eo)[MT_ROWS], const MgConst& m, int l, int sp, int nx, int nz, int ce,
                                         int kw, int slot, int chunks, int S, SH& sh,
                                         const double* __restrict__ inside0, const Load& ld, const Add& add)
{
    const int lane = threadIdx.x & 31, co = ce + 1, k0 = kw + MT_ROWS * slot;
    const RelaxK<double> K = relax_k<double>(m, l, sp);
    MtRows c;
    c.w = K.w; c.p2 = K.w * K.w; c.p3 = c.p2 * K.w; c.p4 = c.p2 * c.p2; c.p9 = c.p4 * c.p4 * K.w;
    c.slot = slot; c.jt = nz - k0; c.bottom = k0 == 0; c.top_levels = l >= m.A - 1;
    const bool oxy = sp == 1;
    MtCol ke, ko;
    ke.left = ce == 0; ke.right = ce == nx; ko.left = false; ko.right = co == nx;
    c.sides = __any_sync(0xffffffffu, ke.left || ke.right || ko.right);
    double Re[MT_ROWS], Ro[MT_ROWS];
#pragma unroll
    for (int j = 0; j < MT_ROWS; j++) {
        Ee[j] = Eo[j] = Re[j] = Ro[j] = 0.0;
        if (k0 + j <= nz) ld(k0 + j, Ee[j], Eo[j], &Re[j], &Ro[j]);
    }
    add(k0, Ee, Eo);
    double ae = 0.0, ao = 0.0;
    if (slot == chunks - 1) {
        if (k0 + MT_ROWS <= nz) ld(k0 + MT_ROWS, ae, ao, (double*)nullptr, (double*)nullptr);
        sh.F[0][slot + 1][lane] = ae; sh.F[1][slot + 1][lane] = ao;
    }
    sh.F[0][slot][lane] = Ee[0]; sh.F[1][slot][lane] = Eo[0];
    if (slot == 0) {
        ae = ao = 0.0;
        if (kw > 0) ld(kw - 1, ae, ao, (double*)nullptr, (double*)nullptr);
#pragma unroll
        for (int d = 0; d < 3; d++) sh.L[0][d][lane] = sh.L[1][d][lane] = 0.0;
        sh.L[0][3][lane] = ae; sh.L[1][3][lane] = ao;
    }
    auto finish = [&](MtCol& col, int i, double (&r)[MT_ROWS], const double (&e)[MT_ROWS]) {
        const bool side = col.left || col.right;
        bool inside = false;
        if (c.bottom) {
            int i0 = (i - nx / 2) * (1 << l) + m.box_x / 2;
            i0 = i0 < 0 ? 0 : (i0 > m.box_x - 1 ? m.box_x - 1 : i0);
            inside = inside0[(size_t)i0 * m.box_z] > 0;
        }
        col.hold = side && (!c.top_levels || oxy);
        col.row0 = inside || oxy || (side && !c.top_levels);
        const bool old = !c.top_levels, old0 = side && old && !inside;
#pragma unroll
        for (int j = 0; j < MT_ROWS; j++) {
            const bool fix = j == 0 && c.bottom ? col.row0 : col.hold;
            const bool keep = j == 0 && c.bottom ? old0 : old;
            r[j] = !fix ? K.c * r[j] : (keep ? e[j] : r[j]);
        }
    };
    finish(ke, ce, Re, Ee);
    finish(ko, co, Ro, Eo);
    asm volatile("bar.sync 0;" ::: "memory");
    if (c.jt < MT_ROWS) {
        if (c.sides) mt_sweeps<true, true>(Ee, Eo, Re, Ro, c, ke, ko, sh, S);
        else mt_sweeps<true, false>(Ee, Eo, Re, Ro, c, ke, ko, sh, S);
    } else {
        if (c.sides) mt_sweeps<false, true>(Ee, Eo, Re, Ro, c, ke, ko, sh, S);
        else mt_sweeps<false, false>(Ee, Eo, Re, Ro, c, ke, ko, sh, S);
    }
}

/* S zebra sweeps of a level, E -> E2.  A warp holds 9 rows of 64 columns
 * (lane t: columns c0 + 2t and c0 + 2t + 1), a block stacks up to 16 warps
 * (144 rows).  A half-sweep is exact where its inputs were, which loses one
 * column at either strip edge: the middle 64 - 4S columns are written.  Levels
 * of more rows are cut into segments that start `warm` rows early (from the
 * values before smoothing, as the other forms do) and end S - 1 rows late.
 * Three sweeps in FP64: 897 x 129 points 37 -> 10.4 us, 449 x 65 25 -> 8.5 us,
 * 1153 x 257 35 -> 12 us, 2305 x 513 57 -> 39 us.  What bounds
 * the small ones is the chain: loads 1.5 us, six half-sweeps of 0.7 us.  The
 * largest repeat 35 of 144 rows and 12 of 64 columns, and a block fills its
 * SM's registers, so loads and sweeps of different blocks do not overlap.
 * INTERP: the values smoothed are E plus the next level's correction
 * (interpolationAga, Multigrid.cpp:407-467), added as they are read; as a launch
 * of its own it took 4.5 us on levels of 129 to 513 columns, so 1.5. */
template <bool INTERP>
__global__ void __launch_bounds__(32 * MT_WARPS, 1) k_mg_tile(MgConst m, MgLvl L, MgLvl Lc, int l, MtPlan plan,
                                                              const double* __restrict__ inside0)
{
    __shared__ MtShare<MT_WARPS> sh;
    const int lane = threadIdx.x, sp = blockIdx.z, S = plan.S;
    const int nx = L.nx, nz = L.nz;
    const int ks = blockIdx.y == 0 ? 0 : plan.n0 + (blockIdx.y - 1) * plan.n1;
    const int ke = min(ks + (blockIdx.y == 0 ? plan.n0 : plan.n1), nz + 1);
    const int kw = max(0, ks - plan.warm);
    const int outp = 32 - 2 * S;
    const int ce = blockIdx.x * 2 * outp - 2 * S + 2 * lane;
    const bool in = ce >= 0 && ce <= nx;
    const double* __restrict__ E = SP(L.e);
    const double* __restrict__ R = SP(L.r);
    /* X 2^A / 2^l / 4, as a shift; the coarse column of the even column (the one
     * beside a last even column is not used: it lies in the plane's padding) */
    const int nxp = min((m.box_x << m.A) >> (l + 2), m.box_x);
    const double* __restrict__ C = SP(Lc.e) + (nxp / 2 - nx / 4 + (ce >> 1));
    double Ee[MT_ROWS], Eo[MT_ROWS];
    auto ld = [&](int k, double& e, double& o, double* re, double* ro) {
        if (!in) return;
        const size_t at = (size_t)k * L.pitch + ce;
        const double2 v = *reinterpret_cast<const double2*>(E + at);
        e = v.x; o = v.y;
        if (INTERP && !re) {
            const double* c = C + (size_t)(k >> 1) * Lc.pitch;
            const double* d = (k & 1) ? c + Lc.pitch : c;
            const double c0 = c[0], c1 = c[1], d0 = d[0], d1 = d[1];
            const double ie = (k & 1) ? 0.5 * (c0 + d0) : c0, io = (k & 1) ? 0.25 * (c0 + d0 + c1 + d1) : 0.5 * (c0 + c1);
            e += ie;
            if (ce < nx) o += io;
        }
        if (re) { const double2 q = *reinterpret_cast<const double2*>(R + at); *re = q.x; *ro = q.y; }
    };
    /* the prolongation on a thread's 9 rows: one coarse column of the six rows
     * they lie between (the next column is the next lane's), an odd row taking the
     * mean of two */
    auto add = [&](int k0, double (&e)[MT_ROWS], double (&o)[MT_ROWS]) {
        if (!INTERP) return;
        constexpr int ROWS = (MT_ROWS + 3) / 2;
        const int p = k0 & 1;
        double c[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int kp = (k0 >> 1) + r;
            c[r] = in && 2 * kp <= nz + 1 ? C[(size_t)kp * Lc.pitch] : 0.0;
        }
        double x[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int kp = (k0 >> 1) + r;
            x[r] = __shfl_down_sync(0xffffffffu, c[r], 1);
            if ((lane == 31 || ce + 2 > nx) && in && 2 * kp <= nz + 1) x[r] = C[(size_t)kp * Lc.pitch + 1];
        }
        const bool odd = ce < nx;
#pragma unroll
        for (int j = 0; j < MT_ROWS; j++) {
            const int a = j >> 1, b = (j + 1) >> 1;       /* the row's coarse row for an even k0, for an odd one */
            const double c0 = p ? c[b] : c[a], c1 = p ? x[b] : x[a];
            double ie = c0, io = 0.5 * (c0 + c1);
            if ((p != 0) != (j & 1)) {
                const double d0 = p ? c[b + 1 < ROWS ? b + 1 : b] : c[a + 1 < ROWS ? a + 1 : a];
                const double d1 = p ? x[b + 1 < ROWS ? b + 1 : b] : x[a + 1 < ROWS ? a + 1 : a];
                ie = 0.5 * (c0 + d0);
                io = 0.25 * (c0 + d0 + c1 + d1);
            }
            if (in && k0 + j <= nz) { e[j] += ie; if (odd) o[j] += io; }
        }
    };
    mt_strip(Ee, Eo, m, l, sp, nx, nz, ce, kw, threadIdx.y, blockDim.y, S, sh, inside0, ld, add);
    if (lane < S || lane > 31 - S || !in) return;
    double* __restrict__ EO = SP(L.e2);
#pragma unroll
    for (int j = 0; j < MT_ROWS; j++) {
        const int k = kw + MT_ROWS * (int)threadIdx.y + j;
        if (k < ks || k >= ke) continue;
        double* dst = EO + (size_t)k * L.pitch + ce;
        if (ce + 1 <= nx) { double2 v; v.x = Ee[j]; v.y = Eo[j]; *reinterpret_cast<double2*>(dst) = v; }
        else dst[0] = Ee[j];
    }
}

int mg_smooth_tile(bcg_ctx* c, const MgConst& m, const MgLvl& L, int l, int S, int warm, const MgLvl* coarse)
{
    const int rows = L.nz + 1, cap = MT_ROWS * MT_WARPS - (S - 1);
    MtPlan p;
    p.S = S; p.warm = warm;
    int nseg = 1;
    if (rows > cap) nseg = 1 + (rows - cap + cap - warm - 1) / (cap - warm);
    /* the first segment has no warm-up rows: equal rows in every block */
    p.n0 = nseg == 1 ? rows : (rows + (nseg - 1) * warm + nseg - 1) / nseg;
    p.n1 = nseg == 1 ? rows : p.n0 - warm;
    if (p.n1 < 1 || p.n0 > cap) return BCG_E_ARG;
    const int held = nseg == 1 ? rows : p.n0 + S - 1;
    const int outp = 32 - 2 * S;
    const dim3 grid((unsigned)((L.nx + 1 + 2 * outp - 1) / (2 * outp)), (unsigned)nseg, 3);
    const dim3 block(32, (unsigned)((held + MT_ROWS - 1) / MT_ROWS));
    if (coarse) k_mg_tile<true><<<grid, block, 0, c->stream>>>(m, L, *coarse, l, p, c->inside);
    else k_mg_tile<false><<<grid, block, 0, c->stream>>>(m, L, L, l, p, c->inside);
    c->launches++;
    return BCG_OK;
}

/* ------------------------------------------------------------------------ */
/* the coarsest levels of a V-cycle in one launch                            */
/* ------------------------------------------------------------------------ */
#define MTAIL_THREADS 256
#define MTAIL_LEVELS 8

/* a level in the tail's shared memory (offsets in values): E in rows of
 * nx + 2 (the prolongation of a level with an odd column count reads one column
 * past the coarse level's last, which is the plane's padding), R in rows of
 * nx + 1; the row-0 flags of its columns at byte `ins` */
struct MtLevel { int nx, nz, pitch, e, r, ins, col0; unsigned mag_e, mag_r; };
struct MtTail {
    MtLevel lv[MTAIL_LEVELS];
    RelaxK<double> k[MTAIL_LEVELS][3];
    double scale[MTAIL_LEVELS][3];    /* of the stencil sum in the restriction from the level */
    double* e[MTAIL_LEVELS][3];
    const double* r0[3];
    int l0, n, cols;
};

/* (i, k) with the reference's flat index i (nz + 1) + k, as at_ref */
__device__ __forceinline__ double mtail_at(const double* a, int row, int nx, int nz, int i, int k)
{
    if (k >= 0 && k <= nz) return a[k * row + i];
    const int f = i * (nz + 1) + k, n = (nx + 1) * (nz + 1);
    if (f < 0 || f >= n) return 0.0;
    return a[(f % (nz + 1)) * row + f / (nz + 1)];
}

/* One zebra sweep of a level held in shared memory, a thread a column; true
 * if the thread changed a value (STOP; false otherwise).  Four rows' loads and
 * neighbour terms come before their chain; a side column takes its inner
 * neighbour on both sides (see MtRows), so that all columns of a warp take
 * the same path.  The block has two or three busy warps, so what counts is
 * the instructions of a row; splitting the columns into chunks as k_mg_tile
 * does took more of them in all and longer (51 to 90 us against 43). */
template <bool STOP>
__device__ __forceinline__ bool mtail_sweep(double* m, const MtLevel& L, const unsigned char* ins, bool oxy, bool top_levels,
                                            const RelaxK<double>& K)
{
    const int nx = L.nx, nz = L.nz, EW = nx + 2, RW = nx + 1;
    bool changed = false;
    for (int par = 0; par < 2; par++) {
        for (int i = 2 * (int)threadIdx.x + par; i <= nx; i += 2 * MTAIL_THREADS) {
            double* e = m + L.e + i;
            const double* r = m + L.r + i;
            const bool side = i == 0 || i == nx;
            const int xm = i == 0 ? 1 : -1, xp = i == nx ? -1 : 1;
            const double r0 = r[0], old0 = e[0];
            if (side && (!top_levels || oxy)) {
                /* a held column */
                const double v0 = (ins[i] & 1) || top_levels ? r0 : old0;
                if (STOP) changed |= v0 != old0;
                e[0] = v0;
                if (top_levels)
                    for (int k = 1; k <= nz; k++) {
                        if (STOP) changed |= e[k * EW] != r[k * RW];
                        e[k * EW] = r[k * RW];
                    }
                continue;
            }
            /* row 0, whose value above follows the flat index where there is no row 1 */
            double v = nz > 0 ? e[EW] : mtail_at(m + L.e, EW, nx, nz, i, 1);      /* the next row's old value */
            double below = rx_k0(r0, v, e[xm], e[xp], K);
            if (oxy || (ins[i] & 1)) below = r0;
            e[0] = below;
            if (STOP) changed |= below != old0;
            int k = 1;
            double* q = e + EW;
            const double* p = r + RW;
            for (; k + 3 < nz; k += 4, q += 4 * EW, p += 4 * RW) {
                double u[5], b[4];
                u[0] = v;
#pragma unroll
                for (int j = 1; j < 5; j++) u[j] = q[j * EW];
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = fma(K.w, (q[j * EW + xm] + q[j * EW + xp]) + u[j + 1], K.c * p[j * RW]);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    below = fma(K.w, below, b[j]);
                    q[j * EW] = below;
                    if (STOP) changed |= below != u[j];
                }
                v = u[4];
            }
            for (; k < nz; k++, q += EW, p += RW) {
                const double up = q[EW];
                below = rx_in(p[0], below, up, q[xm], q[xp], K);
                q[0] = below;
                if (STOP) changed |= below != v;
                v = up;
            }
            if (k == nz && top_levels) {
                below = rx_top(p[0], below, q[xm], q[xp], K);
                q[0] = below;
                if (STOP) changed |= below != v;
            }
        }
        __syncthreads();
    }
    return changed;
}

/* Levels l0 .. l0 + n - 1 (the coarsest) of a V-cycle, one block a species, E
 * and R in shared memory: descent (mu1 sweeps, restriction), mu2 sweeps on the
 * coarsest level, ascent (prolongation, mu1 sweeps).  The levels are plain
 * coarsenings (or the coarsest alone).  They took four launches each and, for
 * the mu2 = 100 sweeps of a few hundred points, 100 to 166 us of barriers.
 * A sweep that leaves every value as it found it is reproduced by every later
 * one, so the coarsest level stops there, with the values that all mu2 sweeps
 * give; at the reference's spacing that is after 5 to 20 (a correction
 * spreads one column a half-sweep, however small it has become).
 * 113 x 17 points and three levels below it: 400 us in 20 launches -> 49 us;
 * 129 x 17 and five below: 60 us.  What bounds it is the chain of some 45
 * half-sweeps on two or three warps, about 120 cycles a row. */
__global__ void __launch_bounds__(MTAIL_THREADS) k_mg_tail(const __grid_constant__ MgConst m, const __grid_constant__ MtTail a, int mu1, int mu2,
                                                           const double* __restrict__ inside0)
{
    extern __shared__ __align__(16) unsigned char mt_smem[];
    __shared__ RelaxK<double> sk[MTAIL_LEVELS];
    double* sm = reinterpret_cast<double*>(mt_smem);
    const int sp = blockIdx.x, th = threadIdx.x;
    /* E of every level and R of the finest, straight into shared memory */
    auto fetch = [&](double* dst, const double* src) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(sizeof(double)));
    };
    for (int q = 0; q < a.n; q++) {
        const MtLevel L = a.lv[q];
        const double* e = SP(a.e[q]);
        for (int f = th; f < (L.nx + 2) * (L.nz + 1); f += MTAIL_THREADS) {
            const int k = (int)__umulhi((unsigned)f, L.mag_e), i = f - k * (L.nx + 2);
            if (i < L.pitch) fetch(sm + L.e + f, e + (size_t)k * L.pitch + i);
            else sm[L.e + f] = 0.0;
        }
    }
    {
        const MtLevel L = a.lv[0];
        const double* r = SP(a.r0);
        for (int f = th; f < (L.nx + 1) * (L.nz + 1); f += MTAIL_THREADS) {
            const int k = (int)__umulhi((unsigned)f, L.mag_r);
            fetch(sm + L.r + f, r + (size_t)k * L.pitch + f - k * (L.nx + 1));
        }
    }
    asm volatile("cp.async.commit_group;");
    if (th < a.n) sk[th] = SP(a.k[th]);
    /* row-0 colony flags per column: bit 0 as the smoother clamps its box
     * column, bit 1 as the restriction does */
    for (int f = th; f < a.cols; f += MTAIL_THREADS) {
        int q = 0;
        while (q + 1 < a.n && f >= a.lv[q + 1].col0) q++;
        const int nx = a.lv[q].nx, i = f - a.lv[q].col0;
        const int i0 = (i - nx / 2) * (1 << (a.l0 + q)) + m.box_x / 2;
        const int is = i0 < 0 ? 0 : (i0 > m.box_x - 1 ? m.box_x - 1 : i0), ir = i0 < 0 ? 0 : i0;
        const bool fs = inside0[(size_t)is * m.box_z] > 0;
        mt_smem[a.lv[q].ins + i] = (unsigned char)((fs ? 1 : 0) | (fs && ir < m.box_x ? 2 : 0));
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    const bool oxy = sp == 1;
    const double half = 0.5, quarter = 0.25;
    /* down to the coarsest level and back up: one place for each phase, since
     * every inlined copy of the sweep costs registers and instruction cache */
    for (int step = 0; step < 2 * a.n - 1; step++) {
        const bool up = step >= a.n;
        const int q = up ? 2 * (a.n - 1) - step : step;
        const MtLevel& L = a.lv[q];
        const bool last = q == a.n - 1, top_levels = a.l0 + q >= m.A - 1;
        if (up) {
            /* interpolationAga: Err of this level += from the next */
            const MtLevel& C = a.lv[q + 1];
            double* E = sm + L.e;
            const double* c = sm + C.e;
            const int EW = L.nx + 2, CW = C.nx + 2;
#define CV(x, z) mtail_at(c, CW, C.nx, C.nz, x, z)
            for (int f = th; f < EW * (L.nz + 1); f += MTAIL_THREADS) {
                const int k = (int)__umulhi((unsigned)f, L.mag_e), i = f - k * EW, j = i >> 1, kp = k >> 1;
                if (i > L.nx) continue;
                double inc = CV(j, kp);
                if (k & 1) {
                    const double c1 = CV(j, kp + 1);
                    if (i & 1) inc = quarter * (inc + c1 + CV(j + 1, kp) + CV(j + 1, kp + 1));
                    else inc = half * (inc + c1);
                } else if (i & 1) inc = half * (inc + CV(j + 1, kp));
                E[f] += inc;
            }
#undef CV
            __syncthreads();
        }
        {
            RelaxK<double> K;
            K.inv = sk[q].inv; K.c = sk[q].c; K.w = sk[q].w; K.cf = 0.0;
            const int sweeps = last ? mu2 : mu1;
            for (int s = 0; s < sweeps; s++) {
                if (!last) mtail_sweep<false>(sm, L, mt_smem + L.ins, oxy, top_levels, K);
                else if (!__syncthreads_or(mtail_sweep<true>(sm, L, mt_smem + L.ins, oxy, top_levels, K))) break;
            }
        }
        if (!up && !last) {
            /* restrictionAgaElementwise for a plain coarsening: ip = 2i, kp = 2k */
            const MtLevel& C = a.lv[q + 1];
            const unsigned char* ins = mt_smem + C.ins;
            const double* E = sm + L.e;
            const double* R = sm + L.r;
            const int EW = L.nx + 2, RW = L.nx + 1;
            const double s = SP(a.scale[q]);
#define EV(x, z) mtail_at(E, EW, L.nx, L.nz, x, z)
            for (int f = th; f < (C.nx + 1) * (C.nz + 1); f += MTAIL_THREADS) {
                const int k = (int)__umulhi((unsigned)f, C.mag_r), i = f - k * (C.nx + 1), ip = 2 * i, kp = 2 * k;
                const double r = R[kp * RW + ip], e = EV(ip, kp);
                double out;
                if (i == 0 || i == C.nx || k == C.nz) {
                    if (k == C.nz && i > 0 && i < C.nx) {
                        out = (r + s * (EV(ip + 1, kp) + EV(ip - 1, kp) + 2 * EV(ip, kp - 1) - 4 * e) - e) / 2;
                    } else {
                        const int sx = i == 0 ? 1 : -1;
                        if (oxy) out = r - e;
                        else if (k == 0) out = (r + s * (2 * EV(ip + sx, kp) + 2 * EV(ip, kp + 1) - 4 * e) - e) / 2;
                        else if (k == C.nz) out = (r + s * (2 * EV(ip + sx, kp) + 2 * EV(ip, kp - 1) - 4 * e) - e) / 2;
                        else out = (r + s * (2 * EV(ip + sx, kp) + EV(ip, kp + 1) + EV(ip, kp - 1) - 4 * e) - e) / 2;
                    }
                } else if (k == 0) {
                    if (ins[i] & 2) out = 0.0;
                    else if (oxy) out = (r - e) * half;
                    else out = (r + s * (EV(ip + 1, 0) + EV(ip - 1, 0) + 2 * EV(ip, 1) - 4 * e) - e) * half;
                } else
                    out = (r + s * (EV(ip + 1, kp) + EV(ip - 1, kp) + EV(ip, kp + 1) + EV(ip, kp - 1) - 4 * e) - e) * half;
                sm[C.r + f] = out;
            }
#undef EV
            __syncthreads();
        }
    }
    for (int q = 0; q < a.n; q++) {
        const MtLevel L = a.lv[q];
        double* e = SP(a.e[q]);
        for (int f = th; f < (L.nx + 2) * (L.nz + 1); f += MTAIL_THREADS) {
            const int k = (int)__umulhi((unsigned)f, L.mag_e), i = f - k * (L.nx + 2);
            if (i <= L.nx) e[(size_t)k * L.pitch + i] = sm[L.e + f];
        }
    }
}

/* shared memory of the tail from level l on, in bytes */
static size_t mtail_smem(const bcg_ctx* c, int l)
{
    size_t v = 0, flags = 0;
    for (; l < c->mg_levels; l++) {
        const MgLevel& L = c->mg[l];
        v += (size_t)(2 * L.nx + 3) * (L.nz + 1);
        flags += (size_t)L.nx + 1;
    }
    return v * sizeof(double) + flags;
}
/* First level of the tail (the level count: none).  A block relaxes a level
 * of MTAIL_POINTS points in about the time of k_mg_tile's launch and the two
 * transfers'; on a larger coarsest level the cluster form is the faster one
 * (145 x 33 points: 107 us against 143 us, 33 sweeps of a thread a column). */
#define MTAIL_POINTS 2600
#define MTAIL_SMEM (196 * 1024)
int mg_tail_level(const bcg_ctx* c, const MgConst& m)
{
    const int last = c->mg_levels - 1;
    int l0 = c->mg_levels;
    for (int l = last; l >= 0; l--) {
        const MgLevel& L = c->mg[l];
        if (last - l >= MTAIL_LEVELS || mtail_smem(c, l) > MTAIL_SMEM) break;
        if ((L.nx + 1) * (L.nz + 1) > MTAIL_POINTS) break;
        if (l < last) {
            if (l < m.A) break;
            /* an odd column count reads the padding beside the coarse level's
             * last column; without padding that is another row's point */
            if ((L.nx & 1) && (c->mg[l + 1].nx + 1) % 32 == 0) break;
        }
        l0 = l;
    }
    return l0;
}
int mg_tail(bcg_ctx* c, const MgConst& m, const MgLvl* lvls, int l0, int mu1, int mu2)
{
    MtTail a;
    memset(&a, 0, sizeof(a));
    a.l0 = l0; a.n = c->mg_levels - l0;
    int at = 0;
    for (int q = 0; q < a.n; q++) {
        MtLevel& L = a.lv[q];
        L.nx = lvls[q].nx; L.nz = lvls[q].nz; L.pitch = lvls[q].pitch;
        L.mag_e = 0xffffffffu / (unsigned)(L.nx + 2) + 1u; L.mag_r = 0xffffffffu / (unsigned)(L.nx + 1) + 1u;
        L.e = at; at += (L.nx + 2) * (L.nz + 1);
        L.r = at; at += (L.nx + 1) * (L.nz + 1);
        L.col0 = a.cols; a.cols += L.nx + 1;
        const int l = l0 + q;
        for (int s = 0; s < 3; s++) {
            /* as relax_k; the restriction to level l + 1 scales by 1/2 D dt 4 / h^2 of that level */
            const double cf = m.bl2 * (double)(1 << (2 * l)) / m.dt / m.D[s], inv = 1.0 / (cf + 2.0);
            a.k[q][s].cf = cf; a.k[q][s].inv = inv; a.k[q][s].c = (cf * inv); a.k[q][s].w = (0.5 * inv);
            a.scale[q][s] = (2.0 * m.D[s] * m.dt / (m.bl2 * (double)(1 << (2 * (l + 1)))));
        }
        for (int s = 0; s < 3; s++) a.e[q][s] = lvls[q].e[s];
    }
    for (int q = 0; q < a.n; q++) a.lv[q].ins = at * (int)sizeof(double) + a.lv[q].col0;
    for (int s = 0; s < 3; s++) a.r0[s] = lvls[0].r[s];
    k_mg_tail<<<3, MTAIL_THREADS, mtail_smem(c, l0), c->stream>>>(m, a, mu1, mu2, c->inside);
    c->launches++;
    return BCG_OK;
}

int mg_tile_attributes()
{
    if (cudaFuncSetAttribute(k_mg_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, MTAIL_SMEM) != cudaSuccess)
        return BCG_E_CUDA;
    return BCG_OK;
}

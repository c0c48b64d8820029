/*
 * fields.cu -- cell-to-grid deposition and the surface fields
 * (AgentBasedModel-BacColonyGrowth/Compute.cpp:120-738).
 *
 * GetDensity / GetHeight walk the bins of the current record buffer (a block
 * or a warp per x column, a thread per box); ShiftDensity, BoxAverage,
 * Height_Average, Smooth and GetSurfaceNormal are stencil kernels bounded by
 * the device-resident bounding box, so the chain runs without host syncs.
 */
#include "ctx.cuh"
#include "cellmath.cuh"

int bin_cells(bcg_ctx* c, int buf);

#define IX(x, z) ((size_t)(x) * Z + (z))

/* keep (may be null): insideColonyDen's row z = 0 as it was */
__global__ void k_bbox_reset(int* bbox, int X, int Z, const double* __restrict__ inside, double* __restrict__ keep)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x == 0) { bbox[0] = X; bbox[1] = 0; bbox[2] = 0; }
    if (keep && x < X) keep[x] = inside[IX(x, 0)];
}

/* one box's share of the column's heights: the highest top among the cells
 * over each of the rgh sub-columns.  h starts from the cell radius, so only
 * positive tops count, and positive doubles order as their bit patterns. */
__device__ __forceinline__ void raise_height(long long* h, int i_ht, int rgh, double top)
{
    if (i_ht < 0) i_ht = 0;
    if (i_ht > rgh - 1) i_ht = rgh - 1;
    if (i_ht < 8 && top > __longlong_as_double(h[i_ht])) atomicMax(&h[i_ht], __double_as_longlong(top));
}

/* GetDensity (Compute.cpp:120-227): per box sum of Length*Radius, the
 * inside flag, and per column the max top of the cells (starting from the
 * cell radius).  One block per column and one thread per box: what bounds it
 * is the chain of loads start -> id -> record of each box, so a box's cells
 * are the only ones walked in series (their sum keeps its order).  One thread
 * per column, over all its boxes, took 95 us at 4096 cells (256 columns), 411
 * at 262144 (2304) and 772 at 1048576 (4608); this form 10, 16 and 43. */
#define COLUMN_THREADS 128
__global__ void __launch_bounds__(COLUMN_THREADS) k_get_density(int X, int Z, int rgh, double box_length, double cell_radius,
                              const CellRec* __restrict__ rec, const int* __restrict__ box_start,
                              const int* __restrict__ box_ids, double* __restrict__ rd,
                              double* __restrict__ inside, double* __restrict__ height, int* bbox)
{
    __shared__ long long h[8];
    __shared__ int top_z;
    const int bx = blockIdx.x;
    if (threadIdx.x < 8) h[threadIdx.x] = __double_as_longlong(cell_radius);
    if (threadIdx.x == 0) top_z = -1;
    __syncthreads();
    const double Vbox = box_length * box_length;
    for (int bz = threadIdx.x; bz < Z; bz += COLUMN_THREADS) {
        int b = bx * Z + bz;
        int s = box_start[b], e = box_start[b + 1];
        double den = 0;
        for (int t = s; t < e; t++) {
            const CellRec& r = rec[box_ids[t]];
            double4 pl = r.pL, qr = r.qR;
            double cmx = (pl.x + qr.x) * 0.5;
            raise_height(h, (int)((cmx / box_length - (bx - X / 2)) * rgh), rgh, pl.z > qr.z ? pl.z : qr.z);
            den += pl.w * qr.w;
        }
        if (e > s) atomicMax(&top_z, bz);
        if (den == 0) { rd[IX(bx, bz)] = 0; inside[IX(bx, bz)] = 0; }
        else { rd[IX(bx, bz)] = den / Vbox; inside[IX(bx, bz)] = 1.0; }
    }
    __syncthreads();
    if (threadIdx.x < rgh && threadIdx.x < 8) height[bx * rgh + threadIdx.x] = __longlong_as_double(h[threadIdx.x]);
    if (threadIdx.x == 0 && top_z >= 0) { atomicMin(&bbox[0], bx); atomicMax(&bbox[1], bx); atomicMax(&bbox[2], top_z); }
}

/* the boundary ring of insideColonyDen, Compute.cpp:228-249 (reads only
 * values > 0.5, so the in-place order does not matter) */
__global__ void k_inside_ring(int X, int Z, double* inside)
{
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= X * Z) return;
    int bx = id / Z, bz = id % Z;
    if (inside[id] < 0.5) {
        if (bz > 0 && bx > 0 && bx < X - 1 && bz < Z - 1) {
            if ((inside[IX(bx + 1, bz)] > 0.5) || (inside[IX(bx - 1, bz)] > 0.5) || (inside[IX(bx, bz + 1)] > 0.5) || (inside[IX(bx, bz - 1)] > 0.5))
                inside[id] = 0.4;
        } else if (bz == 0 && bx > 0 && bx < X - 1) {
            if ((inside[IX(bx + 1, bz)] > 0.5) || (inside[IX(bx - 1, bz)] > 0.5) || (inside[IX(bx, bz + 1)] > 0.5))
                inside[id] = 0.4;
        }
    }
}

/* GetHeight (Compute.cpp:256-340): top four occupied boxes per column.  One
 * warp per column looks at 32 boxes at a time from the top; a lane walks its
 * own box if it is among the first four (8.6 us at 4096 cells; one thread per
 * column 78). */
__global__ void __launch_bounds__(COLUMN_THREADS) k_get_height(int X, int Z, int rgh, double box_length, double cell_radius,
                             const CellRec* __restrict__ rec, const int* __restrict__ box_start,
                             const int* __restrict__ box_ids, double* __restrict__ height, int* bbox)
{
    __shared__ long long hs[COLUMN_THREADS / 32][8];
    const int lane = threadIdx.x & 31, bx = blockIdx.x * (COLUMN_THREADS / 32) + (threadIdx.x >> 5);
    if (bx >= X) return;                       /* whole warp */
    long long* h = hs[threadIdx.x >> 5];
    if (lane < 8) h[lane] = __double_as_longlong(cell_radius);
    __syncwarp();
    int found = 0, top_z = -1;
    for (int z0 = Z - 1; z0 >= 0 && found < 4; z0 -= 32) {
        const int bz = z0 - lane;
        int s = 0, e = 0;
        if (bz >= 0) { s = box_start[bx * Z + bz]; e = box_start[bx * Z + bz + 1]; }
        const unsigned occ = __ballot_sync(0xffffffffu, e > s);
        if (top_z < 0 && occ) top_z = z0 - (__ffs(occ) - 1);
        if (found + __popc(occ & ((1u << lane) - 1)) < 4)
            for (int t = s; t < e; t++) {
                const CellRec& r = rec[box_ids[t]];
                double4 pl = r.pL, qr = r.qR;
                double cmx = (pl.x + qr.x) * 0.5;
                raise_height(h, (int)((cmx - (bx - X / 2) * box_length) / (box_length / rgh)), rgh, pl.z > qr.z ? pl.z : qr.z);
            }
        found += __popc(occ);
    }
    __syncwarp();
    if (lane < rgh && lane < 8) height[bx * rgh + lane] = __longlong_as_double(h[lane]);
    if (lane == 0 && top_z >= 0) { atomicMin(&bbox[0], bx); atomicMax(&bbox[1], bx); atomicMax(&bbox[2], top_z); }
}

/* minx-5, maxx+5, maxz+5 (Compute.cpp:250-252) and the range the stencils
 * below need (the reference reads outside its arrays otherwise) */
__global__ void k_bbox_finish(int* bbox, int X, int Z, int FD, DevStatus* st)
{
    if (threadIdx.x != 0) return;
    if (bbox[0] > bbox[1]) { bbox[0] = X - 5; bbox[1] = 5; bbox[2] = 5; return; }   /* no cells */
    bbox[0] -= 5; bbox[1] += 5; bbox[2] += 5;
    if (bbox[0] - FD < 1 || bbox[1] + FD > X - 2 || bbox[2] + FD > Z) dev_error(st, BCG_E_NEED_MORE_BOXES, bbox[1]);
}

/* ShiftDensity (Compute.cpp:344-463) with Box_y = 1: the y = BoxY-1 passes
 * overwrite the 8-point averages, leaving these values. */
__global__ void k_shift(int X, int Z, const double* __restrict__ D, double* __restrict__ DS, double* __restrict__ WS)
{
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= X * Z) return;
    int x = id / Z, z = id % Z;
    double v;
    if (x < X - 1 && z < Z - 1) v = (D[IX(x, z)] + D[IX(x, z + 1)] + D[IX(x + 1, z)] + D[IX(x + 1, z + 1)]) / 4.0;
    else if (x < X - 1) v = (D[IX(x, Z - 1)] + D[IX(x + 1, Z - 1)]) / 2.0;
    else if (z < Z - 1) v = (D[IX(X - 1, z)] + D[IX(X - 1, z)]) / 2.0;
    else v = D[IX(X - 1, Z - 1)];
    DS[id] = v;
    if (z == 0 && WS) WS[x] = (x < X - 1) ? (D[IX(x, 0)] + D[IX(x + 1, 0)]) / 2.0 : D[IX(X - 1, 0)];
}

struct Filter5 { double w[8][8]; };

/* BoxAverage (Compute.cpp:495-605): filter over x-z of the array with the
 * wall row prepended, min(1, avg / density_threshold), inside the bbox. */
__global__ void k_box_average(int X, int Z, int FL, Filter5 f, double thr, const int* __restrict__ bbox,
                              const double* __restrict__ rough, const double* __restrict__ rough_wall,
                              double* __restrict__ out, double* __restrict__ out_wall)
{
    int minx = bbox[0], maxx = bbox[1], maxz = bbox[2];
    int ia = minx + blockIdx.x * blockDim.x + threadIdx.x;
    int ka = blockIdx.y;
    const int FD = FL / 2;
    if (minx - FD < 0 || maxx + FD > X || maxz + FD > Z) return;   /* reported by k_bbox_finish */
    if (ia >= maxx || ka > maxz) return;
    double a = 0.0;
    for (int fi = -FD; fi <= FD; fi++)
        for (int fk = -FD; fk <= FD; fk++) {
            int i = ia + fi, k = ka + fk;
            double w = f.w[fi + FD][fk + FD];
            if (k < 0) {
                double in0 = rough_wall[i];
                if (in0 > 0.00001) a += w * 1.0;
                else a += w * in0;
            } else {
                double in = (k == 0) ? rough_wall[i] : rough[IX(i, k - 1)];
                a += w * in;
            }
        }
    double v = dmin_(1.0, a / thr);
    if (ka == 0) out_wall[ia] = v;
    else if (ka - 1 < Z) out[IX(ia, ka - 1)] = v;
}

/* Height_Average (Compute.cpp:669-705) */
__global__ void k_height_average(int rgh, int xh, const int* __restrict__ bbox, const double* __restrict__ in, double* __restrict__ out)
{
    int i = bbox[0] * rgh + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (bbox[1] + 1) * rgh || i < 1 || i > xh - 2) return;
    double H0 = in[i], Ht = H0;
    int count = 1;
    double H = in[i - 1];
    if (H < H0) { Ht += H; count++; }
    H = in[i + 1];
    if (H < H0) { Ht += H; count++; }
    out[i] = Ht / count;
}
/* Smooth (Compute.cpp:708-738) with the 1/FilterLen box filter */
__global__ void k_smooth(int rgh, int xh, int FL, double w, const int* __restrict__ bbox, const double* __restrict__ in, double* __restrict__ out)
{
    int i = bbox[0] * rgh + blockIdx.x * blockDim.x + threadIdx.x;
    int FD = FL / 2;
    if (i >= (bbox[1] + 1) * rgh || i - FD < 0 || i + FD > xh - 1) return;
    double a = 0.0;
    for (int f = -FD; f <= FD; f++) a += w * in[i + f];
    out[i] = a;
}
/* GetSurfaceNormal (Compute.cpp:466-491) */
__global__ void k_normal(int rgh, int xh, double box_length, const int* __restrict__ bbox, const double* __restrict__ h,
                         double* __restrict__ nx, double* __restrict__ ny, double* __restrict__ nz)
{
    int i = bbox[0] * rgh + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (bbox[1] + 1) * rgh || i < 1 || i > xh - 2) return;
    double d_x = (h[i + 1] - h[i - 1]) / (2.0 * box_length / rgh);
    double d_z = -1.0;
    double l_n = sqrt(d_x * d_x + d_z * d_z);
    nx[i] = d_x / l_n; ny[i] = 0; nz[i] = d_z / l_n;
}

static Filter5 make_filter(int FL)
{
    /* Filter3D of Simulation.cpp:87-110 */
    Filter5 f;
    double norm = 0;
    for (int ii = 0; ii < FL; ii++)
        for (int kk = 0; kk < FL; kk++)
            norm = norm + exp(-(ii - FL / 2) * (ii - FL / 2) - (kk - FL / 2) * (kk - FL / 2));
    for (int ii = 0; ii < FL; ii++)
        for (int kk = 0; kk < FL; kk++)
            f.w[ii][kk] = exp(-(ii - FL / 2) * (ii - FL / 2) - (kk - FL / 2) * (kk - FL / 2)) / norm;
    return f;
}

static int launch_surface(bcg_ctx* c, bool smooth)
{
    const bcg_params& P = c->P;
    const int rgh = P.refinement_grid_height;
    const int XH = P.box_x * rgh;
    unsigned g = (unsigned)((XH + 255) / 256);
    if (smooth) {
        k_height_average<<<g, 256, 0, c->stream>>>(rgh, XH, c->bbox, c->height, c->rough_height);
        k_smooth<<<g, 256, 0, c->stream>>>(rgh, XH, P.filter_len, 1.0 / (double)(P.filter_len), c->bbox, c->rough_height, c->height);
        c->launches += 2;
    }
    k_normal<<<g, 256, 0, c->stream>>>(rgh, XH, P.box_length, c->bbox, c->height, c->nrm_x, c->nrm_y, c->nrm_z);
    c->launches++;
    return cudaGetLastError() == cudaSuccess ? BCG_OK : BCG_E_CUDA;
}

static int deposit(bcg_ctx* c, bool smooth)
{
    const bcg_params& P = c->P;
    if (P.filter_len > 8 || P.refinement_grid_height > 8) return BCG_E_UNSUPPORTED;
    c->host_bbox[0] = -1;              /* until this deposition has ended well */
    timer_begin(c, BCG_T_DENSITY);
    int rc = bin_cells(c, c->cur);
    if (rc) return rc;
    const int X = P.box_x, Z = P.box_z;
    /* level 0's Res, if a caller asks for it, is worked out from the field as
     * the solve saw it: at a million boxes a column's row costs 2 us to keep, the
     * whole Res 70 */
    const bool keep = c->mg_res0_stale == 1;
    k_bbox_reset<<<(X + 127) / 128, 128, 0, c->stream>>>(c->bbox, X, Z, c->inside, keep ? c->res0_inside : nullptr);
    if (keep) c->mg_res0_stale = 2;
    k_get_density<<<X, COLUMN_THREADS, 0, c->stream>>>(X, Z, P.refinement_grid_height, P.box_length, P.cell_radius,
        c->rec[c->cur], c->box_start, c->box_ids, c->rd, c->inside, c->height, c->bbox);
    k_inside_ring<<<(X * Z + 255) / 256, 256, 0, c->stream>>>(X, Z, c->inside);
    k_bbox_finish<<<1, 32, 0, c->stream>>>(c->bbox, X, Z, P.filter_len / 2, c->status);
    k_shift<<<(X * Z + 255) / 256, 256, 0, c->stream>>>(X, Z, c->rd, c->rds, c->rws);
    Filter5 f = make_filter(P.filter_len);
    dim3 grid((X + 127) / 128, Z + 1);
    /* Density from RoughDensity (RoughWallDensity stays zero, ShiftDensity
     * never writes it) and DensityShiftP from RoughDensityShiftP */
    k_box_average<<<grid, 128, 0, c->stream>>>(X, Z, P.filter_len, f, P.density_threshold, c->bbox, c->rd, c->rw, c->dens, c->wd);
    k_box_average<<<grid, 128, 0, c->stream>>>(X, Z, P.filter_len, f, P.density_threshold, c->bbox, c->rds, c->rws, c->ds, c->wds);
    c->launches += 7;
    rc = launch_surface(c, smooth);
    if (rc) return rc;
    timer_end(c, BCG_T_DENSITY);
    return ctx_check_status_bbox(c);
}

extern "C" int bcg_update_density(bcg_ctx* c) { return c ? deposit(c, true) : BCG_E_ARG; }
extern "C" int bcg_initial_density(bcg_ctx* c) { return c ? deposit(c, false) : BCG_E_ARG; }

extern "C" int bcg_update_height(bcg_ctx* c)
{
    if (!c) return BCG_E_ARG;
    const bcg_params& P = c->P;
    if (P.refinement_grid_height > 8) return BCG_E_UNSUPPORTED;
    c->host_bbox[0] = -1;              /* the box follows the cells, insideColonyDen does not */
    timer_begin(c, BCG_T_DENSITY);
    int rc = bin_cells(c, c->cur);
    if (rc) return rc;
    const int X = P.box_x, Z = P.box_z;
    k_bbox_reset<<<1, 32, 0, c->stream>>>(c->bbox, X, Z, nullptr, nullptr);
    k_get_height<<<(X + 3) / 4, COLUMN_THREADS, 0, c->stream>>>(X, Z, P.refinement_grid_height, P.box_length, P.cell_radius,
        c->rec[c->cur], c->box_start, c->box_ids, c->height, c->bbox);
    k_bbox_finish<<<1, 32, 0, c->stream>>>(c->bbox, X, Z, P.filter_len / 2, c->status);
    c->launches += 3;
    rc = launch_surface(c, true);
    if (rc) return rc;
    timer_end(c, BCG_T_DENSITY);
    return ctx_check_status(c);
}

/*
 * mech.cu -- cell binning, neighbour lists, the mechanics step (MoveCell +
 * GrowCell) and the division loop, as sm_100a kernels.
 *
 * Reference: AgentBasedModel-BacColonyGrowth/ UniformGrid.h, Neighbours.cpp,
 * Forces.cpp, Integrate.cpp, grow.cpp, Cells.cpp, Simulation.cpp:330-413.
 */
#include "ctx.cuh"
#include "cellmath.cuh"
#include "internal.h"
#include <stddef.h>
#include <string.h>

/* ======================================================================= */
/* binning: counting sort of cell ids by UniformGrid address               */
/* ======================================================================= */
__global__ void k_bin_count(int n, const CellRec* __restrict__ rec, MechParams mp,
                            int* __restrict__ cell_box, int* __restrict__ slot,
                            int* __restrict__ box_cnt, DevStatus* st)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 a = rec[i].pL, b = rec[i].qR;
    V3 cm = avg_pq(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z));
    int xi, yi, zi;
    int box = box_address(cm, mp, xi, yi, zi);
    if (box < 0) { dev_error(st, BCG_E_OUT_OF_GRID, i); box = 0; }
    cell_box[i] = box;
    slot[i] = atomicAdd(&box_cnt[box], 1);
}

/* exclusive scan, 3 phases: per-block sums, scan of block sums, apply */
#define SCAN_BLOCK 1024
#define SCAN_ITEMS 4
__device__ __forceinline__ int block_excl_scan(int v, int* sh, int& total)
{
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) { int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = (lane < (blockDim.x >> 5)) ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) { int y = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += y; }
        sh[lane] = s;
    }
    __syncthreads();
    int pre = (wid > 0 ? sh[wid - 1] : 0) + x - v;
    total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return pre;
}
__global__ void k_scan_partial(int n, const int* __restrict__ in, int* __restrict__ block_sums)
{
    __shared__ int sh[32];
    long base = (long)blockIdx.x * SCAN_BLOCK * SCAN_ITEMS;
    int s = 0;
    for (int j = 0; j < SCAN_ITEMS; j++) {
        long idx = base + (long)threadIdx.x * SCAN_ITEMS + j;
        if (idx < n) s += in[idx];
    }
    int total;
    block_excl_scan(s, sh, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}
__global__ void k_scan_blocks(int nb, int* __restrict__ block_sums)
{
    __shared__ int sh[32];
    /* one block; nb <= SCAN_BLOCK * SCAN_ITEMS */
    int v[SCAN_ITEMS]; int s = 0;
    for (int j = 0; j < SCAN_ITEMS; j++) {
        int idx = threadIdx.x * SCAN_ITEMS + j;
        v[j] = idx < nb ? block_sums[idx] : 0;
        s += v[j];
    }
    int total;
    int pre = block_excl_scan(s, sh, total);
    for (int j = 0; j < SCAN_ITEMS; j++) {
        int idx = threadIdx.x * SCAN_ITEMS + j;
        if (idx < nb) block_sums[idx] = pre;
        pre += v[j];
    }
}
/* the whole scan in one block, for up to SCAN_SMALL boxes (6 us at 12800; the
 * three launches of the general form 12 and their gaps): tiles of 4 counts a
 * thread, all loaded before the first is scanned.  Both forms leave the counts 0 for the
 * next binning. */
#define SCAN_SMALL 32768
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_small(int n, int* __restrict__ in, int* __restrict__ out)
{
    __shared__ int sh[32];
    constexpr int TILE = SCAN_BLOCK * SCAN_ITEMS, TILES = SCAN_SMALL / TILE;
    int4 v[TILES];
    const int at = threadIdx.x * SCAN_ITEMS;
#pragma unroll
    for (int t = 0; t < TILES; t++) {
        const int i = t * TILE + at;
        v[t] = make_int4(0, 0, 0, 0);
        if (i + 3 < n) v[t] = *reinterpret_cast<const int4*>(in + i);
        else { if (i < n) v[t].x = in[i]; if (i + 1 < n) v[t].y = in[i + 1]; if (i + 2 < n) v[t].z = in[i + 2]; }
    }
    int carry = 0;
#pragma unroll
    for (int t = 0; t < TILES; t++) {
        if (t * TILE >= n) break;
        int total;
        const int i = t * TILE + at, a = carry + block_excl_scan(v[t].x + v[t].y + v[t].z + v[t].w, sh, total);
        const int4 o = make_int4(a, a + v[t].x, a + v[t].x + v[t].y, a + v[t].x + v[t].y + v[t].z);
        if (i + 3 < n) { *reinterpret_cast<int4*>(out + i) = o; *reinterpret_cast<int4*>(in + i) = make_int4(0, 0, 0, 0); }
        else {
            if (i < n) { out[i] = o.x; in[i] = 0; }
            if (i + 1 < n) { out[i + 1] = o.y; in[i + 1] = 0; }
            if (i + 2 < n) { out[i + 2] = o.z; in[i + 2] = 0; }
        }
        carry += total;
    }
    if (threadIdx.x == 0) out[n] = carry;
}
__global__ void k_scan_apply(int n, int* __restrict__ in, const int* __restrict__ block_sums, int* __restrict__ out)
{
    __shared__ int sh[32];
    long base = (long)blockIdx.x * SCAN_BLOCK * SCAN_ITEMS;
    int v[SCAN_ITEMS]; int s = 0;
    for (int j = 0; j < SCAN_ITEMS; j++) {
        long idx = base + (long)threadIdx.x * SCAN_ITEMS + j;
        v[j] = idx < n ? in[idx] : 0;
        s += v[j];
    }
    int total;
    int pre = block_excl_scan(s, sh, total) + block_sums[blockIdx.x];
    for (int j = 0; j < SCAN_ITEMS; j++) {
        long idx = base + (long)threadIdx.x * SCAN_ITEMS + j;
        if (idx < n) { out[idx] = pre; in[idx] = 0; }
        pre += v[j];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = pre;
}

__global__ void k_bin_scatter(int n, const int* __restrict__ cell_box, const int* __restrict__ slot,
                              const int* __restrict__ box_start, int* __restrict__ box_ids)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    box_ids[box_start[cell_box[i]] + slot[i]] = i;
}

/* ascending ids inside each box (boxes hold at most max_cells_per_box - 1) */
__global__ void k_bin_sort(int nbox, const int* __restrict__ box_start, int* __restrict__ box_ids,
                           int box_cap, DevStatus* st)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbox) return;
    int s = box_start[b], e = box_start[b + 1];
    /* an overfull box is an error (UniformGrid.h:35); leave it unsorted so
     * that the work of this thread stays bounded */
    if (e - s > box_cap - 1) { dev_error(st, BCG_E_BOX_OVERFLOW, b); return; }
    for (int i = s + 1; i < e; i++) {
        int v = box_ids[i], j = i - 1;
        while (j >= s && box_ids[j] > v) { box_ids[j + 1] = box_ids[j]; j--; }
        box_ids[j + 1] = v;
    }
}

static int scan_exclusive(bcg_ctx* c, int* in, int* out, int n)
{
    if (n <= SCAN_SMALL) {
        k_scan_small<<<1, SCAN_BLOCK, 0, c->stream>>>(n, in, out);
        c->launches++;
        return BCG_OK;
    }
    int nb = (n + SCAN_BLOCK * SCAN_ITEMS - 1) / (SCAN_BLOCK * SCAN_ITEMS);
    if (nb < 1) nb = 1;
    if (nb > SCAN_BLOCK * SCAN_ITEMS) return BCG_E_ARG;
    k_scan_partial<<<nb, SCAN_BLOCK, 0, c->stream>>>(n, in, c->scan_tmp);
    k_scan_blocks<<<1, SCAN_BLOCK, 0, c->stream>>>(nb, c->scan_tmp);
    k_scan_apply<<<nb, SCAN_BLOCK, 0, c->stream>>>(n, in, c->scan_tmp, out);
    c->launches += 3;
    return BCG_OK;
}

/* bin the cells of record buffer `buf` (c->cell_box, box_start, box_ids) */
int bin_cells(bcg_ctx* c, int buf)
{
    MechParams mp = mech_params(c);
    int n = c->n;
    int* slot = c->delta_ids;   /* scratch: cap ints, unused outside divisions */
    if (n > 0) {
        k_bin_count<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->rec[buf], mp, c->cell_box, slot, c->box_cnt, c->status);
        c->launches++;
    }
    int rc = scan_exclusive(c, c->box_cnt, c->box_start, c->nbox);
    if (rc) return rc;
    if (n > 0) {
        k_bin_scatter<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->cell_box, slot, c->box_start, c->box_ids);
        c->launches++;
    }
    k_bin_sort<<<(c->nbox + 255) / 256, 256, 0, c->stream>>>(c->nbox, c->box_start, c->box_ids, c->P.max_cells_per_box, c->status);
    c->launches++;
    c->n_binned = n;
    BCG_CUDA_TRY(cudaGetLastError());
    return BCG_OK;
}

/* ======================================================================= */
/* neighbour lists                                                          */
/* ======================================================================= */
/* Rebuild the reduced list of cell `me` with L lanes of a warp: gather the
 * 3x3x3 box stencil (UniformGrid.h:141-170, z outer, y, x inner), apply the
 * reduceNeighbours filter (Neighbours.cpp:57-93).  Candidates come from the
 * bins; when `moved` is given, binned cells flagged as moved are skipped
 * and the (ids, boxes) of the delta list are gathered instead (they follow
 * the binned cells of their box).
 *
 * The warp's groups run the same trips (whole-warp collectives).  Each lane
 * writes the ids of its boxes to the group's list in shared memory, where the
 * candidates are then read side by side: to find a candidate's box by shuffles
 * cost more instructions than the test itself (all lists of 262144 cells: 440 us
 * with 32 lanes a cell and shuffles, 248 so). */
#define REBUILD_LIST 64
template <int L, bool COH>
__device__ __forceinline__ void rebuild_list(int me, int* __restrict__ cand, const CellRec* rec, const MechParams& mp,
                                 const int* __restrict__ box_start, const int* __restrict__ box_ids,
                                 const int* moved, const int* delta_ids,
                                 const int* delta_box, int ndelta,
                                 int* nbr, int* ncount, DevStatus* st)
{
    constexpr int PER = (27 + L - 1) / L;
    const unsigned all = 0xffffffffu, DELTA = 0x80000000u;
    const int lane = threadIdx.x & 31, gl = lane & (L - 1), g0 = lane & ~(L - 1);
    const bool valid = me >= 0;
    Cst a = COH ? load_cst_coh(&rec[valid ? me : 0]) : load_cst(&rec[valid ? me : 0]);
    V3 acm = avg_pq(a.p, a.q);
    int xi, yi, zi;
    int abox = box_address(acm, mp, xi, yi, zi);
    const bool here = valid && abox >= 0;
    if (valid && abox < 0 && gl == 0) dev_error(st, BCG_E_OUT_OF_GRID, me);
    int* out = nbr + (size_t)me * mp.kmax;
    const int YZ = mp.box_y * mp.box_z;
    /* the stencil's boxes in scan order, `per` a lane side by side; layers of
     * y off the grid (all but one where the grid has one) are not counted */
    const int y0 = max(yi - 1, 0), ny = min(yi + 1, mp.box_y - 1) - y0 + 1;
    const int nb = here ? 9 * ny : 0, per = (nb + L - 1) / L;
    int box[PER], bs[PER], num[PER], tot_i = 0;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int q = gl * per + i;
        box[i] = -1; bs[i] = 0; num[i] = 0;
        if (i < per && q < nb) {
            const int za = zi - 1 + q / (3 * ny), ya = y0 + (q / 3) % ny, xa = xi - 1 + q % 3;
            if (za >= 0 && za < mp.box_z && xa >= 0 && xa < mp.box_x) {
                const int b = xa * YZ + ya * mp.box_z + za;
                box[i] = b;
                bs[i] = box_start[b];
                num[i] = min(box_start[b + 1] - bs[i], mp.box_cap);   /* overfull: error already raised by the binning */
                tot_i += num[i];
                for (int t = 0; t < ndelta; t++) tot_i += (delta_box[t] == b);
            }
        }
    }
    /* exclusive prefix of the lanes' candidate counts */
    int incl = tot_i;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
        const int v = __shfl_up_sync(all, incl, o, L);
        if (gl >= o) incl += v;
    }
    const int off = incl - tot_i;
    const int total = __shfl_sync(all, incl, L - 1, L);
    const int most = L == 32 ? total : __reduce_max_sync(all, total);
    int cnt = 0;
    for (int w0 = 0; w0 < most; w0 += REBUILD_LIST) {
        int at = off - w0;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            for (int k = 0; k < num[i]; k++, at++)
                if (at >= 0 && at < REBUILD_LIST) cand[at] = box_ids[bs[i] + k];
            if (box[i] >= 0)
                for (int t = 0; t < ndelta; t++)
                    if (delta_box[t] == box[i]) {
                        if (at >= 0 && at < REBUILD_LIST) cand[at] = (int)((unsigned)delta_ids[t] | DELTA);
                        at++;
                    }
        }
        __syncwarp();
        const int end = min(most - w0, REBUILD_LIST);
        for (int t0 = 0; t0 < end; t0 += L) {
            bool keep = false;
            int j = -1;
            if (w0 + t0 + gl < total) {
                const unsigned e = (unsigned)cand[t0 + gl];
                j = (int)(e & ~DELTA);
                if (j != me && ((e & DELTA) || !(moved && moved[j]))) {
                    Cst bj = COH ? load_cst_coh(&rec[j]) : load_cst(&rec[j]);
                    keep = keep_neighbour(a.p, a.q, a.L, a.R, acm, bj.p, bj.q, mp.rc);
                }
            }
            const unsigned m = (__ballot_sync(all, keep) >> g0) & (L == 32 ? all : (1u << (L & 31)) - 1);
            const int pos = cnt + __popc(m & ((1u << gl) - 1));
            if (keep && pos < mp.kmax) out[pos] = j;
            cnt += __popc(m);
        }
        __syncwarp();
    }
    if (here && gl == 0) {
        if (cnt > mp.kmax) { dev_error(st, BCG_E_NEIGH_OVERFLOW, me); cnt = mp.kmax; }
        ncount[me] = cnt;
    }
}

/* Eight lanes a cell: nine boxes (one layer in y) of a few cells each are 30 to
 * 50 candidates, which leave less of the last trip idle than on 32 lanes, and
 * four cells share what a warp does once. */
#define REBUILD_LANES 8
#define REBUILD_THREADS 128
__global__ void __launch_bounds__(REBUILD_THREADS) k_rebuild_all(int n, const CellRec* __restrict__ rec, MechParams mp,
                              const int* __restrict__ box_start, const int* __restrict__ box_ids,
                              int* __restrict__ nbr, int* __restrict__ ncount, DevStatus* st)
{
    __shared__ int cand[REBUILD_THREADS / REBUILD_LANES][REBUILD_LIST];
    const int w = (blockIdx.x * REBUILD_THREADS + threadIdx.x) / REBUILD_LANES;
    /* walk the cells in bin order so that consecutive groups share boxes */
    rebuild_list<REBUILD_LANES, false>(w < n ? box_ids[w] : -1, cand[threadIdx.x / REBUILD_LANES], rec, mp, box_start, box_ids,
                                       nullptr, nullptr, nullptr, 0, nbr, ncount, st);
}

extern "C" int bcg_rebuild_neighbours(bcg_ctx* c)
{
    if (!c) return BCG_E_ARG;
    timer_begin(c, BCG_T_NEIGHBOURS);
    int rc = bin_cells(c, c->cur);
    if (rc) return rc;
    if (c->n > 0) {
        const long lanes = (long)c->n * REBUILD_LANES;
        k_rebuild_all<<<(unsigned)((lanes + REBUILD_THREADS - 1) / REBUILD_THREADS), REBUILD_THREADS, 0, c->stream>>>(
            c->n, c->rec[c->cur], mech_params(c), c->box_start, c->box_ids, c->nbr, c->ncount, c->status);
        c->launches++;
    }
    BCG_CUDA_TRY(cudaGetLastError());
    timer_end(c, BCG_T_NEIGHBOURS);
    return BCG_OK;
}

/* ======================================================================= */
/* MoveCell + GrowCell                                                      */
/* ======================================================================= */
/* STAGED (one lane per cell): the neighbours' records pass through shared memory.
 * A lane that gathers its own neighbour's 128 bytes touches a line of its own
 * with each of eight loads and waits for them; here the warp fetches its 32
 * neighbours together, eight lanes a record, asynchronously, the next neighbour
 * while it works on this one.  A record's 16-byte pieces are rotated by its lane,
 * so that the lanes' reads of one piece meet no bank twice.  Two slots a warp.
 * The cells' own records come and go the same way.
 *
 * The copies pass L1 by, which serves a gathered record to several lanes, and
 * cost instructions; they gain where a few waves of blocks leave the first loads
 * unhidden and lose on larger colonies.  A launch of a dense colony (6
 * neighbours) within its steps, us, one lane a cell, 4 blocks an SM:
 *   cells             45000  80000  131072  200000  225000  262144  1048576
 *   FP64 staged          48     77      95     143     162     188      647
 *        gathered        50     81      99     137     145     173      557
 *   FP32 staged          57     91     121     199     229     270     1038
 *        gathered        58     91     112     165     190     220      797
 * (with 3 blocks an SM staged 177 and 577 at 262144 and 1048576 cells, FP64).  A
 * loose colony (2 neighbours) crosses at the same sizes: 74 and 75 us at
 * 200000 cells, FP64.  In launches on a standing colony the staged form had looked
 * the faster one at 262144 cells too (145 us, gathered 167). */
#define STAGE_BYTES (32 * 128)
#define STAGE_CELLS 200000           /* largest colony that is staged */
#define STAGE_CELLS_F32 100000       /* ... with the FP32 contact search */
__device__ __forceinline__ void stage_fetch(unsigned char* slot, const CellRec* __restrict__ rec, int id)
{
    const int lane = threadIdx.x & 31, piece = lane & 7;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int who = (lane >> 3) + 4 * r, nid = __shfl_sync(0xffffffffu, id, who);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(slot + who * 128 + ((piece ^ (who & 7)) << 4));
        if (nid >= 0)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(reinterpret_cast<const unsigned char*>(rec + nid) + piece * 16));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
/* one lane's record as eight pieces, and the warp's store of its 32 records */
__device__ __forceinline__ void stage_store(unsigned char* slot, CellRec* __restrict__ rec, int id, const CellRec& r)
{
    const int lane = threadIdx.x & 31, piece = lane & 7;
    const double2 p[8] = {make_double2(r.pL.x, r.pL.y), make_double2(r.pL.z, r.pL.w), make_double2(r.qR.x, r.qR.y), make_double2(r.qR.z, r.qR.w),
                          make_double2(r.v.x, r.v.y), make_double2(r.v.z, r.v.w), make_double2(r.w.x, r.w.y), make_double2(r.w.z, r.w.w)};
#pragma unroll
    for (int i = 0; i < 8; i++) *reinterpret_cast<double2*>(slot + lane * 128 + ((i ^ piece) << 4)) = p[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int who = (lane >> 3) + 4 * i, nid = __shfl_sync(0xffffffffu, id, who);
        if (nid >= 0)
            reinterpret_cast<double2*>(rec + nid)[piece] = *reinterpret_cast<const double2*>(slot + who * 128 + ((piece ^ (who & 7)) << 4));
    }
}
__device__ __forceinline__ Cst stage_read(const unsigned char* slot)
{
    const int lane = threadIdx.x & 31, x = lane & 7;
    const unsigned char* r = slot + lane * 128;
    auto at = [&](int piece) { return *reinterpret_cast<const double2*>(r + ((piece ^ x) << 4)); };
    const double2 a0 = at(0), a1 = at(1), b0 = at(2), b1 = at(3), c0 = at(4), c1 = at(5), d0 = at(6), d1 = at(7);
    Cst s;
    s.p = mk(a0.x, a0.y, a1.x); s.L = a1.y;
    s.q = mk(b0.x, b0.y, b1.x); s.R = b1.y;
    s.v = mk(c0.x, c0.y, c1.x); s.w = mk(d0.x, d0.y, d1.x);
    return s;
}

/* Forces on `a` from its neighbour list (lanes of a G-wide group split the
 * list; the group reduces with a fixed butterfly), plus the wall, drag and
 * surface-tension terms (sum_forces, Forces.cpp:332-381). */
template <int G, bool GEOM32, bool STAGED>
__device__ __forceinline__ void sum_forces_group(const Cst& a, int me, const CellRec* __restrict__ old,
                                                 const int* __restrict__ list, int cnt, double wall_z,
                                                 const FieldPtrs& fp, const MechParams& mp,
                                                 V3& Fnet, V3& Tnet, V3& sf, V3& df, int& near_wall, unsigned char* stage, bool again)
{
    const int gl = threadIdx.x & (G - 1);
    V3 cm = avg_pq(a.p, a.q);
    V3 F = mk(0, 0, 0), T = mk(0, 0, 0);
    if (STAGED) {
        /* the caller has fetched the first neighbours into slot 0 */
        const int most = __reduce_max_sync(0xffffffffu, cnt);
        int next = 1 < cnt ? __ldg(&list[1]) : -1;
        for (int j = 0; j < most; j++) {
            stage_fetch(stage + ((j + 1) & 1) * STAGE_BYTES, old, next);
            next = j + 2 < cnt ? __ldg(&list[j + 2]) : -1;
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            if (j < cnt) {
                const Cst b = stage_read(stage + (j & 1) * STAGE_BYTES);
                V3 f, r;
                if (GEOM32 ? pair_force_f32geom(a, cm, b, mp, f, r) : pair_force(a, cm, b, mp, f, r)) {
                    F = add3(F, f);
                    T = add3(T, cross3(sub3(r, cm), f));
                }
            }
            __syncwarp();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        /* the next pass begins with the same neighbours */
        if (again) stage_fetch(stage, old, 0 < cnt ? __ldg(&list[0]) : -1);
    } else for (int j = gl; j < cnt; j += G) {
        int id = __ldg(&list[j]);
        Cst b = load_cst(&old[id]);
        V3 f, r;
        if (GEOM32 ? pair_force_f32geom(a, cm, b, mp, f, r) : pair_force(a, cm, b, mp, f, r)) {
            F = add3(F, f);
            T = add3(T, cross3(sub3(r, cm), f));
        }
    }
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) {
        F.x += __shfl_xor_sync(0xffffffffu, F.x, o); F.y += __shfl_xor_sync(0xffffffffu, F.y, o);
        F.z += __shfl_xor_sync(0xffffffffu, F.z, o); T.x += __shfl_xor_sync(0xffffffffu, T.x, o);
        T.y += __shfl_xor_sync(0xffffffffu, T.y, o); T.z += __shfl_xor_sync(0xffffffffu, T.z, o);
    }
    sf = mk(0, 0, 0); df = mk(0, 0, 0);
    near_wall = dmin_(a.q.z, a.p.z) < 1.2 * a.R;
    if (near_wall) {
        V3 r1, r2;
        V3 F1 = wall_locus(a, cm, a.p, wall_z, mp, r1, sf, df);
        V3 F2 = wall_locus(a, cm, a.q, wall_z, mp, r2, sf, df);
        F = add3(F, F1); T = add3(T, cross3(sub3(r1, cm), F1));
        F = add3(F, F2); T = add3(T, cross3(sub3(r2, cm), F2));
    }
    /* F_v, Forces.cpp:320-329 */
    F = add3(F, scl3(a.v, -mp.viscosity * 6.0 * BCG_PI * a.R));
    T = add3(T, scl3(a.w, -mp.viscosity * 6.0 * BCG_PI * a.R));
    V3 Fs, Ts;
    surface_tension(a, cm, fp, mp, Fs, Ts);
    F = add3(F, Fs); T = add3(T, Ts);
    T.z = 0; F.y = 0;
    Fnet = F; Tnet = T;
}

/* MB = the blocks of 128 threads an SM is to hold: 4 caps the registers at
 * 128 (some spill), 3 at 170 (none spill); the autotuner picks. */
template <int G, bool GEOM32, int MB, bool STAGED>
__global__ void __launch_bounds__(128, MB) k_move_grow(int n, int nbinned, const int* __restrict__ order,
        const CellRec* __restrict__ old, CellRec* __restrict__ nw,
        const int* __restrict__ nbr, const int* __restrict__ ncount,
        CellSoA soa, FieldPtrs fp, MechParams mp, double dt,
        int* __restrict__ div_list, DevStep* step, DevStep* host)
{
    DevStatus* st = &step->status;
    int t = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int gl = threadIdx.x & (G - 1);
    /* Lanes past the last cell run the body on cell 0 and write nothing:
     * the group reduction is a full-warp shuffle, so every lane of the
     * warp has to reach it (n > 0 at every launch). */
    const bool active = t < n;
    int me = active ? (t < nbinned ? __ldg(&order[t]) : t) : 0;
    int near1 = 0, near2 = 0;
    bool told = false;             /* this lane left something for the last block to read */
    static_assert(!STAGED || G == 1, "a staged record belongs to one lane");
    constexpr int SLOTS = STAGED ? 4 * 2 : 0;        /* two a warp of 128 threads */
    __shared__ __align__(128) unsigned char stages[SLOTS ? SLOTS * STAGE_BYTES : 16];
    unsigned char* stage = stages + (STAGED ? (threadIdx.x >> 5) * 2 * STAGE_BYTES : 0);
    {
        const int* list = nbr + (size_t)me * mp.kmax;
        const int cnt = active || !STAGED ? __ldg(&ncount[me]) : 0;
        Cst o;
        if (STAGED) {
            /* the cells' own records by the same way, then the first neighbours */
            stage_fetch(stage + STAGE_BYTES, old, me);
            stage_fetch(stage, old, cnt > 0 ? __ldg(&list[0]) : -1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            o = stage_read(stage + STAGE_BYTES);
            __syncwarp();
        } else o = load_cst(&old[me]);
        V3 ocm = avg_pq(o.p, o.q);
        int xi, yi, zi;
        int obox = box_address(ocm, mp, xi, yi, zi);
        if (obox < 0) { if (gl == 0 && active) { dev_error(st, BCG_E_OUT_OF_GRID, me); told = true; } xi = 0; yi = 0; }
        double wall_z = __ldg(&fp.wall[xi * mp.box_y + yi]);
        V3 F, T, sf, df;
        /* integrate, Integrate.cpp:11-32 */
        sum_forces_group<G, GEOM32, STAGED>(o, me, old, list, cnt, wall_z, fp, mp, F, T, sf, df, near1, stage, true);
        Cst tmp = o;
        half_kick(dt, F, T, o, tmp.v, tmp.w);
        V3 rcmp = sub3(o.p, ocm), rcmq = sub3(o.q, ocm);
        V3 vp = add3(tmp.v, cross3(tmp.w, rcmp)), vq = add3(tmp.v, cross3(tmp.w, rcmq));
        tmp.p = add3(o.p, scl3(vp, dt));
        tmp.q = add3(o.q, scl3(vq, dt));
        tmp.p.y = 0; tmp.q.y = 0;
        sum_forces_group<G, GEOM32, STAGED>(tmp, me, old, list, cnt, wall_z, fp, mp, F, T, sf, df, near2, stage, false);
        Cst nc = tmp;
        half_kick(dt, F, T, tmp, nc.v, nc.w);
        nc.v.y = 0;
        /* grow, grow.cpp:17-102 */
        V3 ncm = avg_pq(nc.p, nc.q);
        int nbox = box_address(ncm, mp, xi, yi, zi);
        if (nbox < 0) { if (gl == 0 && active) { dev_error(st, BCG_E_OUT_OF_GRID, me); told = true; } nbox = 0; }
        double g;
        if (mp.cross_feeding && __ldg(&soa.type[me]) != 1) g = __ldg(&fp.gr2[nbox]);
        else g = __ldg(&fp.gr1[nbox]);
        g = g * 1.5850;
        V3 v = sub3(nc.q, nc.p);
        double dL = nc.L * dt * g;
        V3 dv = scl3(v, dL * 0.5 / nc.L);
        nc.L += dL;
        nc.p = sub3(nc.p, dv);
        nc.q = add3(nc.q, dv);
        CellRec r;
        r.pL = make_double4(nc.p.x, nc.p.y, nc.p.z, nc.L);
        r.qR = make_double4(nc.q.x, nc.q.y, nc.q.z, nc.R);
        r.v = make_double4(nc.v.x, nc.v.y, nc.v.z, 0.0);
        r.w = make_double4(nc.w.x, nc.w.y, nc.w.z, 0.0);
        if (STAGED) stage_store(stage, nw, active ? me : -1, r);
        if (gl == 0 && active) {
            if (!STAGED) nw[me] = r;
            soa.gr[me] = g;
            soa.dfx[me] = df.x; soa.dfy[me] = df.y; soa.dfz[me] = df.z;
            soa.sfx[me] = sf.x; soa.sfy[me] = sf.y; soa.sfz[me] = sf.z;
            if (nc.L >= __ldg(&soa.ldiv[me])) {
                int k = atomicAdd(&step->div_count, 1);
                div_list[k] = me;
                told = true;
            }
            if (!isfinite(nc.p.x) || !isfinite(nc.p.z) || !isfinite(nc.q.x) || !isfinite(nc.q.z)) {
                dev_error(st, BCG_E_NAN, me);
                told = true;
            }
        }
    }
    /* F_cw calls (one rand() each, Forces.cpp:102): block-reduce then one atomic */
    unsigned long long calls = (active && gl == 0) ? (unsigned long long)(near1 + near2) : 0ull;
    for (int o = 16; o >= 1; o >>= 1) calls += __shfl_xor_sync(0xffffffffu, calls, o);
    __shared__ unsigned long long wsum[8];
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = calls;
    told = __syncthreads_or(told);
    if (threadIdx.x == 0) {
        unsigned long long s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += wsum[w];
        if (s) atomicAdd(&step->fcw, s);
        /* the last block hands the step's counters and the error word to the
         * host (pinned memory: no copies) and clears the counters.  A block
         * that changed none of them has nothing to publish: its fence would
         * wait for its records' stores and hold its place on the SM (at
         * 262144 cells, 16 lanes each, 24 us of 562). */
        if (told || s) __threadfence();
        if (atomicAdd(&step->blocks, 1u) == gridDim.x - 1) {
            __threadfence();
            volatile DevStep* d = step;
            volatile DevStep* h = host;
            h->status.code = d->status.code; h->status.info = d->status.info;
            h->div_count = d->div_count; h->fcw = d->fcw;
            d->div_count = 0; d->fcw = 0; d->blocks = 0;
            __threadfence_system();
        }
    }
}

/* lanes per cell in the force loop: the context's choice (bcg_autotune or
 * bcg_set_force_group), else as many (up to 8) as keep the launch in one wave
 * of 4 blocks of 128 on 148 SMs, and one where a lane a cell fills more than
 * that.  Below the line more lanes shorten the walk over a cell's neighbours;
 * above it they only add what each lane does again.  Dense colonies (6
 * neighbours) that stand still, one lane staged, us a launch:
 *   cells      1000  4096  16384  32768  65536  262144
 *   8 lanes    18.8  21.2   32.5   48.0   77.9   268
 *   4          21.0  21.4   26.9   40.5   61.1   191
 *   2          24.9  24.7   28.0   34.2   56.0   160
 *   1          31.0  32.0   31.9   34.8   42.9   134 */
static int force_group_of(const bcg_ctx* c)
{
    if (c->force_group) return c->force_group;
    int g = 8;
    while (g > 1 && (long)c->n * g > 148L * 4 * 128) g >>= 1;
    return g;
}
static int force_occ_of(const bcg_ctx* c) { return c->force_occ ? c->force_occ : 4; }
extern "C" int bcg_set_force_group(bcg_ctx* c, int g)
{
    if (!c || (g != 1 && g != 2 && g != 4 && g != 8 && g != 16)) return BCG_E_ARG;
    if (g != force_group_of(c)) nutrient_graphs_drop(c);
    c->force_group = g;
    return BCG_OK;
}

/* Cells are walked in the order of the last binning (spatially coherent,
 * so neighbouring groups share record lines in L1/L2); cells created after
 * that binning follow in id order. */
int launch_move_grow(bcg_ctx* c, double dt, int group, int occ)
{
    int n = c->n;
    if (n > 0) {
        MechParams mp = mech_params(c);
        FieldPtrs fp = field_ptrs(c);
        int nb = c->n_binned < n ? c->n_binned : n;
        const int threads = 128;
        long tot = (long)n * group;
        unsigned blocks = (unsigned)((tot + threads - 1) / threads);
        const CellRec* old = c->rec[c->cur];
        CellRec* nw = c->rec[c->cur ^ 1];
        const bool staged = n <= (c->pair_f32 ? STAGE_CELLS_F32 : STAGE_CELLS);
#define MG_ARGS(G, M, B, S) k_move_grow<G, M, B, S><<<blocks, threads, 0, c->stream>>>(n, nb, c->box_ids, old, nw, c->nbr, c->ncount, \
            c->soa, fp, mp, dt, c->div_list, c->step, c->step_host)
#define MG_GROUPS(M, B) switch (group) { \
            case 1: if (staged) MG_ARGS(1, M, B, true); else MG_ARGS(1, M, B, false); break; \
            case 2: MG_ARGS(2, M, B, false); break; case 4: MG_ARGS(4, M, B, false); break; \
            case 8: MG_ARGS(8, M, B, false); break; default: MG_ARGS(16, M, B, false); break; }
        if (c->pair_f32) { if (occ == 3) { MG_GROUPS(true, 3) } else { MG_GROUPS(true, 4) } }
        else { if (occ == 3) { MG_GROUPS(false, 3) } else { MG_GROUPS(false, 4) } }
#undef MG_GROUPS
#undef MG_ARGS
        c->launches++;
        BCG_CUDA_TRY(cudaGetLastError());
    }
    return BCG_OK;
}

/* split halves of bcg_move_grow (used by the ensemble runner to overlap
 * colonies): the launch, and the wait for what its last block hands over */
int move_grow_launch(bcg_ctx* c, double dt)
{
    return launch_move_grow(c, dt, force_group_of(c), force_occ_of(c));
}
int move_grow_finish(bcg_ctx* c, int* n_div, int64_t* fcw_calls)
{
    int rc;
    if (c->n > 0 && !c->pending_error) {
        BCG_CUDA_TRY(cudaStreamSynchronize(c->stream));
        rc = ctx_take_status(c);
    } else {
        c->step_host->div_count = 0;
        c->step_host->fcw = 0;
        rc = ctx_check_status(c);
    }
    if (rc) return rc;
    c->move_pending = 1;
    c->last_ndiv = c->step_host->div_count;
    if (n_div) *n_div = c->last_ndiv;
    if (fcw_calls) *fcw_calls = (int64_t)c->step_host->fcw;
    return BCG_OK;
}

extern "C" int bcg_move_grow(bcg_ctx* c, double dt, int* n_div, int64_t* fcw_calls)
{
    if (!c) return BCG_E_ARG;
    timer_begin(c, BCG_T_MOVE_GROW);
    int rc = launch_move_grow(c, dt, force_group_of(c), force_occ_of(c));
    if (rc) return rc;
    timer_end(c, BCG_T_MOVE_GROW);
    return move_grow_finish(c, n_div, fcw_calls);
}

/* time `reps` launches of MoveCell+GrowCell with `group` lanes per cell;
 * the records of the current buffer are read only, so the state is kept */
static int time_move_grow(bcg_ctx* c, int group, int occ, int reps, float* ms)
{
    cudaEvent_t a, b;
    BCG_CUDA_TRY(cudaEventCreate(&a));
    BCG_CUDA_TRY(cudaEventCreate(&b));
    int rc = launch_move_grow(c, c->P.dt, group, occ);      /* warm-up */
    if (!rc) rc = (cudaEventRecord(a, c->stream) == cudaSuccess) ? BCG_OK : BCG_E_CUDA;
    for (int r = 0; r < reps && !rc; r++) rc = launch_move_grow(c, c->P.dt, group, occ);
    if (!rc) rc = (cudaEventRecord(b, c->stream) == cudaSuccess) ? BCG_OK : BCG_E_CUDA;
    if (!rc) rc = (cudaEventSynchronize(b) == cudaSuccess) ? BCG_OK : BCG_E_CUDA;
    if (!rc) cudaEventElapsedTime(ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return rc;
}

extern "C" int bcg_set_pair_precision(bcg_ctx* c, int bits)
{
    if (!c || (bits != 32 && bits != 64)) return BCG_E_ARG;
    int f32 = bits == 32;
    if (f32 != c->pair_f32) { c->pair_f32 = f32; nutrient_graphs_drop(c); }
    return BCG_OK;
}

extern "C" int bcg_autotune(bcg_ctx* c, int what, int* choice)
{
    if (!c) return BCG_E_ARG;
    if (what == BCG_TUNE_SMOOTHER) return mg_tune_smoother(c, choice);
    if (what != BCG_TUNE_FORCE_GROUP) return BCG_E_ARG;
    if (c->n == 0) { if (choice) *choice = force_group_of(c); return BCG_OK; }
    const int saved_ndiv = c->last_ndiv;
    /* the trial launches rewrite the per-cell outputs of a step (growth
     * rate, friction accumulators): keep a copy and put it back */
    double* keep[7] = {c->soa.gr, c->soa.dfx, c->soa.dfy, c->soa.dfz, c->soa.sfx, c->soa.sfy, c->soa.sfz};
    const size_t nb = (size_t)c->n * sizeof(double);
    double* save = nullptr;
    BCG_CUDA_TRY(cudaMallocAsync((void**)&save, 7 * nb, c->stream));
    for (int a = 0; a < 7; a++)
        BCG_CUDA_TRY(cudaMemcpyAsync(save + a * (size_t)c->n, keep[a], nb, cudaMemcpyDeviceToDevice, c->stream));
    const int groups[5] = {1, 2, 4, 8, 16};
    float best = 3.4e38f;
    int best_g = force_group_of(c), best_o = force_occ_of(c);
    int rc = BCG_OK;
    for (int gi = 0; gi < 5 && !rc; gi++)
        for (int occ = 3; occ <= 4 && !rc; occ++) {
            float ms = 0;
            rc = time_move_grow(c, groups[gi], occ, 3, &ms);
            if (!rc && ms < best) { best = ms; best_g = groups[gi]; best_o = occ; }
        }
    for (int a = 0; a < 7; a++)
        cudaMemcpyAsync(keep[a], save + a * (size_t)c->n, nb, cudaMemcpyDeviceToDevice, c->stream);
    cudaFreeAsync(save, c->stream);
    int rc2 = ctx_check_status(c);
    c->last_ndiv = saved_ndiv;
    if (rc) return rc;
    if (rc2) return rc2;
    if (best_g != c->force_group || best_o != c->force_occ) { c->force_group = best_g; c->force_occ = best_o; nutrient_graphs_drop(c); }
    if (choice) *choice = best_g;
    return BCG_OK;
}

/* ======================================================================= */
/* division loop                                                            */
/* ======================================================================= */

/* divide(), grow.cpp:107-186, for mother m into daughter d; u[0..8] are the
 * nine (float)rand()/RAND_MAX draws in call order.  Reads the mother's
 * record, writes the SoA fields of both cells (no other division reads
 * them) and returns the two new records in out_m / out_d; the records are
 * stored in rec[] later, in division order. */
__device__ void divide_compute(int m, int d, const float* u, double t, const CellRec* rec, CellSoA soa,
                               const MechParams& mp, CellRec& out_m, CellRec& out_d)
{
    Cst M = load_cst(&rec[m]);
    double dl = ((double)u[0] - 0.5) * mp.var_l;
    double dangle = ((double)u[1] - 0.5) * mp.var_angle;
    V3 pq = sub3(M.p, M.q);
    V3 dd1 = mk((double)u[2] - 0.5, (double)u[3] - 0.5, (double)u[4] - 0.5);
    dd1 = sub3(dd1, scl3(pq, dot3(dd1, pq) / dot3(pq, pq)));
    dd1 = scl3(dd1, 1 / sqrt(dot3(dd1, dd1)));
    V3 dO1 = scl3(dd1, dangle);
    V3 dd2 = mk((double)u[5] - 0.5, (double)u[6] - 0.5, (double)u[7] - 0.5);
    dd2 = sub3(dd2, scl3(pq, dot3(dd2, pq) / dot3(pq, pq)));
    dd2 = scl3(dd2, 1 / sqrt(dot3(dd2, dd2)));
    V3 dO2 = scl3(dd2, dangle);
    V3 uv = sub3(M.p, M.q);
    double L = M.L;
    uv = scl3(uv, 1 / L);
    double dR = mp.cell_radius;
    double mL = L / 2 - M.R + dl;
    double dLen = L / 2 + M.R - 2 * dR - dl;
    V3 dq = M.q;
    V3 dw = mk(0, 0, ((double)u[8] - 0.5) * 0.001);
    V3 mq = sub3(M.p, scl3(uv, mL));
    double tq_m = soa.tq[m];
    V3 dp = sub3(mq, scl3(uv, dR + M.R));
    dq = sub3(dp, scl3(uv, dLen));
    V3 mp_ = add3(M.p, scl3(dO1, mL));
    mq = sub3(mq, scl3(dO1, mL));
    dp = add3(dp, scl3(dO2, dLen));
    dq = sub3(dq, scl3(dO2, dLen));
    CellRec rm, rd;
    rm.pL = make_double4(mp_.x, mp_.y, mp_.z, mL);
    rm.qR = make_double4(mq.x, mq.y, mq.z, M.R);
    rm.v = make_double4(M.v.x, M.v.y, M.v.z, 0.0);
    rm.w = make_double4(0.0, 0.0, 0.0, 0.0);
    rd.pL = make_double4(dp.x, dp.y, dp.z, dLen);
    rd.qR = make_double4(dq.x, dq.y, dq.z, dR);
    rd.v = make_double4(M.v.x, M.v.y, M.v.z, 0.0);
    rd.w = make_double4(dw.x, dw.y, dw.z, 0.0);
    out_m = rm;
    out_d = rd;
    soa.gr[d] = soa.gr[m];
    soa.tq[d] = tq_m;
    soa.tq[m] = t;
    soa.tp[d] = t;
    soa.ap[m] = soa.ap[m] + 1;
    soa.aq[d] = soa.aq[m] + 1;
    soa.ap[d] = 0;
    soa.dfx[d] = 0; soa.dfy[d] = 0; soa.dfz[d] = 0;
    soa.sfx[d] = 0; soa.sfy[d] = 0; soa.sfz[d] = 0;
    soa.type[d] = soa.type[m];
    soa.anc[d] = soa.anc[m];
    soa.ldiv[m] = mp.l_divide / 2 + mp.cell_radius + mL;
    soa.ldiv[d] = mp.l_divide / 2 + mp.cell_radius + dLen;
}

/* Simulation.cpp:380-404.  The reference divides the parents one after
 * another in ascending id order; each division moves the mother and adds
 * the daughter in the box structure and rebuilds the lists of {mother,
 * mother's neighbours, daughter} (Neighbours.cpp:39-55) against the state
 * left by the divisions before it.
 *
 * Here the divisions run as independent groups.  A division's footprint is
 * the rectangle of boxes, widened by 2, around the boxes of every cell whose
 * list it can rebuild (the mother before and after, her listed neighbours,
 * the daughter).  Every box a rebuild scans, and every box whose content
 * the division changes, lies inside it.  Divisions whose footprints overlap
 * are joined into one group (connected components), and a group runs its
 * divisions in ascending order on one block.  Divisions of different groups
 * neither change a box the other scans nor rebuild a common list, so the
 * lists come out as in the sequential loop.
 *
 * k_div_plan (one CTA): sort the parents, apply the reference's MaxCells
 * cut, compute all divisions' geometry (divide_compute; SoA fields written
 * here), footprints, groups (label propagation over the overlapping pairs,
 * then a sort by (group, division)), and the group-ordered division list.
 * k_div_groups (one block per group): store the records, mark the mother
 * moved, append both cells to the group's delta list, rebuild the lists. */
__global__ void __launch_bounds__(1024) k_div_plan(int n_start, int ndiv, int cap, double t,
        const float* __restrict__ draws, const CellRec* __restrict__ rec, CellSoA soa, MechParams mp,
        const int* __restrict__ div_list, const int* __restrict__ cell_box,
        const int* __restrict__ nbr, const int* __restrict__ ncount,
        CellRec* __restrict__ new_rec, int* __restrict__ new_box, int4* __restrict__ rect,
        int2* __restrict__ pairs, int* __restrict__ par_out, int* __restrict__ order, int* __restrict__ grp,
        int* __restrict__ lineage, int* __restrict__ lineage_host, int* __restrict__ out, DevStatus* st)
{
    /* dynamic shared memory: the sorted parents (later the group of each
     * root), the union-find parents, the groups' fill counters */
    extern __shared__ int div_smem[];
    int* sd = div_smem;
    int* par = div_smem + DIV_SORT_MAX;
    int* fill = div_smem + 2 * DIV_SORT_MAX;
    __shared__ int s_npairs;
    int P2 = 1;
    while (P2 < ndiv) P2 <<= 1;
    for (int i = threadIdx.x; i < P2; i += blockDim.x) sd[i] = i < ndiv ? div_list[i] : 0x7fffffff;
    if (threadIdx.x == 0) s_npairs = 0;
    __syncthreads();
    for (int k = 2; k <= P2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < P2; i += blockDim.x) {
                int ixj = i ^ j;
                if (ixj > i) {
                    int a = sd[i], b = sd[ixj];
                    bool up = (i & k) == 0;
                    if ((a > b) == up) { sd[i] = b; sd[ixj] = a; }
                }
            }
            __syncthreads();
        }
    /* the loop stops at the first division that would pass MaxCells */
    int nd = cap - n_start;
    if (nd < 0) nd = 0;
    if (nd > ndiv) nd = ndiv;
    if (nd < ndiv && threadIdx.x == 0) dev_error(st, BCG_E_MAXCELLS, nd);
    const int YZ = mp.box_y * mp.box_z;
    for (int d = threadIdx.x; d < nd; d += blockDim.x) {
        const int m = sd[d], N = n_start + d;
        CellRec rm, rd;
        divide_compute(m, N, draws + 9 * (size_t)d, t, rec, soa, mp, rm, rd);
        new_rec[2 * d] = rm; new_rec[2 * d + 1] = rd;
        int xi, yi, zi;
        int bm = box_address(avg_pq(mk(rm.pL.x, rm.pL.y, rm.pL.z), mk(rm.qR.x, rm.qR.y, rm.qR.z)), mp, xi, yi, zi);
        int bd = box_address(avg_pq(mk(rd.pL.x, rd.pL.y, rd.pL.z), mk(rd.qR.x, rd.qR.y, rd.qR.z)), mp, xi, yi, zi);
        if (bm < 0) { dev_error(st, BCG_E_OUT_OF_GRID, m); bm = 0; }
        if (bd < 0) { dev_error(st, BCG_E_OUT_OF_GRID, N); bd = 0; }
        new_box[2 * d] = bm; new_box[2 * d + 1] = bd;
        lineage[2 * d] = m; lineage[2 * d + 1] = N;
        *reinterpret_cast<int2*>(lineage_host + 2 * d) = make_int2(m, N);
        int b0 = cell_box[m];
        int x0 = b0 / YZ, z0 = b0 % mp.box_z;
        int xlo = x0, xhi = x0, zlo = z0, zhi = z0;
        int x = bm / YZ, z = bm % mp.box_z;
        xlo = min(xlo, x); xhi = max(xhi, x); zlo = min(zlo, z); zhi = max(zhi, z);
        x = bd / YZ; z = bd % mp.box_z;
        xlo = min(xlo, x); xhi = max(xhi, x); zlo = min(zlo, z); zhi = max(zhi, z);
        rect[d] = make_int4(xlo, xhi, zlo, zhi);
        par[d] = d;
    }
    __syncthreads();
    /* the boxes of the mother's listed neighbours, one warp per division,
     * then the footprint's margin of 2 boxes */
    {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
        for (int d = wid; d < nd; d += nw) {
            const int m = sd[d];
            const int cnt = ncount[m];
            int xlo = 0x7fffffff, xhi = -0x7fffffff, zlo = 0x7fffffff, zhi = -0x7fffffff;
            for (int j = lane; j < cnt; j += 32) {
                const int bb = cell_box[nbr[(size_t)m * mp.kmax + j]];
                const int x = bb / YZ, z = bb % mp.box_z;
                xlo = min(xlo, x); xhi = max(xhi, x); zlo = min(zlo, z); zhi = max(zhi, z);
            }
            for (int o = 16; o >= 1; o >>= 1) {
                xlo = min(xlo, __shfl_xor_sync(0xffffffffu, xlo, o));
                xhi = max(xhi, __shfl_xor_sync(0xffffffffu, xhi, o));
                zlo = min(zlo, __shfl_xor_sync(0xffffffffu, zlo, o));
                zhi = max(zhi, __shfl_xor_sync(0xffffffffu, zhi, o));
            }
            if (lane == 0) {
                int4 r = rect[d];
                r.x = min(r.x, xlo); r.y = max(r.y, xhi); r.z = min(r.z, zlo); r.w = max(r.w, zhi);
                rect[d] = make_int4(r.x - 2, r.y + 2, r.z - 2, r.w + 2);
            }
        }
    }
    __syncthreads();
    /* overlapping footprints */
    const int np2 = nd * nd;
    for (int q = threadIdx.x; q < np2; q += blockDim.x) {
        int a = q / nd, b = q - a * nd;
        if (a >= b) continue;
        int4 ra = rect[a], rb = rect[b];
        if (ra.x <= rb.y && rb.x <= ra.y && ra.z <= rb.w && rb.z <= ra.w) {
            int k = atomicAdd(&s_npairs, 1);
            if (k < DIV_PAIR_CAP) pairs[k] = make_int2(a, b);
        }
    }
    __syncthreads();
    const int npairs = s_npairs;
    if (npairs > DIV_PAIR_CAP) {
        /* too many overlaps to list: one sequential group */
        for (int d = threadIdx.x; d < nd; d += blockDim.x) par[d] = 0;
        __syncthreads();
    } else {
        /* connected components by label propagation: every division takes
         * the smallest label among the divisions its footprint overlaps,
         * then follows its label's label, until nothing changes; the label
         * ends as the smallest division of its component */
        for (;;) {
            __shared__ int s_changed;
            if (threadIdx.x == 0) s_changed = 0;
            __syncthreads();
            for (int k = threadIdx.x; k < npairs; k += blockDim.x) {
                const int a = pairs[k].x, b = pairs[k].y;
                const int la = par[a], lb = par[b];
                if (la != lb) {
                    const int lo = la < lb ? la : lb;
                    atomicMin(&par[a], lo);
                    atomicMin(&par[b], lo);
                    atomicMin(&par[la], lo);
                    atomicMin(&par[lb], lo);
                    s_changed = 1;
                }
            }
            __syncthreads();
            for (int d = threadIdx.x; d < nd; d += blockDim.x) {
                const int l = par[d], ll = par[l];
                if (ll < l) { atomicMin(&par[d], ll); s_changed = 1; }
            }
            __syncthreads();
            const int ch = s_changed;
            __syncthreads();
            if (!ch) break;
        }
    }
    /* groups in order of their first division, members ascending: sort the
     * keys (label, division) and cut the sorted list where the label
     * changes.  grp[2g] = start in order[], grp[2g+1] = length. */
    int P2n = 1;
    while (P2n < nd) P2n <<= 1;
    for (int i = threadIdx.x; i < P2n; i += blockDim.x) sd[i] = i < nd ? par[i] * DIV_SORT_MAX + i : 0x7fffffff;
    __syncthreads();
    for (int k = 2; k <= P2n; k <<= 1)
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            for (int i = threadIdx.x; i < P2n; i += blockDim.x) {
                int ixj = i ^ jj;
                if (ixj > i) {
                    int a = sd[i], b = sd[ixj];
                    bool up = (i & k) == 0;
                    if ((a > b) == up) { sd[i] = b; sd[ixj] = a; }
                }
            }
            __syncthreads();
        }
    /* fill[i] = 1 where a group starts, then its inclusive prefix sum */
    for (int i = threadIdx.x; i < P2n; i += blockDim.x)
        fill[i] = (i < nd && (i == 0 || sd[i] / DIV_SORT_MAX != sd[i - 1] / DIV_SORT_MAX)) ? 1 : 0;
    __syncthreads();
    for (int off = 1; off < P2n; off <<= 1) {
        int v[DIV_SORT_MAX / 1024];
        int c = 0;
        for (int i = threadIdx.x; i < P2n; i += blockDim.x) v[c++] = i >= off ? fill[i - off] : 0;
        __syncthreads();
        c = 0;
        for (int i = threadIdx.x; i < P2n; i += blockDim.x) fill[i] += v[c++];
        __syncthreads();
    }
    for (int i = threadIdx.x; i < nd; i += blockDim.x) {
        const int d = sd[i] - (sd[i] / DIV_SORT_MAX) * DIV_SORT_MAX;
        order[i] = d;
        const int g = fill[i] - 1;
        const bool start = i == 0 || sd[i] / DIV_SORT_MAX != sd[i - 1] / DIV_SORT_MAX;
        if (start) grp[2 * g] = i;
    }
    __syncthreads();
    /* the group's length, from its last member and its start */
    for (int i = threadIdx.x; i < nd; i += blockDim.x) {
        const bool last = i == nd - 1 || sd[i] / DIV_SORT_MAX != sd[i + 1] / DIV_SORT_MAX;
        if (last) {
            const int g = fill[i] - 1;
            grp[2 * g + 1] = i + 1 - grp[2 * g];
        }
    }
    if (threadIdx.x == 0) { out[0] = nd; out[1] = n_start + nd; out[2] = nd > 0 ? fill[nd - 1] : 0; }
    (void)par_out;
}

/* One block per group.  The group's divisions run in ascending order; the
 * lists one division rebuilds (the mother's, her listed neighbours', the
 * daughter's) each depend only on the records and the boxes, which the
 * rebuilds do not change, so the block's warps share them out. */
#define DIV_GROUP_WARPS 8
__global__ void __launch_bounds__(32 * DIV_GROUP_WARPS) k_div_groups(int n_start, const int* __restrict__ div_out,
        const int* __restrict__ grp, const int* __restrict__ order, const int* __restrict__ lineage,
        const CellRec* __restrict__ new_rec, const int* __restrict__ new_box,
        CellRec* rec, MechParams mp, int* nbr, int* ncount,
        const int* __restrict__ box_start, const int* __restrict__ box_ids,
        int* moved, int* delta_ids, int* delta_box, DevStatus* st)
{
    __shared__ int idl[1 + 1024 + 1];
    __shared__ int cand[DIV_GROUP_WARPS][REBUILD_LIST];
    const int w = threadIdx.x >> 5;
    const int g = blockIdx.x;
    if (g >= div_out[2]) return;                       /* whole block */
    const int gs = grp[2 * g], gl = grp[2 * g + 1];
    int* dids = delta_ids + 2 * gs;
    int* dbox = delta_box + 2 * gs;
    for (int j = 0; j < gl; j++) {
        const int d = order[gs + j];
        const int m = lineage[2 * d], N = n_start + d;
        /* the previous division's rebuilds are done (they may have written
         * this mother's list) before her records and list change hands */
        __syncthreads();
        if (threadIdx.x == 0) {
            rec[m] = new_rec[2 * d];
            rec[N] = new_rec[2 * d + 1];
            moved[m] = 1;
            dids[2 * j] = m; dbox[2 * j] = new_box[2 * d];
            dids[2 * j + 1] = N; dbox[2 * j + 1] = new_box[2 * d + 1];
        }
        const int cnt = ncount[m];
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) idl[1 + i] = nbr[(size_t)m * mp.kmax + i];
        if (threadIdx.x == 0) { idl[0] = m; idl[cnt + 1] = N; }
        /* every thread has read the mother's old list before a warp rewrites it */
        __syncthreads();
        for (int k = w; k < cnt + 2; k += DIV_GROUP_WARPS)
            rebuild_list<32, true>(idl[k], cand[w], rec, mp, box_start, box_ids, moved, dids, dbox, 2 * (j + 1), nbr, ncount, st);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < gl; j += blockDim.x) moved[lineage[2 * order[gs + j]]] = 0;
}

/* the division planner's shared memory: sorted parents, union-find
 * parents and group fill counters, DIV_SORT_MAX ints each */
int mech_kernel_attributes()
{
    /* set on every context creation: the attribute belongs to the current
     * device, and the call is cheap and thread-safe */
    if (cudaFuncSetAttribute(k_div_plan, cudaFuncAttributeMaxDynamicSharedMemorySize, DIV_PLAN_SMEM) != cudaSuccess)
        return BCG_E_CUDA;
    return BCG_OK;
}

extern "C" int bcg_get_dividing(bcg_ctx* c, int* ids, int capacity)
{
    if (!c || (!ids && capacity > 0)) return BCG_E_ARG;
    int n = c->last_ndiv < capacity ? c->last_ndiv : capacity;
    if (n > 0) {
        BCG_CUDA_TRY(cudaMemcpyAsync(ids, c->div_list, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost, c->stream));
        BCG_CUDA_TRY(cudaStreamSynchronize(c->stream));
        /* ascending, as the 1-thread reference collects them */
        for (int i = 1; i < n; i++) { int v = ids[i], j = i - 1; while (j >= 0 && ids[j] > v) { ids[j + 1] = ids[j]; j--; } ids[j + 1] = v; }
    }
    return BCG_OK;
}

/* split halves of bcg_divide: the launch queues the binning, the draw
 * upload, the two division kernels and the read of the counts; the
 * finish waits, copies the lineage and advances the context */
int divide_launch(bcg_ctx* c, const float* draws, int n_draw_sets, double t)
{
    if (n_draw_sets != c->last_ndiv) return BCG_E_ARG;
    const int ndiv = c->last_ndiv;
    if (ndiv > DIV_SORT_MAX) return BCG_E_UNSUPPORTED;
    if (ndiv == 0) return BCG_OK;
    if (!draws) return BCG_E_ARG;
    int nb = c->cur ^ 1;
    int rc = bin_cells(c, nb);
    if (rc) return rc;
    size_t db = sizeof(float) * 9 * (size_t)ndiv;
    rc = ensure_pinned(c, db + 64);
    if (rc) return rc;
    memcpy(c->pinned, draws, db);
    /* a few draws are read from the pinned memory as they are; more are worth
     * the copy, since the kernel's threads would fetch them word by word */
    const float* src = (const float*)c->pinned;
    if (ndiv > 64) {
        BCG_CUDA_TRY(cudaMemcpyAsync(c->draws_dev, c->pinned, db, cudaMemcpyHostToDevice, c->stream));
        src = c->draws_dev;
    }
    MechParams mp = mech_params(c);
    k_div_plan<<<1, 1024, DIV_PLAN_SMEM, c->stream>>>(c->n, ndiv, c->cap, t, src, c->rec[nb], c->soa, mp,
        c->div_list, c->cell_box, c->nbr, c->ncount, c->div_rec, c->div_box, c->div_rect, c->div_pairs,
        c->div_par, c->div_order, c->div_grp, c->lineage, c->lineage_host, c->step->n_done, c->status);
    k_div_groups<<<ndiv, 32 * DIV_GROUP_WARPS, 0, c->stream>>>(c->n, c->step->n_done, c->div_grp, c->div_order,
        c->lineage, c->div_rec, c->div_box, c->rec[nb], mp, c->nbr, c->ncount, c->box_start, c->box_ids,
        c->moved, c->delta_ids, c->delta_box, c->status);
    c->launches += 2;
    BCG_CUDA_TRY(cudaGetLastError());
    /* the error word and the counts, in one copy */
    BCG_CUDA_TRY(cudaMemcpyAsync(c->step_host, c->step, offsetof(DevStep, fcw), cudaMemcpyDeviceToHost, c->stream));
    return BCG_OK;
}
int divide_finish(bcg_ctx* c, int* n_done, int* lineage)
{
    const int ndiv = c->last_ndiv;
    int done = 0, rc = BCG_OK;
    if (ndiv > 0) {
        BCG_CUDA_TRY(cudaStreamSynchronize(c->stream));
        if (c->pending_error) rc = ctx_check_status(c);
        else rc = ctx_take_status(c);
        done = c->step_host->n_done[0];
        if (lineage && done > 0) memcpy(lineage, c->lineage_host, sizeof(int) * 2 * (size_t)done);
        c->n += done;
    }
    c->cur ^= 1;
    c->move_pending = 0;
    c->last_ndiv = 0;
    if (n_done) *n_done = done;
    return rc;
}

extern "C" int bcg_divide(bcg_ctx* c, const float* draws, int n_draw_sets, double t, int* n_done, int* lineage)
{
    if (!c) return BCG_E_ARG;
    timer_begin(c, BCG_T_DIVIDE);
    int rc = divide_launch(c, draws, n_draw_sets, t);
    if (rc) return rc;
    rc = divide_finish(c, n_done, lineage);
    timer_end(c, BCG_T_DIVIDE);
    return rc;
}

/* ======================================================================= */
/* mean_stress (Compute.cpp:18-117)                                         */
/* ======================================================================= */
__global__ void k_mean_stress(int n, const CellRec* __restrict__ rec, const int* __restrict__ nbr,
                              const int* __restrict__ ncount, FieldPtrs fp, MechParams mp,
                              double* __restrict__ stress, double* __restrict__ fnet,
                              unsigned long long* fcw_count, DevStatus* st)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int near = 0;
    if (i < n) {
        Cst c = load_cst(&rec[i]);
        double V = c.L * BCG_PI * c.R * c.R + 4.0 / 3.0 * BCG_PI * c.R * c.R * c.R;
        V3 CM = avg_pq(c.p, c.q);
        int xi, yi, zi;
        if (box_address(CM, mp, xi, yi, zi) < 0) { dev_error(st, BCG_E_OUT_OF_GRID, i); xi = 0; yi = 0; }
        double sxx = 0, syy = 0, szz = 0;
        V3 Fn = mk(0, 0, 0);
        const int* list = nbr + (size_t)i * mp.kmax;
        int cnt = ncount[i];
        for (int j = 0; j < cnt; j++) {
            Cst b = load_cst(&rec[list[j]]);
            V3 F, r;
            if (!pair_force(c, CM, b, mp, F, r)) { F = mk(0, 0, 0); continue; }
            Fn = add3(Fn, F);
            r = sub3(r, CM);
            sxx -= F.x * r.x; syy -= F.y * r.y; szz -= F.z * r.z;
        }
        if (dmin_(c.q.z, c.p.z) < 1.2 * c.R) {
            near = 1;
            double wall_z = fp.wall[xi * mp.box_y + yi];
            V3 r1, r2, sf = mk(0, 0, 0), df = mk(0, 0, 0);
            V3 F1 = wall_locus(c, CM, c.p, wall_z, mp, r1, sf, df);
            V3 F2 = wall_locus(c, CM, c.q, wall_z, mp, r2, sf, df);
            Fn = add3(Fn, F1);
            r1 = sub3(r1, CM);
            sxx -= F1.x * r1.x; syy -= F1.y * r1.y; szz -= F1.z * r1.z;
            Fn = add3(Fn, F2);
            r2 = sub3(r2, CM);
            sxx -= F2.x * r2.x; syy -= F2.y * r2.y; szz -= F2.z * r2.z;
        }
        V3 F, T;
        surface_tension(c, CM, fp, mp, F, T);
        Fn = add3(Fn, F);
        V3 r = sub3(c.p, CM); r.z += c.R;
        V3 r2 = sub3(c.q, CM); r2.z += c.R;
        sxx -= F.x * r.x * 0.5 - F.x * r2.x * 0.5;
        syy -= F.y * r.y * 0.5 - F.y * r2.y * 0.5;
        szz -= F.z * r.z * 0.5 - F.z * r2.z * 0.5;
        sxx /= V; syy /= V; szz /= V;
        double rr, tt;
        double Lcm = sqrt(CM.x * CM.x + CM.y * CM.y);
        if (Lcm > DBL_EPSILON) {
            V3 uv = scl3(CM, 1.0 / Lcm);
            rr = sxx * uv.x + syy * uv.y;
            tt = -sxx * uv.y + syy * uv.x;
        } else { rr = (sxx + syy); tt = 0.0; }
        stress[5 * (size_t)i + 0] = sxx; stress[5 * (size_t)i + 1] = syy; stress[5 * (size_t)i + 2] = szz;
        stress[5 * (size_t)i + 3] = rr; stress[5 * (size_t)i + 4] = tt;
        if (fnet) { fnet[3 * (size_t)i] = Fn.x; fnet[3 * (size_t)i + 1] = Fn.y; fnet[3 * (size_t)i + 2] = Fn.z; }
    }
    unsigned long long v = near;
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(fcw_count, v);
}

void launch_mean_stress(bcg_ctx* c, double* stress, unsigned long long* fcw, cudaStream_t s)
{
    if (c->n <= 0) return;
    k_mean_stress<<<(c->n + 127) / 128, 128, 0, s>>>(c->n, c->rec[c->cur], c->nbr, c->ncount, field_ptrs(c),
                                                     mech_params(c), stress, nullptr, fcw, c->status);
    c->launches++;
}

/* F_surf_tension's force on every cell (Forces.cpp:209-317), the cell
 * line's three force columns in the initial output block
 * (Simulation.cpp:229-238) */
__global__ void k_surface_force(int n, const CellRec* __restrict__ rec, FieldPtrs fp, MechParams mp,
                                double* __restrict__ force)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Cst c = load_cst(&rec[i]);
    V3 F, T;
    surface_tension(c, avg_pq(c.p, c.q), fp, mp, F, T);
    force[3 * (size_t)i] = F.x; force[3 * (size_t)i + 1] = F.y; force[3 * (size_t)i + 2] = F.z;
}

void launch_surface_force(bcg_ctx* c, double* force, cudaStream_t s)
{
    if (c->n <= 0) return;
    k_surface_force<<<(c->n + 127) / 128, 128, 0, s>>>(c->n, c->rec[c->cur], field_ptrs(c), mech_params(c), force);
    c->launches++;
}

extern "C" int bcg_mean_stress(bcg_ctx* c, double* stress, double* fnet, int64_t* fcw_calls)
{
    if (!c || !stress) return BCG_E_ARG;
    int n = c->n;
    BCG_CUDA_TRY(cudaMemsetAsync(c->fcw_count, 0, sizeof(unsigned long long), c->stream));
    if (n > 0) {
        double *ds = nullptr, *df = nullptr;
        BCG_CUDA_TRY(cudaMallocAsync((void**)&ds, sizeof(double) * 5 * (size_t)n, c->stream));
        if (fnet) BCG_CUDA_TRY(cudaMallocAsync((void**)&df, sizeof(double) * 3 * (size_t)n, c->stream));
        k_mean_stress<<<(n + 127) / 128, 128, 0, c->stream>>>(n, c->rec[c->cur], c->nbr, c->ncount, field_ptrs(c),
                                                              mech_params(c), ds, df, c->fcw_count, c->status);
        c->launches++;
        BCG_CUDA_TRY(cudaMemcpyAsync(stress, ds, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToHost, c->stream));
        if (fnet) BCG_CUDA_TRY(cudaMemcpyAsync(fnet, df, sizeof(double) * 3 * (size_t)n, cudaMemcpyDeviceToHost, c->stream));
        BCG_CUDA_TRY(cudaFreeAsync(ds, c->stream));
        if (df) BCG_CUDA_TRY(cudaFreeAsync(df, c->stream));
    }
    unsigned long long h = 0;
    BCG_CUDA_TRY(cudaMemcpyAsync(&h, c->fcw_count, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    int rc = ctx_check_status(c);
    if (fcw_calls) *fcw_calls = (int64_t)h;
    return rc;
}

/* ======================================================================= */
/* bcg_mean_stress_noalloc: the same kernel with its staging in a device   */
/* array compiled into the library (no allocation on any call)             */
/* ======================================================================= */
/* 5 stress + 3 force doubles per cell, then the F_cw counter */
static __device__ __align__(256) double g_noalloc_stress[8 * BCG_NOALLOC_MAX_CELLS + 32];

/* The array's device address on the current device.  Looked up on every
 * call rather than kept: the lookup allocates nothing, and an address kept
 * from before a cudaDeviceReset would point into a released context.  In
 * host code the array's name is only a host-side stand-in; kernels must be
 * given this address. */
static int noalloc_staging(double** out)
{
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_stress);
    if (e != cudaSuccess) { bcg_set_cuda_error(e); return BCG_E_CUDA; }
    *out = (double*)p;
    return BCG_OK;
}

extern "C" int bcg_mean_stress_noalloc(bcg_ctx* c, double* stress, double* fnet, int64_t* fcw_calls)
{
    if (!c || !stress) return BCG_E_ARG;
    const int n = c->n;
    if (n > BCG_NOALLOC_MAX_CELLS) return BCG_E_UNSUPPORTED;
    int dev = -1;
    BCG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev != c->device) return BCG_E_ARG;
    double* base = nullptr;
    int rc = noalloc_staging(&base);
    if (rc) return rc;
    double* ds = base;
    double* df = base + 5 * (size_t)BCG_NOALLOC_MAX_CELLS;
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(base + 8 * (size_t)BCG_NOALLOC_MAX_CELLS);
    /* the counter still holds the previous call's count */
    BCG_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(*cnt), c->stream));
    if (n > 0) {
        k_mean_stress<<<(n + 127) / 128, 128, 0, c->stream>>>(n, c->rec[c->cur], c->nbr, c->ncount, field_ptrs(c),
                                                              mech_params(c), ds, fnet ? df : nullptr, cnt, c->status);
        c->launches++;
        BCG_CUDA_TRY(cudaGetLastError());
        BCG_CUDA_TRY(cudaMemcpyAsync(stress, ds, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToHost, c->stream));
        if (fnet) BCG_CUDA_TRY(cudaMemcpyAsync(fnet, df, sizeof(double) * 3 * (size_t)n, cudaMemcpyDeviceToHost, c->stream));
    }
    unsigned long long h = 0;
    BCG_CUDA_TRY(cudaMemcpyAsync(&h, cnt, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    rc = ctx_check_status(c);
    if (fcw_calls) *fcw_calls = (int64_t)h;
    return rc;
}

extern "C" int bcg_int_move_grow_launch(bcg_ctx* c, double dt) { return c ? move_grow_launch(c, dt) : BCG_E_ARG; }
extern "C" int bcg_int_move_grow_finish(bcg_ctx* c, int* n_div, int64_t* fcw) { return c ? move_grow_finish(c, n_div, fcw) : BCG_E_ARG; }
extern "C" int bcg_int_divide_launch(bcg_ctx* c, const float* draws, int n, double t) { return c ? divide_launch(c, draws, n, t) : BCG_E_ARG; }
extern "C" int bcg_int_divide_finish(bcg_ctx* c, int* done, int* lineage) { return c ? divide_finish(c, done, lineage) : BCG_E_ARG; }


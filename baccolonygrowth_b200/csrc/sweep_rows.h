/*
 * sweep_rows.h -- the rows of a colony sweep's tiles (nutrients.cu): which
 * rows of the bounding box z = 0 .. maxz each row of tiles owns.  Every box row
 * has one owner.  Plain C++ so that the host, the kernels and a test on the CPU
 * share it.
 */
#ifndef BCG_SWEEP_ROWS_H
#define BCG_SWEEP_ROWS_H
#ifdef __CUDACC__
#define SW_FN __host__ __device__ __forceinline__
#else
#define SW_FN inline
#endif

#define SW_K 4               /* sweeps a launch, even: the buffers' roles return */
#define SW_RZ 40             /* rows of a tile with its halo */
#define SW_OWN0 (SW_RZ - 1 - SW_K)        /* rows z = 0 .. of the bottom tile where others follow */
#define SW_OWN (SW_RZ - 2 * SW_K)         /* rows of the tiles above it */

/* the box with one row of points above it, which no sweep writes, fits the
 * bottom tile: no tile above */
SW_FN bool sw_one_row(int maxz) { return maxz + 2 < SW_RZ; }
/* rows of tiles of a box */
SW_FN int sw_tile_rows(int maxz) { return sw_one_row(maxz) ? 1 : 1 + (maxz + 1 - SW_OWN0 + SW_OWN - 1) / SW_OWN; }
/* the points z0 <= z < z1 that row zt of the tiles owns */
SW_FN int sw_first(int zt) { return zt == 0 ? 0 : SW_OWN0 + (zt - 1) * SW_OWN; }
/* whether row zt has any (zt < sw_tile_rows(maxz), without its division) */
SW_FN bool sw_runs(int zt, int maxz) { return sw_first(zt) <= maxz && (zt == 0 || !sw_one_row(maxz)); }
SW_FN int sw_end(int zt, int maxz) { return zt > 0 ? sw_first(zt) + SW_OWN : sw_one_row(maxz) ? maxz + 1 : SW_OWN0; }
#endif

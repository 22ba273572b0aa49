// fx_plan.h — index maps and launch plans that need no CUDA: included by the kernels and the engine,
// and compiled by the host compiler alone in the CPU tests.
#pragma once

#ifdef __CUDACC__
#define FX_HOST_DEVICE __host__ __device__ inline
#else
#define FX_HOST_DEVICE inline
#endif

// Index of a plane or row outside 0 .. n - 1 reflected into it (-1 is 0, n is n - 1), for an index
// less than n outside.
FX_HOST_DEVICE int fx_zs_reflect(int q, int n) { return q < 0 ? -1 - q : (q >= n ? 2 * n - 1 - q : q); }

// Row of the grid that a strip tile's input row q is copied from (fx_jacobi_zs.cuh): rows below the
// floor are reflected, rows above the open top (q >= Y, whose values reach no stored cell) are
// the top row. q is -2 or more; a tile of few rows reaches far above the top of a flat grid.
FX_HOST_DEVICE int fx_zs_input_row(int q, int Y) { return q < 0 ? -1 - q : (q < Y ? q : Y - 1); }

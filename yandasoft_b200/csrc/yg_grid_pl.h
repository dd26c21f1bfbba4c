// Gridding over plane-major (k_grid_pl) and CF-major records (k_grid_cf).
#pragma once
#include "yg_internal.h"

namespace yg {

// How the plane-major kernel takes this CF table: 0, not at all (matrices of
// several sizes); n > 0, blocks of n consecutive matrices staged
// in shared memory; -n, planes of n matrices read through L1 / L2.  |n| is the
// number of matrices that the plane-major order treats as one CF plane.
int grid_pl_block(const CFView& cf, int os, int cf_mode, int npol);

// Whether plane-major records are the better choice where the order of a cell's
// sum is free (AWProject), and whether that depends on the samples per CF plane
// and cell (plan_samples_per_cell).
bool grid_pl_asks(const CFView& cf, int tile, int npol, int os, long long n);
bool grid_pl_better(const CFView& cf, int tile, int npol, int os, long long n, double per_cell);

// Grids the plane-major records of a plan (pl.rec_pos, pl.pl_fs).
int plan_grid_pl(const Plan& pl, const VisArgs& v, const CFView& cf, float2* grid, int nx, int ny, int nchan_img,
                 DevBuf& scratch, DevBuf& svis, DevError* err, cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1);

// CF-major gridding with exact residue widths (k_grid_cf): whether it is to grid
// n samples with the table at this tile side (k_grid grids the others), and a
// pass over the plan's CF-major records.
bool grid_cf_takes(const CFView& cf, int tile, int npol, int os, long long n);
int plan_grid_cf(const Plan& pl, const VisArgs& v, const CFView& cf, float2* grid, int nx, int ny, int nchan_img,
                 int os, DevBuf& scratch, DevBuf& svis, DevError* err, cudaStream_t st, cudaEvent_t ev0,
                 cudaEvent_t ev1);

}  // namespace yg

// Work distribution of the KEEP marches (keep_march_kernel), shared by the box
// lists and the allocation-free entry point.
#pragma once
#include "amrs_boxes.cuh"

namespace amrs {

// Columns of box R crossed by the march along dir (1 y, 2 z), in blocks of one
// warp, and the cells of a column.
__host__ __device__ inline int march_blocks(const BoxRec& R, int dir) {
  const int t = dir == 1 ? 2 : 1;
  return ((R.hi[0] - R.lo[0] + 1) * (R.hi[t] - R.lo[t] + 1) + 31) / 32;
}
__host__ __device__ inline int march_cells(const BoxRec& R, int dir) { return R.hi[dir] - R.lo[dir] + 1; }

// (Column block x cell) items of both marches of a box, in the order
// keep_march_kernel deals them to warps: y march, z march; block; cell.
inline long long march_items(const BoxRec& R) {
  return (long long)march_blocks(R, 1) * march_cells(R, 1) + (long long)march_blocks(R, 2) * march_cells(R, 2);
}

// Shares (warps) the items are cut into.  Every segment of a share pays a
// prologue of about one cell, so a share is a run of at least four cells on
// average (waves = 1; more waves: shorter runs) up to `waves` times the resident
// warps (two or eight cells: the same within 0.3% from 16^3 to 128^3).  While
// that leaves fewer than eight warps per SM the runs are cut shorter: 45 x 33 x
// 27 at order 6 takes 271 us per step so, 295 with four warps per SM, 316 with
// sixteen.
inline long long march_shares(long long items, int waves, long long resident, int nsm) {
  long long g = items * waves / 4;
  if (g > waves * resident) g = waves * resident;
  if (g < 8LL * nsm) g = 8LL * nsm;
  return g < items ? g : items;
}
// Warps per CTA: as many as give every SM a CTA, at most eight.
inline int march_cta_warps(long long shares, int nsm) {
  const long long w = shares / nsm;
  return w < 1 ? 1 : (w > 8 ? 8 : (int)w);
}

}  // namespace amrs

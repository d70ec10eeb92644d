// Balanced static schedule of the KEEP marches (keep_march_kernel), shared by
// the box lists and the allocation-free entry point.
#pragma once
#include "amrs_boxes.cuh"

namespace amrs {

// Columns of box R crossed by the march along dir (1 y, 2 z), in blocks of one
// warp, and the cells of a column.
inline int march_blocks(const BoxRec& R, int dir) {
  const int t = dir == 1 ? 2 : 1;
  return ((R.hi[0] - R.lo[0] + 1) * (R.hi[t] - R.lo[t] + 1) + 31) / 32;
}
inline int march_cells(const BoxRec& R, int dir) { return R.hi[dir] - R.lo[dir] + 1; }

// (Column block x cell) items of both marches over the boxes.
inline long long march_items(const BoxRec* box, int n) {
  long long s = 0;
  for (int b = 0; b < n; ++b)
    for (int d = 1; d <= 2; ++d) s += (long long)march_blocks(box[b], d) * march_cells(box[b], d);
  return s;
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

// Cuts the items into G equal shares: runs of segments (box, 2 * block + (dir - 1),
// m0, m1).  seg(int4) appends a segment, share() ends the current warp's share.
template <class Seg, class Share>
inline void march_schedule(const BoxRec* box, int n, long long G, Seg&& seg, Share&& share) {
  const double per = (double)march_items(box, n) / (double)G;
  long long w = 0, done = 0;
  for (int b = 0; b < n; ++b)
    for (int d = 1; d <= 2; ++d)
      for (int c = 0; c < march_blocks(box[b], d); ++c) {
        int m = box[b].lo[d];
        while (m <= box[b].hi[d]) {
          long long fit = (long long)((double)(w + 1) * per - (double)done + 0.5);
          if (fit < 1) fit = 1;
          const int end = (int)(box[b].hi[d] + 1 - m < fit ? box[b].hi[d] + 1 : m + fit);
          seg(make_int4(b, 2 * c + d - 1, m, end));
          done += end - m;
          m = end;
          if ((double)done >= (double)(w + 1) * per - 0.5 && w < G - 1) {
            ++w;
            share();
          }
        }
      }
  for (; w < G; ++w) share();
}

}  // namespace amrs

// Device box table shared by every launch: one record per box of a level
// (a single-box list for the per-box entry points).
#pragma once
#include "amrs_device.cuh"

namespace amrs {

constexpr int MAX_SLOTS = 4;
constexpr int F_THREADS = 256;  // threads per CTA of the face/divergence kernel

struct BoxRec {
  int lo[3], hi[3];
  double dxinv[3];
  double dx[3];
  DArr slot[MAX_SLOTS];  // caller-owned ghosted state arrays (3 ghosts)
  DArr q;                // primitives scratch over grow(box,3), NQ comps
  DArr vf;               // viscous cell fluxes over grow(box,1), NVF comps
  DArr div;              // KEEP path: y and z parts of the divergence, valid box, 2 NCONS comps
  int cl;                // closure index
  int tx, ty, kc;        // tile of the tuning interface (recorded; the marches deal columns to warps)
  // y walls of boundary code 6 that this box touches (walls == 0: none):
  // viscous cell fluxes of rows wrow_lo / wrow_hi use one-sided y
  // derivatives (ViscousWallFluxes); KEEP y faces j <= red_lo or
  // red_hi <= j <= hi[1] take the second-order pair (Flux_2nd_Order_KEEP)
  int walls;
  int wrow_lo, wrow_hi;
  int red_lo, red_hi;
};

// The KEEP path's range flag of a list, by stage numbers instead of clears, so that
// it holds whatever launches follow each other (a recorded step of any number
// of stages, one stage alone): the primitives' kernel takes the number `stage`,
// passes it on in `face` and marks a cell outside keep_range by raised = stage +
// 1; the face kernels see raised == face + 1 (every product on the FP64 pipe
// then), and the x kernel sets stage = face + 1.  No block reads a word that another
// block of its kernel writes.  All zero at first; `plain` counts the stages that ran on
// the FP64 pipe.
struct alignas(16) KeepRange {
  unsigned face, raised;
  unsigned stage, plain;
};

// Prefix tables for flattening launches over boxes.
struct BoxTable {
  const BoxRec* box;
  const long long* pcell;  // prefix of primitive-region cells, size n+1
  const long long* vcell;  // prefix of viscous-region cells, size n+1
  const int* fwork;        // prefix of the KEEP x kernel's blocks, size n+1
  const long long* mitem;  // prefix of the KEEP marches' items (march_items), size n+1
  int nshare;              // equal shares (warps) the items are cut into
  const DClosures* cls;
  int n;
  int gq;                  // ghost depth of the primitive region
  // device-resident time loop: every kernel of a step returns at once while
  // *active == 0 (steps after the stop time); null outside such loops
  const int* active;
  // whether a cell of this stage is outside keep_range; null: taken as if one were
  KeepRange* range;
  long long tot_p, tot_v, tot_m;  // cells of the primitive and viscous regions, march items
  // a list of one box carries its record and closures in the launch itself, so
  // that a kernel's first load is already data and per-box calls copy nothing
  int one;
  BoxRec rec;
  DClosures rec_cls;
};

__device__ __forceinline__ const BoxRec& box_rec(const BoxTable& tb, int b) { return tb.one ? tb.rec : tb.box[b]; }
__device__ __forceinline__ const DClosures& box_cls(const BoxTable& tb, const BoxRec& R) {
  return tb.one ? tb.rec_cls : tb.cls[R.cl];
}
// entry b of a prefix table
template <class T>
__device__ __forceinline__ T box_base(const BoxTable& tb, const T* prefix, int b) {
  return tb.one ? T(0) : prefix[b];
}

__device__ __forceinline__ bool list_idle(const BoxTable& tb) { return tb.active && *tb.active == 0; }

__device__ __forceinline__ int find_box_ll(const long long* pref, int n, long long x) {
  int lo = 0, hi = n;  // pref[lo] <= x < pref[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (pref[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int find_box_i(const int* pref, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (pref[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

}  // namespace amrs

// KEEP split-form + viscous RHS and the fused RK-stage epilogue.
//
// Four kernels per stage (all flattened over a box list):
//   prims_kernel      cons2prim over grow(box, gq)            (src/rhs/CNS_hydro_K.h:15-34)
//   visc_cell_kernel  cell-centred viscous fluxes, grow(box,1) (src/rhs/CNS_hydro_K.h:108-172)
//   keep_march_kernel y and z: KEEP face fluxes (src/rhs/CentralKEEP.h:40-145),
//                     viscous face averages (src/rhs/CNS_hydro_K.h:254-261) and
//                     their parts of the divergence (src/tim/CNS_advance.cpp:384-390)
//   keep_x_kernel     x: the same, the sum of the three parts and the stage's
//                     BLAS-1 program (src/tim/CNS_advance.cpp:51-166)
//
// Bound: GB300's FP64 pipe (one warp instruction per 16 clocks and SM, ~60x
// slower than its HBM relative to this path's 9 flop/byte).  So nothing is
// computed twice (primitives and viscous cell fluxes go through HBM; a pair
// term (a+l, a) that feeds l faces is kept in a register along the march or in
// shared memory along x), all products run on the integer pipe, and the work
// is cut so that warps never wait for each other while they hold FP64 work:
// the march's warps are independent, the x kernel's blocks are small (64
// registers, 32 warps per SM).  One kernel for all three directions, streaming
// z-planes through shared memory, held the FP64 pipe 73% busy (16 warps per SM,
// two barriers per plane) with 272 FP64 instructions per cell; 128^3, KEEP4 +
// viscous, per stage: 1257 us before, 430 + 320 us now with 167, FP64 pipe 72-79%
// busy (in between, with one kernel for x and y tiles and a z march: 890 us).  With a
// cell outside keep_range every product is on the FP64 pipe: a step with fluid at
// rest takes 4.09 ms instead of 2.88 (4.75 with the one kernel).
#include <type_traits>

#include "amrs_boxes.cuh"
#include "amrs_kernels.h"
#include "keep_schedule.h"

namespace amrs {

// ------------------------------------------------------------- prims ----
// Bound: the FP64 pipe (74% busy; nine instructions a cell and the copy's loads).
__global__ void __launch_bounds__(256, 5) prims_kernel(const __grid_constant__ BoxTable tb, int s_in) {
  dep_begin();
  if (list_idle(tb)) return;
  const long long total = tb.tot_p;
  const int g = tb.gq;
  bool outside = false;  // some cell of this thread is outside keep_range
  if (tb.range && blockIdx.x == 0 && threadIdx.x == 0) tb.range->face = tb.range->stage;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total;
       c += (long long)gridDim.x * blockDim.x) {
    const int b = find_box_ll(tb.pcell, tb.n, c);
    const BoxRec& R = box_rec(tb, b);
    const int l = (int)(c - box_base(tb, tb.pcell, b));
    const int nx = R.hi[0] - R.lo[0] + 1 + 2 * g, ny = R.hi[1] - R.lo[1] + 1 + 2 * g;
    const int i = l % nx + R.lo[0] - g;
    const int t = l / nx;
    const int j = t % ny + R.lo[1] - g;
    const int k = t / ny + R.lo[2] - g;
    const DArr U = R.slot[s_in];
    const long long o = U.off(i, j, k);
    double u[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) u[n] = U.p[o + n * U.ns];
    double q[NQ];
    cons2prim(u, q, box_cls(tb, R));
    outside = outside || !keep_range(q);
    const long long oq = R.q.off(i, j, k);
#pragma unroll
    for (int n = 0; n < NQ; ++n) R.q.p[oq + n * R.q.ns] = q[n];
  }
  if (outside && tb.range) {
    // mostly a read: with one store per thread to the one word a step with fluid
    // at rest (order 4, 128^3) takes 4.68 ms, so 4.09
    const unsigned mark = tb.range->stage + 1u;
    if (tb.range->raised != mark) tb.range->raised = mark;
  }
}

// ------------------------------------------------- viscous cell fluxes ----
// Bound: the FP64 pipe and the integer pipes about equally (37 additions and 40
// products a cell; 77% and half of the issue slots at 128^3, 170 us); three CTAs per
// SM (80 registers), two 2% of a step slower, four the same.
__global__ void __launch_bounds__(256, 3) visc_cell_kernel(const __grid_constant__ BoxTable tb) {
  dep_begin();
  if (list_idle(tb)) return;
  const long long total = tb.tot_v;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total;
       c += (long long)gridDim.x * blockDim.x) {
    const int b = find_box_ll(tb.vcell, tb.n, c);
    const BoxRec& R = box_rec(tb, b);
    const int l = (int)(c - box_base(tb, tb.vcell, b));
    const int nx = R.hi[0] - R.lo[0] + 3, ny = R.hi[1] - R.lo[1] + 3;
    const int i = l % nx + R.lo[0] - 1;
    const int t = l / nx;
    const int j = t % ny + R.lo[1] - 1;
    const int k = t / ny + R.lo[2] - 1;
    const DArr Q = R.q;
    const long long o = Q.off(i, j, k);
    const long long sx = 1, sy = Q.js, sz = Q.ks, sn = Q.ns;
    double qc[NQ], qxm[NQ], qxp[NQ], qym[NQ], qyp[NQ], qzm[NQ], qzp[NQ];
#pragma unroll
    for (int n = QU; n <= QT; ++n) {
      qc[n] = Q.p[o + n * sn];
      qxm[n] = Q.p[o - sx + n * sn];
      qxp[n] = Q.p[o + sx + n * sn];
      qym[n] = Q.p[o - sy + n * sn];
      qyp[n] = Q.p[o + sy + n * sn];
      qzm[n] = Q.p[o - sz + n * sn];
      qzp[n] = Q.p[o + sz + n * sn];
    }
    double f[NVF];
    if (R.walls && (j == R.wrow_lo || j == R.wrow_hi)) {
      // ghost row of a code-6 y wall: one-sided y derivatives into the box
      const int loc = (j == R.wrow_lo) ? 0 : 1;
      const long long s1 = loc == 0 ? sy : -sy;
      double q1[NQ], q2[NQ];
#pragma unroll
      for (int n = QU; n <= QT; ++n) {
        q1[n] = Q.p[o + s1 + n * sn];
        q2[n] = Q.p[o + 2 * s1 + n * sn];
      }
      viscous_wall_cell(loc, qc, qxm, qxp, q1, q2, qzm, qzp, R.dxinv, box_cls(tb, R), f);
    } else {
      viscous_cell(qc, qxm, qxp, qym, qyp, qzm, qzp, R.dxinv, box_cls(tb, R), f);
    }
    const long long ov = R.vf.off(i, j, k);
#pragma unroll
    for (int n = 0; n < NVF; ++n) R.vf.p[ov + n * R.vf.ns] = f[n];
  }
}

// ------------------------------------------------ fused face kernel -----
// Products of the divergence on the integer pipe (see kmul): bit 0 x, 1 y and z
// (on the FP64 pipe the 128^3 step takes 3.36 ms instead of 3.24).
#ifndef AMRS_DIV_IMUL
#define AMRS_DIV_IMUL 0x3
#endif

__device__ __forceinline__ void keep_coeffs(int order, double c[3]) {
  // CPU-branch coefficients of the reference (src/CNS.cpp:241-252)
  if (order == 6) { c[0] = 6.0 / 4; c[1] = -6.0 / 20; c[2] = 2.0 / 60; }
  else if (order == 4) { c[0] = 4.0 / 3; c[1] = -2.0 / 12; c[2] = 0.0; }
  else { c[0] = 1.0; c[1] = 0.0; c[2] = 0.0; }
}

// ---- x direction: one slot per thread.  Slot f of a row computes the pair
// terms T_l(f-1) = pair (f-1+l, f-1), l = 1..H; the face flux F(f) adds the
// terms T_l(f-l) .. T_l(f-2) of the H-1 slots below (shared memory), and
// cell f the flux F(f+1) of the slot above.  The slots of a box's rows
// (nx + H each: the first H-1 only feed the ones above) lie end to end in
// x, y, z order; a block takes blockDim of them and its neighbours overlap by H, so
// tiles leave no idle lanes whatever nx is.  The cell then adds the y and z parts
// the march left and applies the stage program.
template <int ORDER, bool VISC, bool SRC, bool FAST>
__device__ __forceinline__ void keep_x_body(const BoxTable& tb, int s_in, int s_s1, int s_out, const DProg& prog,
                                            int rhs_only, double* smem) {
  constexpr int H = ORDER / 2;
  const int tid = threadIdx.x, nth = blockDim.x;
  double coef[3];
  keep_coeffs(ORDER, coef);
  const int b = find_box_i(tb.fwork, tb.n, blockIdx.x);
  const BoxRec& R = box_rec(tb, b);
  const int nx = R.hi[0] - R.lo[0] + 1, ny = R.hi[1] - R.lo[1] + 1, nz = R.hi[2] - R.lo[2] + 1;
  const int row_slots = nx + H;
  // (a box's grown cells fit 31 bits, and with them the slots)
  const int g = (blockIdx.x - box_base(tb, tb.fwork, b)) * (nth - H) + tid;
  const bool in = g < row_slots * ny * nz;
  const int row = in ? g / row_slots : 0;
  const int s = in ? g - row * row_slots : 0;
  const int kk = row / ny;
  const int i = R.lo[0] + s - (H - 1), j = R.lo[1] + row - kk * ny, k = R.lo[2] + kk;
  double* ts = smem;                    // [H-1][5][nth]: T_l(f-1) of each slot, l = 2..H
  double* fs = smem + (H - 1) * 5 * nth;  // [5][nth]: F(f)
  double F[5];
  if (in) {
    const double* Q = R.q.p + R.q.off(i - 1, j, k);
    const long long qn = R.q.ns;
    double q2[NQ], q1[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) q2[n] = Q[n * qn];
#pragma unroll
    for (int l = H; l >= 2; --l) {
      double T[5];
#pragma unroll
      for (int n = 0; n < NQ; ++n) q1[n] = Q[l + n * qn];
      keep_pair<0, FAST>(q1, q2, coef[l - 1], T);
#pragma unroll
      for (int n = 0; n < 5; ++n) ts[((l - 2) * 5 + n) * nth + tid] = T[n];
    }
#pragma unroll
    for (int n = 0; n < NQ; ++n) q1[n] = Q[1 + n * qn];
    keep_pair<0, FAST>(q1, q2, coef[0], F);
  }
  if (H >= 2) __syncthreads();
  const bool face = in && s >= H - 1 && tid >= H - 1;
  if (face) {
#pragma unroll
    for (int l = 2; l <= H; ++l)
#pragma unroll
      for (int m = 0; m < l; ++m) {
        const double* t = ts + (l - 2) * 5 * nth + tid - (l - 1 - m);
#pragma unroll
        for (int n = 0; n < 5; ++n) F[n] = F[n] + t[n * nth];
      }
    if (VISC) {
      const double* V = R.vf.p + R.vf.off(i, j, k);
#pragma unroll
      for (int n = 0; n < 4; ++n) F[1 + n] = fma(0.5, V[n * R.vf.ns - 1] + V[n * R.vf.ns], F[1 + n]);
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) fs[n * nth + tid] = F[n];
  }
  __syncthreads();
  if (face && s < row_slots - 1 && tid < nth - 1) {
    const DArr& Uin = R.slot[s_in];
    const DArr& U1 = R.slot[s_s1];
    const DArr& Uo = R.slot[s_out];
    const double* D = R.div.p + R.div.off(i, j, k);
    const long long dn = R.div.ns, oin = Uin.off(i, j, k), o1 = U1.off(i, j, k), oo = Uo.off(i, j, k);
    const bool src = SRC && box_cls(tb, R).source != 0;  // SRC: a list with a source term
    // all loads of a kind before the products: their range tests are branches
    // that loads do not cross
    double ds[5], y[5], z[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      y[n] = D[n * dn];
      z[n] = D[(5 + n) * dn];
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      ds[n] = kmul<AMRS_DIV_IMUL & 1>(R.dxinv[0], F[n] - fs[n * nth + tid + 1]) + y[n] + z[n];
      if (src) ds[n] = add_source(box_cls(tb, R), Uin.p, oin, Uin.ns, n, ds[n]);
    }
    if (!rhs_only) {
      double s1[5], s2[5];
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        s1[n] = U1.p[o1 + n * U1.ns];
        s2[n] = Uin.p[oin + n * Uin.ns];
      }
#pragma unroll
      for (int n = 0; n < 5; ++n) ds[n] = apply_prog(prog, s1[n], s2[n], ds[n]);
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) Uo.p[oo + n * Uo.ns] = ds[n];
  }
}

// ---- y and z directions: one thread per column, a warp marching its 32 columns
// over a run of cells with the shared pair terms in registers.  Writes
// dxinv (F(m) - F(m+1)) of its direction over cells [m0, m1) of column block
// `blk`, columns consecutive in x, then in z (y march) or y (z march).
template <int ORDER, int DIR, bool VISC, bool FAST>
__device__ __forceinline__ void keep_march(const BoxRec& R, int blk, int m0, int m1, const double coef[3]) {
  constexpr int H = ORDER / 2;
  const int nx = R.hi[0] - R.lo[0] + 1, nt = DIR == 1 ? R.hi[2] - R.lo[2] + 1 : R.hi[1] - R.lo[1] + 1;
  const int c = blk * 32 + (threadIdx.x & 31);
  if (c >= nx * nt) return;
  const int ct = c / nx, ci = R.lo[0] + c - ct * nx;
  const int j0 = DIR == 1 ? m0 : R.lo[1] + ct, k0 = DIR == 1 ? R.lo[2] + ct : m0;
  const double dxi = R.dxinv[DIR];
  // the scratch arrays' strides fit 32 bits (a box's grown cells do): orders 2
  // and 4, at their 128 registers, keep half as many for them
  using Stride = typename std::conditional<ORDER == 6, long long, int>::type;
  const Stride qk = (Stride)(DIR == 1 ? R.q.js : R.q.ks), vk = (Stride)(DIR == 1 ? R.vf.js : R.vf.ks),
               dk = (Stride)(DIR == 1 ? R.div.js : R.div.ks);
  const Stride qn = (Stride)R.q.ns, vn = (Stride)R.vf.ns, dn = (Stride)R.div.ns;
  // pointers at cell m0 of the column
  const double* Q = R.q.p + R.q.off(ci, j0, k0);
  const double* V = VISC ? R.vf.p + R.vf.off(ci, j0, k0) + 4ll * DIR * vn : nullptr;
  double* D = R.div.p + R.div.off(ci, j0, k0) + 5ll * (DIR - 1) * dn;
  // code-6 y walls: faces of second order (halfsten 1, coefficient 1)
  auto reduced = [&](int f) { return DIR == 1 && R.walls && (f <= R.red_lo || (f >= R.red_hi && f <= R.hi[1])); };
  // carries: tc[l][m] = T_l(c+1-l+m) for m=0..l-2 (l>=2); ring of Q(c..c+H-1)
  double tc[3][2][5];
  double ring[3][NQ];
  double fl[5], vl[4];  // flux and viscous cell flux below the current cell
  {
    // the flux at face m0 (between m0-1 and m0) and the carries
    double qcol[2 * H][NQ];  // cells m0-H .. m0+H-1
#pragma unroll
    for (int p = 0; p < 2 * H; ++p)
#pragma unroll
      for (int n = 0; n < NQ; ++n) qcol[p][n] = Q[(long long)(p - H) * qk + (long long)n * qn];
    const bool red = reduced(m0);
    keep_pair<DIR, FAST>(qcol[H], qcol[H - 1], red ? 1.0 : coef[0], fl);  // T_1(m0-1)
#pragma unroll
    for (int l = 2; l <= H; ++l) {
#pragma unroll
      for (int m = 0; m < l; ++m) {
        const int a = -l + m;  // T_l(m0+a), pair (m0+a+l, m0+a)
        double T[5];
        keep_pair<DIR, FAST>(qcol[H + a + l], qcol[H + a], coef[l - 1], T);
        if (!red) {
#pragma unroll
          for (int n = 0; n < 5; ++n) fl[n] = fl[n] + T[n];
        }
        if (m >= 1) {
#pragma unroll
          for (int n = 0; n < 5; ++n) tc[l - 1][m - 1][n] = T[n];
        }
      }
    }
    if (VISC) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        vl[n] = V[(long long)n * vn];
        fl[1 + n] = fma(0.5, V[(long long)n * vn - vk] + vl[n], fl[1 + n]);
      }
    }
#pragma unroll
    for (int p = 0; p < H; ++p)
#pragma unroll
      for (int n = 0; n < NQ; ++n) ring[p][n] = qcol[H + p][n];
  }
#pragma unroll 1
  for (int m = m0; m < m1; ++m) {
    // T_l(m) = pair (m+l, m), l = 1..H: the flux at face m+1
    double qtop[NQ], F[5];
#pragma unroll
    for (int n = 0; n < NQ; ++n) qtop[n] = Q[(long long)H * qk + (long long)n * qn];
    const bool red = reduced(m + 1);
    keep_pair<DIR, FAST>(H == 1 ? qtop : ring[1], ring[0], red ? 1.0 : coef[0], F);
#pragma unroll
    for (int l = 2; l <= H; ++l) {
      // F += T_l(m+1-l+p), p = 0..l-1 (p = l-1 is the new term), then the
      // carries drop T_l(m+1-l) and append T_l(m)
      double Tn[5];
      if (!red) {
#pragma unroll
        for (int p = 0; p < l - 1; ++p)
#pragma unroll
          for (int n = 0; n < 5; ++n) F[n] = F[n] + tc[l - 1][p][n];
      }
      keep_pair<DIR, FAST>(l == H ? qtop : ring[l], ring[0], coef[l - 1], Tn);
      if (!red) {
#pragma unroll
        for (int n = 0; n < 5; ++n) F[n] = F[n] + Tn[n];
      }
#pragma unroll
      for (int p = 0; p < l - 2; ++p)
#pragma unroll
        for (int n = 0; n < 5; ++n) tc[l - 1][p][n] = tc[l - 1][p + 1][n];
#pragma unroll
      for (int n = 0; n < 5; ++n) tc[l - 1][l - 2][n] = Tn[n];
    }
    if (VISC) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const double c1 = V[vk + (long long)n * vn];
        F[1 + n] = fma(0.5, vl[n] + c1, F[1 + n]);
        vl[n] = c1;
      }
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      D[(long long)n * dn] = kmul<(AMRS_DIV_IMUL >> 1) & 1>(dxi, fl[n] - F[n]);
      fl[n] = F[n];
    }
#pragma unroll
    for (int p = 0; p < H - 1; ++p)
#pragma unroll
      for (int n = 0; n < NQ; ++n) ring[p][n] = ring[p + 1][n];
#pragma unroll
    for (int n = 0; n < NQ; ++n) ring[H - 1][n] = qtop[n];
    Q += qk;
    V += vk;
    D += dk;
  }
}

// Resident CTAs of the march: 128 registers hold the carries of orders 2 and 4
// (three CTAs per SM spill and are 2% slower over a step), order 6 takes all 255
// (two CTAs: 288 instead of 272 us per step of 45 x 33 x 27).
template <int ORDER> constexpr int march_ctas() { return ORDER == 6 ? 1 : 2; }

// every cell of the stage is inside keep_range (BoxTable::range), uniform over the grid
__device__ __forceinline__ bool fast_range(const BoxTable& tb) {
  return tb.range && tb.range->raised != tb.range->face + 1u;
}

template <int ORDER, bool VISC, bool FAST>
__device__ __forceinline__ void keep_march_warp(const BoxTable& tb) {
  // warp w takes items [w N / G, (w+1) N / G) of the list: a run of segments,
  // each within one column block
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (w >= tb.nshare) return;
  double coef[3];
  keep_coeffs(ORDER, coef);
  const long long N = tb.tot_m;
  const long long at = w * N / tb.nshare;
  int left = (int)((w + 1) * N / tb.nshare - at);
  int b = find_box_ll(tb.mitem, tb.n, at);
  int r = (int)(at - box_base(tb, tb.mitem, b));
#pragma unroll 1
  while (left > 0) {
    const BoxRec& R = box_rec(tb, b);
    const int ny = march_cells(R, 1), nz = march_cells(R, 2);
    const int ytot = march_blocks(R, 1) * ny, ztot = march_blocks(R, 2) * nz;
    if (r == ytot + ztot) { ++b; r = 0; continue; }
    const bool z = r >= ytot;
    const int p = z ? r - ytot : r, cells = z ? nz : ny;
    const int blk = p / cells, m = p - blk * cells;
    const int run = min(left, cells - m), m0 = R.lo[z ? 2 : 1] + m;
    left -= run;
    r += run;
    if (z) keep_march<ORDER, 2, VISC, FAST>(R, blk, m0, m0 + run, coef);
    else keep_march<ORDER, 1, VISC, FAST>(R, blk, m0, m0 + run, coef);
  }
}

template <int ORDER, bool VISC>
__global__ void __launch_bounds__(F_THREADS, march_ctas<ORDER>())
keep_march_kernel(const __grid_constant__ BoxTable tb) {
  dep_begin();
  if (list_idle(tb)) return;
  if (fast_range(tb)) keep_march_warp<ORDER, VISC, true>(tb);
  else keep_march_warp<ORDER, VISC, false>(tb);
}

template <int ORDER, bool VISC, bool SRC>
__global__ void __launch_bounds__(F_THREADS, 4)
keep_x_kernel(const __grid_constant__ BoxTable tb, int s_in, int s_s1, int s_out, DProg prog_in, int rhs_only) {
  dep_begin();
  if (list_idle(tb)) return;  // uniform over the CTA: before any barrier
  const DProg prog = resolve_prog(prog_in);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* smem = reinterpret_cast<double*>(smem_raw);
  const bool fast = fast_range(tb);
  if (tb.range && blockIdx.x == 0 && threadIdx.x == 0) {
    // (a stage in several launches counts once)
    if (!fast && tb.range->stage == tb.range->face) ++tb.range->plain;
    tb.range->stage = tb.range->face + 1u;
  }
  if (fast) keep_x_body<ORDER, VISC, SRC, true>(tb, s_in, s_s1, s_out, prog, rhs_only, smem);
  else keep_x_body<ORDER, VISC, SRC, false>(tb, s_in, s_s1, s_out, prog, rhs_only, smem);
}

// explicit instantiations + launchers
template <int ORDER, bool VISC, bool SRC>
static cudaError_t launch_face_t(const BoxTable& tb, int s_in, int s_s1, int s_out, const DProg& prog, int rhs_only,
                                 const KeepGrid& g, cudaStream_t st) {
  launch_dep(keep_march_kernel<ORDER, VISC>, g.march_ctas, g.march_threads, 0, st, tb);
  launch_dep(keep_x_kernel<ORDER, VISC, SRC>, g.x_ctas, g.x_threads, (ORDER / 2) * 5 * 8 * g.x_threads, st, 
      tb, s_in, s_s1, s_out, prog, rhs_only);
  return cudaGetLastError();
}

cudaError_t launch_prims(const BoxTable& tb, int s_in, long long ncells, int nsm, cudaStream_t st) {
  if (ncells <= 0) return cudaSuccess;
  long long blocks = (ncells + 255) / 256;
  const long long cap = (long long)nsm * GRID_CTAS;
  if (blocks > cap) blocks = cap;
  launch_dep(prims_kernel, (int)blocks, 256, 0, st, tb, s_in);
  return cudaGetLastError();
}

cudaError_t launch_visc(const BoxTable& tb, long long ncells, int nsm, cudaStream_t st) {
  if (ncells <= 0) return cudaSuccess;
  long long blocks = (ncells + 255) / 256;
  const long long cap = (long long)nsm * GRID_CTAS;
  if (blocks > cap) blocks = cap;
  launch_dep(visc_cell_kernel, (int)blocks, 256, 0, st, tb);
  return cudaGetLastError();
}

cudaError_t launch_keep_face(int order, bool visc, bool src, const BoxTable& tb, int s_in, int s_s1, int s_out,
                             const DProg& prog, int rhs_only, const KeepGrid& g, cudaStream_t st) {
  if (g.x_ctas <= 0) return cudaSuccess;
#define AMRS_FACE(O, V, S) launch_face_t<O, V, S>(tb, s_in, s_s1, s_out, prog, rhs_only, g, st)
#define AMRS_FACE_VS(O) \
  (visc ? (src ? AMRS_FACE(O, true, true) : AMRS_FACE(O, true, false)) \
        : (src ? AMRS_FACE(O, false, true) : AMRS_FACE(O, false, false)))
  if (order == 2) return AMRS_FACE_VS(2);
  if (order == 4) return AMRS_FACE_VS(4);
  return AMRS_FACE_VS(6);
#undef AMRS_FACE_VS
#undef AMRS_FACE
}

int keep_ctas_per_sm(int order) { return order == 6 ? march_ctas<6>() : march_ctas<4>(); }

int keep_x_blocks(int order, const int n[3], int threads) {
  const int H = order / 2;
  const long long slots = (long long)(n[0] + H) * n[1] * n[2];
  return (int)((slots - H + threads - H - 1) / (threads - H));
}

// The tile shapes that the tuning interface accepts (and records: no kernel reads
// them any more): those whose planes once fitted a block's shared memory.
bool keep_tile_fits(int order, int tx, int ty) {
  if (tx < 8 || ty < 1 || (tx % 2) || tx * ty > F_THREADS) return false;
  const int H = order / 2;
  if ((tx + 6) * (ty + 2 * H) > (order == 6 ? 544 : 480)) return false;
  if ((tx + H) * ty > 352 || tx * (ty + H) > 352) return false;
  return (tx + 1) * ty <= 288 && tx * (ty + 1) <= 288;
}

}  // namespace amrs

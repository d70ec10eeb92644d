// Hand-written adjoint (vector-Jacobian product) of the KEEP + viscous RHS
// and of one RK stage.
//
// Forward map of one RHS (src/tim/CNS_advance.cpp:186-391):
//   U --cons2prim--> Q --KEEP pairs, viscous cell fluxes--> face fluxes F
//     --divergence--> dSdt.
// Reverse, given a cotangent vbar on the valid cells of dSdt:
//   Fbar_d(face f) = dxinv_d (vbar(f) - vbar(f-1))            (divergence^T)
//   adj_pair_kernel : every KEEP pair (a, a+l) once: Tbar = sum of Fbar over
//                     the l faces it feeds; pair VJP -> Qbar contributions of
//                     both ends into per-(direction, separation) buffers
//   adj_visc_kernel : every cell of grow(box,1): Vbar = average of Fbar over
//                     its two faces per direction; VJP of the cell viscous
//                     flux -> Qbar at the centre and gradient cotangents
//   adj_gather_kernel: Qbar(c) = sum of the buffers + gradient cotangents of
//                     the six neighbours; then the cons2prim VJP -> Ubar(c)
// Non-smooth points follow the branch the forward pass takes (max(1e-40,rho)
// passes the derivative only when rho > 1e-40).  Sums are deterministic:
// every output element is written by exactly one thread.
#include "adjoint_common.cuh"
#include "amrs_kernels.h"

namespace amrs {

struct AdjRec {
  DArr vbar;    // cotangent of dSdt, valid cells
  DArr ubar;    // output cotangent of the state, grow(box,3)
  DArr pair[3][3];  // [d][l-1]: NQA comps lo-end (0..5) + hi-end (6..11) over grow(box,3)
  DArr vg;      // viscous cotangents over grow(box,1): centre u,v,w,T (0..3), gradients (4..15)
  int visc;     // vg holds data (the viscous reverse pass ran)
  double* part; // per-block partial sums of d/d(visc_ref), d/d(cond_ref): 2 per block of adj_visc_kernel
};

__device__ __forceinline__ double vget(const DArr& v, const BoxRec& R, int i, int j, int k, int n) {
  if (i < R.lo[0] || i > R.hi[0] || j < R.lo[1] || j > R.hi[1] || k < R.lo[2] || k > R.hi[2]) return 0.0;
  return v(i, j, k, n);
}

// Fbar of the d-face below cell (i,j,k), component n.
__device__ __forceinline__ double fbar(const DArr& v, const BoxRec& R, int d, int i, int j, int k, int n) {
  const int di = d == 0, dj = d == 1, dk = d == 2;
  return R.dxinv[d] * (vget(v, R, i, j, k, n) - vget(v, R, i - di, j - dj, k - dk, n));
}

// VJP of one KEEP pair term (keep_pair in amrs_device.cuh) given half its
// cotangent, a[5] (already times the coefficient): contributions to the
// primitive cotangents of point 1 (larger index) and point 2.  With sums
// R, N, U, E of the two ends and K = sum of the velocity products, the pair is
// (R N) / 8 times (2, U + .., E + K) plus pressure terms, so the cotangents of
// U and E are t4 a with t4 = R N / 4, those of R and N are N and R times one
// factor, and the kinetic term's is that of E (exact scalings; the reverse
// pass has no bit-exact counterpart).  Products that no addition consumes go
// to the integer pipe: 32 FP64 instructions are left, 55 before.
template <int D>
__device__ __forceinline__ void keep_pair_vjp(const double* q1, const double* q2, const double a[5], double cv,
                                              double b1[NQA], double b2[NQA]) {
  constexpr int QN = QU + D;
  const double R = q1[QRHO] + q2[QRHO];
  const double U[3] = {q1[QU] + q2[QU], q1[QV] + q2[QV], q1[QW] + q2[QW]};
  const double N = U[D];
  const double K = q1[QU] * q2[QU] + q1[QV] * q2[QV] + q1[QW] * q2[QW];
  const double t4 = 0.25 * dmul_rn(R, N);
  const double s4 =
      0.25 * (2.0 * a[0] + (a[1] * U[0] + a[2] * U[1] + a[3] * U[2] + a[4] * ((q1[QE] + q2[QE]) + K)));
  const double Eb = dmul_rn(a[4], t4);
  double Ub[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) Ub[c] = dmul_rn(a[1 + c], t4);
  Ub[D] += dmul_rn(R, s4);
  const double Rb = dmul_rn(N, s4), cvE = dmul_rn(cv, Eb);
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const double* qo = s ? q1 : q2;
    double* b = s ? b2 : b1;
    b[0] = Rb;
#pragma unroll
    for (int c = 0; c < 3; ++c) b[1 + c] = Ub[c] + Eb * qo[QU + c];
    b[1 + D] += a[4] * qo[QPRES];
    b[4] = cvE;
    b[5] = a[1 + D] + a[4] * qo[QN];
  }
}

// One thread per (direction, separation, pair): pairs (a, a+l) along d
// with a in [lo-l, hi] and transverse indices in the valid box.  Bound: the FP64
// pipe (76% busy at 64^3, order 4: 121 us; 158 with 55 FP64 instructions a pair).
// Four CTAs per SM (64 registers); with two, 96 registers and 153 us.
template <int ORDER>
__global__ void __launch_bounds__(256, 4)
adj_pair_kernel(const __grid_constant__ BoxTable tb, AdjRec ar, long long total) {
  dep_begin();
  constexpr int H = ORDER / 2;
  double coef[3];
  if (ORDER == 6) { coef[0] = 6.0 / 4; coef[1] = -6.0 / 20; coef[2] = 2.0 / 60; }
  else if (ORDER == 4) { coef[0] = 4.0 / 3; coef[1] = -2.0 / 12; coef[2] = 0.0; }
  else { coef[0] = 1.0; coef[1] = 0.0; coef[2] = 0.0; }
  const BoxRec& R = box_rec(tb, 0);
  const DClosures& cl = box_cls(tb, R);
  const int n0 = R.hi[0] - R.lo[0] + 1, n1 = R.hi[1] - R.lo[1] + 1, n2 = R.hi[2] - R.lo[2] + 1;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    // decode (d, l, i, j, k): per (d,l) block, extent n_d + l in d
    long long r = g;
    int d = 0, l = 1;
    bool found = false;
    for (int dd = 0; dd < 3 && !found; ++dd)
      for (int ll = 1; ll <= H && !found; ++ll) {
        const long long cnt = (long long)(n0 + (dd == 0) * ll) * (n1 + (dd == 1) * ll) * (n2 + (dd == 2) * ll);
        if (r < cnt) { d = dd; l = ll; found = true; }
        else r -= cnt;
      }
    if (!found) continue;
    const int e0 = n0 + (d == 0) * l, e1 = n1 + (d == 1) * l;
    const unsigned ru = (unsigned)r, t = ru / (unsigned)e0;  // fewer than 2^31 pairs of one direction and separation
    const int ii = (int)(ru - t * (unsigned)e0), kk = (int)(t / (unsigned)e1);
    const int jj = (int)(t - (unsigned)kk * (unsigned)e1);
    const int i = R.lo[0] + ii - (d == 0) * l, j = R.lo[1] + jj - (d == 1) * l, k = R.lo[2] + kk - (d == 2) * l;
    const int di = d == 0, dj = d == 1, dk = d == 2;
    // pair (a = (i,j,k), a + l e_d); faces a+1 .. a+l.  Next to a code-6 y
    // wall the reduced y faces take only the l = 1 pair, with coefficient 1
    // (Flux_2nd_Order_KEEP, src/rhs/CentralKEEP.h:232-287).
    double a[5] = {0, 0, 0, 0, 0};
    if (d == 1 && R.walls) {
      for (int m = 1; m <= l; ++m) {
        double w = 0.5 * coef[l - 1];
        const int jf = j + m;
        if (jf <= R.red_lo || (jf >= R.red_hi && jf <= R.hi[1])) w = (l == 1) ? 0.5 : 0.0;
        if (w == 0.0) continue;
#pragma unroll
        for (int n = 0; n < 5; ++n) a[n] += w * fbar(ar.vbar, R, d, i + m * di, j + m * dj, k + m * dk, n);
      }
    } else {
      // one coefficient for all l faces: sum_m Fbar(a + m) telescopes to
      // dxinv_d (vbar(a + l) - vbar(a))
      const double wd = 0.5 * coef[l - 1] * R.dxinv[d];
#pragma unroll
      for (int n = 0; n < 5; ++n)
        a[n] = dmul_rn(wd, vget(ar.vbar, R, i + l * di, j + l * dj, k + l * dk, n) - vget(ar.vbar, R, i, j, k, n));
    }
    double q1[NQ], q2[NQ], b1[NQA], b2[NQA];
    const long long o2 = R.q.off(i, j, k), o1 = R.q.off(i + l * di, j + l * dj, k + l * dk);
#pragma unroll
    for (int n = 0; n < NQ; ++n) { q1[n] = R.q.p[o1 + n * R.q.ns]; q2[n] = R.q.p[o2 + n * R.q.ns]; }
    if (d == 0) keep_pair_vjp<0>(q1, q2, a, cl.cv, b1, b2);
    else if (d == 1) keep_pair_vjp<1>(q1, q2, a, cl.cv, b1, b2);
    else keep_pair_vjp<2>(q1, q2, a, cl.cv, b1, b2);
    const DArr P = ar.pair[d][l - 1];
    const long long olo = P.off(i, j, k), ohi = P.off(i + l * di, j + l * dj, k + l * dk);
#pragma unroll
    for (int n = 0; n < NQA; ++n) {
      P.p[olo + n * P.ns] = b2[n];
      P.p[ohi + (NQA + n) * P.ns] = b1[n];
    }
  }
}

// VJP of the cell viscous fluxes (viscous_cell in amrs_device.cuh) for every
// cell of grow(box,1).  With `pbar`, each block also sums d/d(visc_ref) and
// d/d(cond_ref) over its cells in a fixed order (grid-stride, then warp
// shuffles, then the warps in order) into ar.part; adj_param_sum_kernel adds
// the blocks' sums in block order.  No atomics: the result is the same bits
// on every run.  Bound: the FP64 pipe (94 instructions a cell) behind the loads'
// latency: four CTAs per SM 58 us at 64^3, two 65.  Its products on the integer
// pipe gained nothing (within 0.3% of a step's gradient at 64^3).
__global__ void __launch_bounds__(256, 4)
adj_visc_kernel(const __grid_constant__ BoxTable tb, AdjRec ar, long long total, double* pbar) {
  dep_begin();
  const BoxRec& R = box_rec(tb, 0);
  const DClosures& cl = box_cls(tb, R);
  const int nx = R.hi[0] - R.lo[0] + 3, ny = R.hi[1] - R.lo[1] + 3;
  double mu_acc = 0.0, la_acc = 0.0;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int l = (int)g;
    const int i = l % nx + R.lo[0] - 1;
    const int t = l / nx;
    const int j = t % ny + R.lo[1] - 1;
    const int k = t / ny + R.lo[2] - 1;
    const double hx = 0.5 * R.dxinv[0], hy = 0.5 * R.dxinv[1], hz = 0.5 * R.dxinv[2];
    // Vbar: each cell flux enters the faces below and above it with 0.5, and
    // Fbar(c) + Fbar(c + e_d) = dxinv_d (vbar(c + e_d) - vbar(c - e_d))
    double fb[NVF];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int di = d == 0, dj = d == 1, dk = d == 2;
      const double h = d == 0 ? hx : (d == 1 ? hy : hz);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        fb[4 * d + n] = h * (vget(ar.vbar, R, i + di, j + dj, k + dk, 1 + n) -
                             vget(ar.vbar, R, i - di, j - dj, k - dk, 1 + n));
    }
    const DArr Q = R.q;
    const long long o = Q.off(i, j, k);
    auto q = [&](long long off, int n) { return Q.p[off + n * Q.ns]; };
    const long long sx = 1, sy = Q.js, sz = Q.ks;
    const double u = q(o, QU), v = q(o, QV), w = q(o, QW), T = q(o, QT);
    auto central = [&](long long st, int n, double h) { return (q(o + st, n) - q(o - st, n)) * h; };
    const double dudx = central(sx, QU, hx), dvdx = central(sx, QV, hx);
    const double dwdx = central(sx, QW, hx), dTdx = central(sx, QT, hx);
    // y derivatives: central, or one-sided on the ghost row beyond a code-6
    // wall (ViscousWallFluxes, src/rhs/CNS_hydro_K.h:177-251)
    auto ddy = [&](int n) {
      if (R.walls && j == R.wrow_lo) return (4.0 * q(o + sy, n) - q(o + 2 * sy, n) - 3.0 * q(o, n)) * hy;
      if (R.walls && j == R.wrow_hi) return (-4.0 * q(o - sy, n) + 3.0 * q(o, n) + q(o - 2 * sy, n)) * hy;
      return central(sy, n, hy);
    };
    const double dudy = ddy(QU), dvdy = ddy(QV), dwdy = ddy(QW), dTdy = ddy(QT);
    const double dudz = central(sz, QU, hz), dvdz = central(sz, QV, hz);
    const double dwdz = central(sz, QW, hz), dTdz = central(sz, QT, hz);
    const double div = dudx + dvdy + dwdz;
    const double mu = visc(cl, T), lam = cond(cl, T);
    const double r13 = 1.0 / 3.0;
    const double mu2 = 2.0 * mu, d3 = r13 * div;
    const double exx = dudx - d3, eyy = dvdy - d3, ezz = dwdz - d3;
    const double exy = dudy + dvdx, exz = dudz + dwdx, eyz = dvdz + dwdy;
    const double txx = mu2 * exx, tyy = mu2 * eyy, tzz = mu2 * ezz;
    const double txy = mu * exy, txz = mu * exz, tyz = mu * eyz;
    const double txxb = -fb[0] - fb[3] * u;
    const double txyb = -fb[1] - fb[3] * v - fb[4] - fb[7] * u;
    const double txzb = -fb[2] - fb[3] * w - fb[8] - fb[11] * u;
    const double tyyb = -fb[5] - fb[7] * v;
    const double tyzb = -fb[6] - fb[7] * w - fb[9] - fb[11] * v;
    const double tzzb = -fb[10] - fb[11] * w;
    const double ub = -(fb[3] * txx + fb[7] * txy + fb[11] * txz);
    const double vb = -(fb[3] * txy + fb[7] * tyy + fb[11] * tyz);
    const double wb = -(fb[3] * txz + fb[7] * tyz + fb[11] * tzz);
    const double divb = -(2.0 / 3.0) * mu * (txxb + tyyb + tzzb);
    double gb[12];
    const double gxy = mu * txyb, gxz = mu * txzb, gyz = mu * tyzb;
    gb[0] = mu2 * txxb + divb;  // dudx
    gb[1] = gxy;                     // dvdx
    gb[2] = gxz;                     // dwdx
    gb[3] = -lam * fb[3];            // dTdx
    gb[4] = gxy;                     // dudy
    gb[5] = mu2 * tyyb + divb;  // dvdy
    gb[6] = gyz;                     // dwdy
    gb[7] = -lam * fb[7];            // dTdy
    gb[8] = gxz;                     // dudz
    gb[9] = gyz;                     // dvdz
    gb[10] = mu2 * tzzb + divb; // dwdz
    gb[11] = -lam * fb[11];          // dTdz
    double Tb = 0.0;
    if (cl.visc_law == 1 || pbar) {
      const double mub =
          2.0 * (txxb * exx + tyyb * eyy + tzzb * ezz) + txyb * exy + txzb * exz + tyzb * eyz;
      if (cl.visc_law == 1) Tb += mub * mu * (ddiv_rn(1.5, T) - ddiv_rn(1.0, cl.Tvisc_ref + T));
      else mu_acc += mub;
    }
    if (cl.cond_law == 1 || pbar) {
      const double lamb = -(fb[3] * dTdx + fb[7] * dTdy + fb[11] * dTdz);
      if (cl.cond_law == 1) Tb += lamb * lam * (ddiv_rn(1.5, T) - ddiv_rn(1.0, cl.Tcond_ref + T));
      else la_acc += lamb;
    }
    const DArr G = ar.vg;
    const long long og = G.off(i, j, k);
    G.p[og] = ub;
    G.p[og + G.ns] = vb;
    G.p[og + 2 * G.ns] = wb;
    G.p[og + 3 * G.ns] = Tb;
#pragma unroll
    for (int n = 0; n < 12; ++n) G.p[og + (4 + n) * G.ns] = gb[n];
  }
  if (pbar) {
    __shared__ double wsum[2][8];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      mu_acc += __shfl_down_sync(0xffffffffu, mu_acc, off);
      la_acc += __shfl_down_sync(0xffffffffu, la_acc, off);
    }
    if ((threadIdx.x & 31) == 0) {
      wsum[0][threadIdx.x >> 5] = mu_acc;
      wsum[1][threadIdx.x >> 5] = la_acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = 0.0, a = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        m += wsum[0][w];
        a += wsum[1][w];
      }
      ar.part[2 * blockIdx.x] = m;
      ar.part[2 * blockIdx.x + 1] = a;
    }
  }
}

// pbar += the per-block sums of adj_visc_kernel, in block order.
__global__ void adj_param_sum_kernel(const double* part, int nblocks, double* pbar) {
  dep_begin();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double m = 0.0, a = 0.0;
  for (int b = 0; b < nblocks; ++b) {
    m += part[2 * b];
    a += part[2 * b + 1];
  }
  pbar[0] += m;
  pbar[1] += a;
}

// Qbar gather + cons2prim VJP for every cell of grow(box,3).  Bound: the FP64 pipe
// (82% busy: 72 of its additions at order 4 are the pairs'); 84 us at 64^3, four
// CTAs per SM (two: 93).
template <int ORDER>
__global__ void __launch_bounds__(256, 4)
adj_gather_kernel(const __grid_constant__ BoxTable tb, AdjRec ar, long long total, int gpair) {
  dep_begin();
  constexpr int H = ORDER / 2;
  const BoxRec& R = box_rec(tb, 0);
  const DClosures& cl = box_cls(tb, R);
  const int g3 = NGHOST;
  const int nx = R.hi[0] - R.lo[0] + 1 + 2 * g3, ny = R.hi[1] - R.lo[1] + 1 + 2 * g3;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int l0 = (int)g;
    const int i = l0 % nx + R.lo[0] - g3;
    const int t = l0 / nx;
    const int j = t % ny + R.lo[1] - g3;
    const int k = t / ny + R.lo[2] - g3;
    const DArr Ub = ar.ubar;
    const long long ou = Ub.off(i, j, k);
    // cells any cotangent of this pass reaches (viscous stencils: 2 ghosts);
    // beyond them Q is not computed and ubar is zero
    const int gvisc = ar.visc ? 2 : 0;
    const int gact = gpair > gvisc ? gpair : gvisc;
    if (i < R.lo[0] - gact || i > R.hi[0] + gact || j < R.lo[1] - gact || j > R.hi[1] + gact ||
        k < R.lo[2] - gact || k > R.hi[2] + gact) {
#pragma unroll
      for (int n = 0; n < 5; ++n) Ub.p[ou + n * Ub.ns] = 0.0;
      continue;
    }
    double qb[NQA] = {0, 0, 0, 0, 0, 0};
    const bool in_pair = i >= R.lo[0] - gpair && i <= R.hi[0] + gpair && j >= R.lo[1] - gpair &&
                         j <= R.hi[1] + gpair && k >= R.lo[2] - gpair && k <= R.hi[2] + gpair;
    if (in_pair) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int l = 1; l <= H; ++l) {
          // pairs (a, a + l) exist for a in [lo - l, hi] along d and valid
          // transverse indices: this cell's as the lower and as the upper end
          const DArr& P = ar.pair[d][l - 1];
          const int c[3] = {i, j, k};
          bool across = true;
#pragma unroll
          for (int t = 0; t < 3; ++t) across = across && (t == d || (c[t] >= R.lo[t] && c[t] <= R.hi[t]));
          const double* p = P.p + P.off(i, j, k);
          if (across && c[d] >= R.lo[d] - l && c[d] <= R.hi[d]) {
#pragma unroll
            for (int n = 0; n < NQA; ++n) qb[n] += p[n * P.ns];
          }
          if (across && c[d] >= R.lo[d] && c[d] <= R.hi[d] + l) {
#pragma unroll
            for (int n = 0; n < NQA; ++n) qb[n] += p[(NQA + n) * P.ns];
          }
        }
    }
    const DArr G = ar.vg;
    auto inside1 = [&](int a, int b, int c) {
      return ar.visc && a >= R.lo[0] - 1 && a <= R.hi[0] + 1 && b >= R.lo[1] - 1 && b <= R.hi[1] + 1 &&
             c >= R.lo[2] - 1 && c <= R.hi[2] + 1;
    };
    if (inside1(i, j, k)) {
      const long long o = G.off(i, j, k);
      qb[QU] += G.p[o];
      qb[QV] += G.p[o + G.ns];
      qb[QW] += G.p[o + 2 * G.ns];
      qb[QT] += G.p[o + 3 * G.ns];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int di = d == 0, dj = d == 1, dk = d == 2;
      const double h = 0.5 * R.dxinv[d];
      // the gradient at e = c + s e_d reads q(c) with weight wt: central
      // differences give +h at s = -1 and -h at s = +1; the one-sided y
      // derivative of a wall's ghost row e reads e, e+1, e+2 (lower wall)
      // with -3h, 4h, -h, or e, e-1, e-2 (upper wall) with 3h, -4h, h
#pragma unroll
      for (int s = -2; s <= 2; ++s) {
        const int a = i + s * di, b = j + s * dj, c = k + s * dk;
        if (!inside1(a, b, c)) continue;
        double wt = 0.0;
        if (d == 1 && R.walls && b == R.wrow_lo) wt = (s == 0) ? -3.0 * h : (s == -1 ? 4.0 * h : (s == -2 ? -h : 0.0));
        else if (d == 1 && R.walls && b == R.wrow_hi) wt = (s == 0) ? 3.0 * h : (s == 1 ? -4.0 * h : (s == 2 ? h : 0.0));
        else wt = (s == -1) ? h : (s == 1 ? -h : 0.0);
        if (wt == 0.0) continue;
        const long long o = G.off(a, b, c);
#pragma unroll
        for (int n = 0; n < 4; ++n) qb[QU + n] += wt * G.p[o + (4 + 4 * d + n) * G.ns];
      }
    }
    // cons2prim VJP (src/rhs/CNS_hydro_K.h:15-34)
    double ub5[5];
    cons2prim_vjp(R, cl, i, j, k, qb, ub5);
#pragma unroll
    for (int n = 0; n < 5; ++n) Ub.p[ou + n * Ub.ns] = ub5[n];
  }
}

// Reverse of one stage's BLAS-1 program per valid cell: given the cotangent
// of the stage result (register S2), the cotangents of S1 (c1 times it), of the
// stage input's valid values (c2, register S2 before the program) and of dSdt
// (cd).  A register that the program does not read (its bit of `used` is clear)
// gets nothing, and its array is not read; a coefficient that is zero still
// multiplies, so a NaN or an infinity of the cotangent shows.  64^3: 20 us
// with the program reversed per value, 12 now; bound by memory.
__global__ void __launch_bounds__(256) adj_prog_kernel(BoxRec R, double c1, double c2, double cd, int used, DArr wbar,
                                                       DArr s1bar, DArr inbar, DArr vbar, long long total,
                                                       int accumulate) {
  dep_begin();
  const int nx = R.hi[0] - R.lo[0] + 1, ny = R.hi[1] - R.lo[1] + 1;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int l = (int)g, t = l / nx;
    const int i = l - t * nx + R.lo[0], k = t / ny + R.lo[2], j = t - (t / ny) * ny + R.lo[1];
    double w[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) w[n] = wbar(i, j, k, n);
    auto give = [&](const DArr& to, int reg, double c, bool add) {
      const bool any = (used >> reg) & 1;
      if (add && !any) return;
      double v[5];
#pragma unroll
      for (int n = 0; n < 5; ++n) v[n] = add ? to(i, j, k, n) : 0.0;
#pragma unroll
      for (int n = 0; n < 5; ++n) to(i, j, k, n) = v[n] + (any ? c * w[n] : 0.0);
    };
    give(s1bar, 0, c1, accumulate);
    give(inbar, 1, c2, accumulate);
    give(vbar, 2, cd, false);
  }
}

// Ghost fold: the adjoint of amrs_fill_halo_box.  Every valid cell adds the
// cotangents of the ghost cells filled from it (with the reflect_odd sign).
// The images of coordinate c along dir: itself, then the ghosts below and
// above that read it; neg: the components (bits) whose sign each changes.
__device__ __forceinline__ int images(int c, int lo, int hi, int bcl, int bch, int dir, int* out, unsigned* neg) {
  int nimg = 1;
  out[0] = c;
  neg[0] = 0u;
  const int n = hi - lo + 1;
  if (c - lo >= NGHOST && hi - c >= NGHOST) return 1;  // no ghost reads it
  for (int side = 0; side < 2; ++side) {
    const int phys = side ? bch : bcl;
    for (int gidx = 1; gidx <= NGHOST; ++gidx) {
      const int gc = side ? hi + gidx : lo - gidx;  // ghost coordinate
      int src;
      unsigned s = 0u;
      if (phys == -1) {
        int r = (gc - lo) % n;
        if (r < 0) r += n;
        src = lo + r;
      } else if (phys == 2) {
        src = side ? hi : lo;
      } else if (phys == 3 || phys == 4 || phys == 5) {
        src = side ? 2 * hi - gc + 1 : 2 * lo - gc - 1;
        s = phys == 5 ? 7u << UMX : 1u << (UMX + dir);
      } else {
        continue;
      }
      if (src == c) { out[nimg] = gc; neg[nimg] = s; ++nimg; }
    }
  }
  return nimg;
}

// `to` null: in place; otherwise the folded cotangents are added to `to`.  Cells
// more than two from every side have no images: nothing to do in place, one
// addition otherwise (64^3: 67,000 of 262,000 cells fold; computing every cell's
// images per component took 56 us, then a pass of 15 us added the result; 47 us
// component by component, 31 with five components' loads in flight).
__global__ void __launch_bounds__(256) adj_halo_kernel(HaloBox hb, DArr to, long long total) {
  dep_begin();
  const int nx = hb.hi[0] - hb.lo[0] + 1, ny = hb.hi[1] - hb.lo[1] + 1;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int l = (int)g;
    const int t = l / nx;
    const int i = l - t * nx + hb.lo[0], k = t / ny + hb.lo[2], j = t - (t / ny) * ny + hb.lo[1];
    int xi[8], yi[8], zi[8];
    unsigned xs[8], ys[8], zs[8];
    const int nxi = images(i, hb.lo[0], hb.hi[0], hb.bc_lo[0], hb.bc_hi[0], 0, xi, xs);
    const int nyi = images(j, hb.lo[1], hb.hi[1], hb.bc_lo[1], hb.bc_hi[1], 1, yi, ys);
    const int nzi = images(k, hb.lo[2], hb.hi[2], hb.bc_lo[2], hb.bc_hi[2], 2, zi, zs);
    if (!to.p && nxi * nyi * nzi == 1) continue;
    // five components at a time share the images' offsets and signs
    for (int n0 = 0; n0 < hb.ncomp; n0 += 5) {
      double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      for (int a = 0; a < nzi; ++a)
        for (int b = 0; b < nyi; ++b)
          for (int c = 0; c < nxi; ++c) {
            const double* p = hb.u.p + hb.u.off(xi[c], yi[b], zi[a]) + n0 * hb.u.ns;
            const unsigned neg = n0 == 0 ? xs[c] ^ ys[b] ^ zs[a] : 0u;  // momenta only
#pragma unroll
            for (int m = 0; m < 5; ++m) {
              const double v = n0 + m < hb.ncomp ? p[m * hb.u.ns] : 0.0;
              s[m] += (neg >> m) & 1u ? -v : v;
            }
          }
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        if (n0 + m >= hb.ncomp) break;
        if (to.p) to(i, j, k, n0 + m) += s[m];
        else hb.u(i, j, k, n0 + m) = s[m];
      }
    }
  }
}

// Reverse of the body-force source (add_source) on the valid cells:
// ubar(URHO) += vbar(UMX+d) f_d and ubar(UMX+d) += vbar(UET) f_d.
__global__ void __launch_bounds__(256) adj_source_kernel(BoxRec R, double f0, double f1, double f2, DArr vbar,
                                                         DArr ubar, long long total) {
  dep_begin();
  const int nx = R.hi[0] - R.lo[0] + 1, ny = R.hi[1] - R.lo[1] + 1;
  const double f[3] = {f0, f1, f2};
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int l = (int)g;
    const int i = l % nx + R.lo[0];
    const int t = l / nx;
    const int j = t % ny + R.lo[1];
    const int k = t / ny + R.lo[2];
    const double ve = vbar(i, j, k, UET);
    double rb = 0.0;
    for (int d = 0; d < 3; ++d) {
      if (f[d] == 0.0) continue;
      rb += vbar(i, j, k, UMX + d) * f[d];
      ubar(i, j, k, UMX + d) += ve * f[d];
    }
    ubar(i, j, k, URHO) += rb;
  }
}

// ------------------------------------------------------------ launchers --
static int grid256(long long n, int nsm, int ctas = GRID_CTAS) {
  long long b = (n + 255) / 256;
  const long long cap = (long long)nsm * ctas;
  return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

cudaError_t launch_rhs_vjp(int order, const BoxTable& tb, const AdjRecHost& ah, double* pbar, int nsm,
                           cudaStream_t st) {
  AdjRec ar;
  ar.vbar = ah.vbar;
  ar.ubar = ah.ubar;
  for (int d = 0; d < 3; ++d)
    for (int l = 0; l < 3; ++l) ar.pair[d][l] = ah.pair[d][l];
  ar.vg = ah.vg;
  ar.visc = ah.visc;
  ar.part = ah.part;
  if (pbar && !ah.part) return cudaErrorInvalidValue;
  const int H = order / 2;
  const long long n0 = ah.n[0], n1 = ah.n[1], n2 = ah.n[2];
  long long npair = 0;
  for (int d = 0; d < 3; ++d)
    for (int l = 1; l <= H; ++l) npair += (n0 + (d == 0) * l) * (n1 + (d == 1) * l) * (n2 + (d == 2) * l);
  // order 0: no KEEP pairs (the viscous part of another scheme's RHS)
  if (order == 2) launch_dep(adj_pair_kernel<2>, grid256(npair, nsm), 256, 0, st, tb, ar, npair);
  else if (order == 4) launch_dep(adj_pair_kernel<4>, grid256(npair, nsm), 256, 0, st, tb, ar, npair);
  else if (order == 6) launch_dep(adj_pair_kernel<6>, grid256(npair, nsm), 256, 0, st, tb, ar, npair);
  const long long nv = (n0 + 2) * (n1 + 2) * (n2 + 2);
  if (ah.visc) {
    const int nbv = grid256(nv, nsm, 8);  // at most 8 blocks per SM: ah.part holds 2 x 8 x nsm doubles
    launch_dep(adj_visc_kernel, nbv, 256, 0, st, tb, ar, nv, pbar);
    if (pbar) launch_dep(adj_param_sum_kernel, 1, 32, 0, st, ah.part, nbv, pbar);
  }
  const long long ng = (n0 + 6) * (n1 + 6) * (n2 + 6);
  if (order == 0) launch_dep(adj_gather_kernel<0>, grid256(ng, nsm), 256, 0, st, tb, ar, ng, 0);
  else if (order == 2) launch_dep(adj_gather_kernel<2>, grid256(ng, nsm), 256, 0, st, tb, ar, ng, H);
  else if (order == 4) launch_dep(adj_gather_kernel<4>, grid256(ng, nsm), 256, 0, st, tb, ar, ng, H);
  else launch_dep(adj_gather_kernel<6>, grid256(ng, nsm), 256, 0, st, tb, ar, ng, H);
  return cudaGetLastError();
}

cudaError_t launch_adj_prog(const BoxRec& R, const DProg& prog, const DArr& wbar, const DArr& s1bar, const DArr& inbar,
                            const DArr& vbar, int accumulate, int nsm, cudaStream_t st) {
  const long long n = (long long)(R.hi[0] - R.lo[0] + 1) * (R.hi[1] - R.lo[1] + 1) * (R.hi[2] - R.lo[2] + 1);
  // the program is linear in its registers: its reverse on the unit cotangent
  double b[3] = {0.0, 1.0, 0.0};
  bool used[3] = {false, true, false};
  for (int o = prog.nops - 1; o >= 0; --o) {
    const DOp& q = prog.ops[o];
    const double g = b[q.dst];
    const bool u = used[q.dst];
    if (q.kind == 0) {
      b[q.dst] = 0.0;
      used[q.dst] = false;
      b[q.x] += q.a * g;
      b[q.y] += q.b * g;
      used[q.x] = used[q.x] || u;
      used[q.y] = used[q.y] || u;
    } else if (q.kind == 1) {
      b[q.x] += q.a * g;
      used[q.x] = used[q.x] || u;
    } else if (q.kind == 2) {
      b[q.dst] = q.a * g;
      b[q.x] += g;
      used[q.x] = used[q.x] || u;
    } else {
      b[q.dst] = 0.0;
      used[q.dst] = false;
      b[q.x] += g;
      used[q.x] = used[q.x] || u;
    }
  }
  launch_dep(adj_prog_kernel, grid256(n, nsm), 256, 0, st, R, b[0], b[1], b[2], used[0] + 2 * used[1] + 4 * used[2], wbar,
             s1bar, inbar, vbar, n, accumulate);
  return cudaGetLastError();
}

cudaError_t launch_source_vjp(const BoxRec& R, const double force[3], const DArr& vbar, const DArr& ubar, int nsm,
                              cudaStream_t st) {
  const long long n = (long long)(R.hi[0] - R.lo[0] + 1) * (R.hi[1] - R.lo[1] + 1) * (R.hi[2] - R.lo[2] + 1);
  launch_dep(adj_source_kernel, grid256(n, nsm), 256, 0, st, R, force[0], force[1], force[2], vbar, ubar, n);
  return cudaGetLastError();
}

cudaError_t launch_adj_halo(const HaloBox& hb, const DArr* to, int nsm, cudaStream_t st) {
  const long long n = (long long)(hb.hi[0] - hb.lo[0] + 1) * (hb.hi[1] - hb.lo[1] + 1) * (hb.hi[2] - hb.lo[2] + 1);
  launch_dep(adj_halo_kernel, grid256(n, nsm), 256, 0, st, hb, to ? *to : DArr{}, n);
  return cudaGetLastError();
}

}  // namespace amrs

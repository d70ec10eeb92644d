// Face-array RHS path: the reference's kernel sequence, one kernel per
// sub-operation, flattened over a box list.  It carries the schemes that
// have no fused kernel yet (WENO5-JS LLF, MUSCL + Riemann, JST dissipation)
// and a KEEP variant kept as the "plain per-box" baseline.
//
//   Euler face fluxes  -> FaceRec::f[d]   (KEEP / WENO / Riemann)
//   JST dissipation    -> subtracted from f[d]
//   viscous averages   -> added to f[d]   (cell fluxes from visc_cell_kernel)
//   divergence + RK stage program -> output slot
//
// Operation order follows the cited reference functions and the file is
// built with -fmad=false, so results match the reference's CPU build
// (WENO5 squares its smoothness terms directly, where the reference calls
// pow(x, 2); the two can differ in the last bit).  The default WENO5 face
// kernel instead forms the nonlinear weights over a common denominator
// with explicit fused multiply-adds (weno5js_cd): the same function in
// exact arithmetic, a quarter of the divisions, rounding differences only.
#include "amrs_kernels.h"
#include "ddiv.cuh"
#include "weno_int.cuh"

namespace amrs {

// face index -> (box, direction, i, j, k) over faces nodal in d
struct FaceIdx {
  int b, d, i, j, k;
};

__device__ __forceinline__ bool decode_face(const BoxTable& tb, const FaceTable& ft, long long g, FaceIdx& f) {
  long long base = 0;
  for (int d = 0; d < 3; ++d) {
    const long long tot = ft.ftot[d];
    if (g < base + tot) {
      const long long l = g - base;
      const int b = find_box_ll(ft.fpre[d], tb.n, l);
      const BoxRec& R = box_rec(tb, b);
      const int loc = (int)(l - box_base(tb, ft.fpre[d], b));
      const int nx = R.hi[0] - R.lo[0] + 1 + (d == 0), ny = R.hi[1] - R.lo[1] + 1 + (d == 1);
      f.b = b;
      f.d = d;
      f.i = loc % nx + R.lo[0];
      const int t = loc / nx;
      f.j = t % ny + R.lo[1];
      f.k = t / ny + R.lo[2];
      return true;
    }
    base += tot;
  }
  return false;
}

__device__ __forceinline__ void decode_cell(const BoxRec& R, int loc, int g, int& i, int& j, int& k) {
  const int nx = R.hi[0] - R.lo[0] + 1 + 2 * g, ny = R.hi[1] - R.lo[1] + 1 + 2 * g;
  i = loc % nx + R.lo[0] - g;
  const int t = loc / nx;
  j = t % ny + R.lo[1] - g;
  k = t / ny + R.lo[2] - g;
}

static int grid_for(long long n, int nsm, int ctas = GRID_CTAS) {
  long long blocks = (n + 255) / 256;
  const long long cap = (long long)nsm * ctas;
  return (int)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}

// ------------------------------------------------------- KEEP, plain ----
// src/rhs/CentralKEEP.h:40-145, one face per thread, pairs summed in the
// reference's (l, m) order without sharing between faces.
template <int ORDER>
__global__ void __launch_bounds__(256)
keep_faces_plain_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  constexpr int H = ORDER / 2;
  double coef[3];
  if (ORDER == 6) { coef[0] = 6.0 / 4; coef[1] = -6.0 / 20; coef[2] = 2.0 / 60; }
  else if (ORDER == 4) { coef[0] = 4.0 / 3; coef[1] = -2.0 / 12; coef[2] = 0.0; }
  else { coef[0] = 1.0; coef[1] = 0.0; coef[2] = 0.0; }
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const DArr Q = R.q;
    const int di = f.d == 0, dj = f.d == 1, dk = f.d == 2;
    // y faces next to a code-6 wall: second-order KEEP, coefficient 1
    // (Flux_2nd_Order_KEEP, src/rhs/CentralKEEP.h:232-287)
    const bool red = f.d == 1 && R.walls && (f.j <= R.red_lo || (f.j >= R.red_hi && f.j <= R.hi[1]));
    const int hs = red ? 1 : H;
    double F[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int l = 1; l <= H; ++l)
#pragma unroll
      for (int m = 0; m < l; ++m) {
        if (l > hs) continue;
        double q1[NQ], q2[NQ], T[5];
        const long long o1 = Q.off(f.i + m * di, f.j + m * dj, f.k + m * dk);
        const long long o2 = Q.off(f.i + (m - l) * di, f.j + (m - l) * dj, f.k + (m - l) * dk);
#pragma unroll
        for (int n = 0; n < NQ; ++n) { q1[n] = Q.p[o1 + n * Q.ns]; q2[n] = Q.p[o2 + n * Q.ns]; }
        const double c = red ? 1.0 : coef[l - 1];
        if (f.d == 0) keep_pair<0>(q1, q2, c, T);
        else if (f.d == 1) keep_pair<1>(q1, q2, c, T);
        else keep_pair<2>(q1, q2, c, T);
#pragma unroll
        for (int n = 0; n < 5; ++n) F[n] = F[n] + T[n];
      }
    const DArr Fd = face_rec(tb, ft, f.b).f[f.d];
    const long long of = Fd.off(f.i, f.j, f.k);
#pragma unroll
    for (int n = 0; n < 5; ++n) Fd.p[of + n * Fd.ns] = F[n];
  }
}

// Viscous face average added to component n >= 1 of an Euler flux at face f
// (src/rhs/CNS_hydro_K.h:254-261; the mass component adds zero).
__device__ __forceinline__ double visc_average(const BoxRec& R, const FaceIdx& f, int n, double flx) {
  const DArr& V = R.vf;
  const long long s = (f.d == 0) ? 1 : (f.d == 1 ? V.js : V.ks);
  const double* v = V.p + V.off(f.i, f.j, f.k) + (4 * f.d + n - 1) * V.ns;
  return fma(0.5, v[-s] + v[0], flx);
}

// ------------------------------------------------------------- WENO5 ----
// Physical Euler fluxes + max eigenvalue: src/rhs/High_resolution.h:83-121.
#ifndef AMRS_WPF_IMUL
#define AMRS_WPF_IMUL 0x0B
#endif
__global__ void __launch_bounds__(256)
weno_flux_lambda_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, int s_in,
                        long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = find_box_ll(ft.gpre, tb.n, g);
    const BoxRec& R = box_rec(tb, b);
    const FaceRec& FR = face_rec(tb, ft, b);
    int i, j, k;
    decode_cell(R, (int)(g - box_base(tb, ft.gpre, b)), NGHOST, i, j, k);
    const DArr U = R.slot[s_in];
    const long long o = U.off(i, j, k);
    const double gam = box_cls(tb, R).gamma;
    const double rhoinv = ddiv_rn(1.0, U.p[o]);
    const double momx = U.p[o + U.ns], momy = U.p[o + 2 * U.ns], momz = U.p[o + 3 * U.ns];
    const double rhoet = U.p[o + 4 * U.ns];
    // products on the integer pipe (kmul), by bit of AMRS_WPF_IMUL: 0 the
    // velocities, 1 the kinetic energy, 2 the pressure, 3 the fluxes, 4 the
    // sound speed's argument
    constexpr int M = AMRS_WPF_IMUL;
    constexpr bool M0 = M & 1, M1 = (M >> 1) & 1, M2 = (M >> 2) & 1, M3 = (M >> 3) & 1, M4 = (M >> 4) & 1;
    const double ux = kmul<M0>(momx, rhoinv), uy = kmul<M0>(momy, rhoinv), uz = kmul<M0>(momz, rhoinv);
    const double rhoekin = kmul<M1>(kmul<M1>(0.5, rhoinv), kmul<M1>(momx, momx) + kmul<M1>(momy, momy) +
                                                               kmul<M1>(momz, momz));
    const double rhoeint = rhoet - rhoekin;
    const double P = kmul<M2>(gam - 1.0, rhoeint);
    const long long op = FR.pf[0].off(i, j, k);
    const long long ns = FR.pf[0].ns;
    double* fx = FR.pf[0].p + op;
    double* fy = FR.pf[1].p + op;
    double* fz = FR.pf[2].p + op;
    const double rhoh = rhoet + P;
    fx[0] = momx; fx[ns] = kmul<M3>(momx, ux) + P; fx[2 * ns] = kmul<M3>(momy, ux); fx[3 * ns] = kmul<M3>(momz, ux);
    fx[4 * ns] = kmul<M3>(rhoh, ux);
    fy[0] = momy; fy[ns] = kmul<M3>(momx, uy); fy[2 * ns] = kmul<M3>(momy, uy) + P; fy[3 * ns] = kmul<M3>(momz, uy);
    fy[4 * ns] = kmul<M3>(rhoh, uy);
    fz[0] = momz; fz[ns] = kmul<M3>(momx, uz); fz[2 * ns] = kmul<M3>(momy, uz); fz[3 * ns] = kmul<M3>(momz, uz) + P;
    fz[4 * ns] = kmul<M3>(rhoh, uz);
    const double cs = dsqrt_rn(kmul<M4>(kmul<M4>(gam, P), rhoinv));
    const long long ol = FR.lam.off(i, j, k);
    // |max(max(u + c, u - c), u)| of the reference: with c >= 0 and rounding
    // monotonic, fl(u + c) >= u >= fl(u - c), so the maximum is u + c itself
    // (a NaN c gives NaN either way)
    FR.lam.p[ol] = fabs(ux + cs);
    FR.lam.p[ol + FR.lam.ns] = fabs(uy + cs);
    FR.lam.p[ol + 2 * FR.lam.ns] = fabs(uz + cs);
  }
}

// WENO5-JS (src/rhs/High_resolution.h:124-159), beta[1] with the fourth power.
// Operation order of the reference; a sum x + 2^k*y (power-of-two factor,
// exact product) is one fma, which rounds exactly like the reference's
// separate multiply and add.  The four divisions are correctly rounded on
// the integer pipe (ddiv_rn): the same quotients as the reference's, at a
// fraction of the FP64 issue slots.
// Products formed on the integer pipe (kmul), by bit of M: 0 the shared 3 s2,
// 1 the (13/12) x^2 terms, 2 the quarter-scaled squares b^2 and f^2, 3 the
// fourth power of beta1, 4 the squares of eps + beta, 5 the stencil
// coefficients 7, 11, 5, 6 the final scaling, 7 the weight products.
// AMRS_WRREC_IMUL: the WENO5-Riemann face kernel's.
#ifndef AMRS_WRREC_IMUL
#define AMRS_WRREC_IMUL 0x001
#endif
template <int M>
__device__ __forceinline__ double weno5js(const double s0, const double s1, const double s2, const double s3,
                                          const double s4) {
  constexpr bool M0 = M & 1, M1 = (M >> 1) & 1, M2 = (M >> 2) & 1, M3 = (M >> 3) & 1, M4 = (M >> 4) & 1,
                 M5 = (M >> 5) & 1, M6 = (M >> 6) & 1, M7 = (M >> 7) & 1;
  const double eps = 1e-40;
  const double s2x3 = kmul<M0>(3.0, s2);
  const double a = fma(-2.0, s1, s0) + s2;         // s0 - 2 s1 + s2
  const double b = fma(-4.0, s1, s0) + s2x3;       // s0 - 4 s1 + 3 s2
  const double c = fma(-2.0, s2, s1) + s3;         // s1 - 2 s2 + s3
  const double g = s1 - s3;
  const double d = fma(-2.0, s3, s2) + s4;         // s2 - 2 s3 + s4
  const double f = fma(-4.0, s3, s2x3) + s4;       // 3 s2 - 4 s3 + s4
  // 0.25*b*b == 0.25*(b*b) and 0.25*g*g*g*g == 0.25*(((g*g)*g)*g): the
  // quarter scales exactly, so x + 0.25*y is one fma(0.25, y, x) (normal range)
  constexpr double c1312 = 13.0 / 12.0;
  const double beta0 = fma(0.25, kmul<M2>(b, b), kmul<M1>(kmul<M1>(c1312, a), a));
  const double beta1 = fma(0.25, kmul<M3>(kmul<M3>(kmul<M3>(g, g), g), g), kmul<M1>(kmul<M1>(c1312, c), c));
  const double beta2 = fma(0.25, kmul<M2>(f, f), kmul<M1>(kmul<M1>(c1312, d), d));
  const double e0 = eps + beta0, e1 = eps + beta1, e2 = eps + beta2;
  const double alpha0 = ddiv_rn(0.1, kmul<M4>(e0, e0));
  const double alpha1 = ddiv_rn(0.6, kmul<M4>(e1, e1));
  const double alpha2 = ddiv_rn(0.3, kmul<M4>(e2, e2));
  const double sum = ddiv_rn(1.0, alpha0 + alpha1 + alpha2);
  const double vl0 = fma(2.0, s0, -kmul<M5>(7.0, s1)) + kmul<M5>(11.0, s2);  // 2 s0 - 7 s1 + 11 s2
  const double vl1 = fma(2.0, s3, -s1 + kmul<M5>(5.0, s2));                  // -s1 + 5 s2 + 2 s3
  const double vl2 = fma(2.0, s2, kmul<M5>(5.0, s3)) - s4;                   // 2 s2 + 5 s3 - s4
  return kmul<M6>(kmul<M6>(1.0 / 6.0, sum),
                  kmul<M7>(alpha0, vl0) + kmul<M7>(alpha1, vl1) + kmul<M7>(alpha2, vl2));
}

// The same reconstruction, same bits, with its products and quotients on the
// integer pipe from end to end: they stay in the operands' words (dmul_core,
// ddiv_core), and `ok` collects one range test per value that enters in place
// of a test in every operation; where it ends up false the caller takes the
// plain form.  The smoothness differences are below 2^60 (weno_diff).  eps + beta is
// beta from 2^-78 up (eps is below half its last place) and eps below 2^-187 (the
// other way round); in between the hardware adds them out of line.

__device__ __forceinline__ DWords weno_sq(DWords e) { return dmul_core(e, e); }

// K x for a small integer K
template <uint32_t K>
__device__ __forceinline__ double weno_times(const ZWords& x) {
  const DWords r = dmul_small<K>(x.w);
  return dfrom(x.zero ? x.w.hi : r.hi, x.zero ? 0u : r.lo);
}

__device__ __forceinline__ double weno5js_int(const double s0, const double s1, const double s2, const double s3,
                                              const double s4, bool& ok) {
  const DWords c1312{0x3FF15555u, 0x55555555u};
  auto quarter = [](DWords w) { return DWords{w.hi - (2u << 20), w.lo}; };
  bool slow0, slow1, slow2, slow3;
  const ZWords z2 = weno_fac(s2, ok);
  const double s2x3 = weno_times<3>(z2);
  const DWords a = weno_diff(fma(-2.0, s1, s0) + s2, ok), b = weno_diff(fma(-4.0, s1, s0) + s2x3, ok);
  const double beta0 = dfrom(dadd_pos(quarter(dmul_core(b, b)), dmul_core(dmul_core(c1312, a), a)));
  const DWords alpha0 = ddiv_core(DWords{0x3FB99999u, 0x9999999Au}, weno_sq(weno_e(beta0)), &slow0);
  const DWords c = weno_diff(fma(-2.0, s2, s1) + s3, ok), g = weno_diff(s1 - s3, ok);
  const double beta1 = fma(0.25, dfrom(dmul_core(dmul_core(dmul_core(g, g), g), g)),
                           dfrom(dmul_core(dmul_core(c1312, c), c)));
  const DWords alpha1 = ddiv_core(DWords{0x3FE33333u, 0x33333333u}, weno_sq(weno_e(beta1)), &slow1);
  const DWords d = weno_diff(fma(-2.0, s3, s2) + s4, ok), f = weno_diff(fma(-4.0, s3, s2x3) + s4, ok);
  const double beta2 = fma(0.25, dfrom(dmul_core(f, f)), dfrom(dmul_core(dmul_core(c1312, d), d)));
  const DWords alpha2 = ddiv_core(DWords{0x3FD33333u, 0x33333333u}, weno_sq(weno_e(beta2)), &slow2);
  const DWords sum = ddiv_core(DWords{0x3FF00000u, 0u}, dadd_pos(dadd_pos(alpha0, alpha1), alpha2), &slow3);
  const ZWords z1 = weno_fac(s1, ok), z3 = weno_fac(s3, ok);
  // 2 s0 - 7 s1 + 11 s2, -s1 + 5 s2 + 2 s3, 2 s2 + 5 s3 - s4
  const double vl0 = fma(2.0, s0, -weno_times<7>(z1)) + weno_times<11>(z2);
  const double vl1 = fma(2.0, s3, -s1 + weno_times<5>(z2));
  const double vl2 = fma(2.0, s2, weno_times<5>(z3)) - s4;
  const double S = weno_mul(alpha0, weno_fac(vl0, ok)) + weno_mul(alpha1, weno_fac(vl1, ok)) +
                   weno_mul(alpha2, weno_fac(vl2, ok));
  ok = ok && !(slow0 || slow1 || slow2 || slow3);
  return weno_mul(dmul_core(DWords{0x3FC55555u, 0x55555555u}, sum), weno_fac(S, ok));
}

// The same reconstruction with its weights over a common denominator, for
// inputs t = 2s (the LLF halves are folded into the caller):
//   w_k = a_k / (a0+a1+a2),  a_k = c_k / e_k^2,  e_k = beta_k + eps
//   sum_k w_k v_k / 6 = (sum_k c_k v_k P_k) / (6 sum_k c_k P_k),  P_k = prod_{j!=k} e_j^2.
// 4 beta(s) is evaluated from t and eps becomes 4 eps, so the weights are
// unchanged in exact arithmetic; the 1/6 and the final 1/2 go into the v_k coefficients.
// One division instead of four; every product and sum is a fused
// multiply-add where one fits.  Range: the products P_k stay finite for
// |t| up to about 1e38 and normal for eps = 4e-40 (P_k >= 2.6e-158).
__device__ __forceinline__ double weno5js_cd(const double t0, const double t1, const double t2, const double t3,
                                             const double t4) {
  constexpr double eps4 = 4e-40;
  constexpr double c1312 = 13.0 / 12.0;
  // beta_0: (13/12) d1^2 + (1/4) d2^2
  const double d1 = fma(-2.0, t1, t0) + t2;
  const double d2 = fma(3.0, t2, fma(-4.0, t1, t0));
  const double e0 = fma(c1312 * d1, d1, fma(0.25 * d2, d2, eps4));
  // beta_1: (13/12) d3^2 + (1/4) (s1 - s3)^4; its fourth-power term is not
  // homogeneous of degree 2, so in t = 2s: 4 beta_1 = (13/12) d3^2 + (1/16) g^4
  const double d3 = fma(-2.0, t2, t1) + t3;
  const double g = t1 - t3;
  const double g2 = g * g;
  const double e1 = fma(c1312 * d3, d3, fma(0.0625 * g2, g2, eps4));
  // beta_2: (13/12) d4^2 + (1/4) d5^2
  const double d4 = fma(-2.0, t3, t2) + t4;
  const double d5 = fma(-4.0, t3, fma(3.0, t2, t4));
  const double e2 = fma(c1312 * d4, d4, fma(0.25 * d5, d5, eps4));
  const double E0 = e0 * e0, E1 = e1 * e1, E2 = e2 * e2;
  const double P0 = E1 * E2, P1 = E0 * E2, P2 = E0 * E1;
  const double den = fma(0.1, P0, fma(0.6, P1, 0.3 * P2));
  // c_k v_k / 12 with v0 = 2t0 - 7t1 + 11t2, v1 = -t1 + 5t2 + 2t3, v2 = 2t2 + 5t3 - t4
  constexpr double k0 = 0.1 / 12.0, k1 = 0.6 / 12.0, k2 = 0.3 / 12.0;
  const double v0 = fma(11.0 * k0, t2, fma(-7.0 * k0, t1, (2.0 * k0) * t0));
  const double v1 = fma(2.0 * k1, t3, fma(5.0 * k1, t2, -k1 * t1));
  const double v2 = fma(-k2, t4, fma(5.0 * k2, t3, (2.0 * k2) * t2));
  const double num = fma(v0, P0, fma(v1, P1, v2 * P2));
  return num / den;
}

// The plain form of one face and component, every operation on the FP64 pipe:
// for the lanes whose values weno5js_int does not cover.
static __device__ __noinline__ double weno_llf_plain(const double* p0, long long st, const double* u0, long long su,
                                                    double me) {
  const double hme = 0.5 * me;
  double p[6], h[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    p[q] = p0[(q - 3) * st];
    h[q] = hme * u0[(q - 3) * su];
  }
  return weno5js<0>(fma(0.5, p[0], h[0]), fma(0.5, p[1], h[1]), fma(0.5, p[2], h[2]), fma(0.5, p[3], h[3]),
                    fma(0.5, p[4], h[4])) +
         weno5js<0>(fma(0.5, p[5], -h[5]), fma(0.5, p[4], -h[4]), fma(0.5, p[3], -h[3]), fma(0.5, p[2], -h[2]),
                    fma(0.5, p[1], -h[1]));
}

// LLF-split WENO face flux (src/rhs/High_resolution.h:162-246), one thread per
// face and component (blockIdx.y).  REF_ORDER: the reference's operation
// order; otherwise the split halves 0.5 (f +- alpha U) enter weno5js_cd doubled
// as fma(+-alpha, U, f).
//
// Bound: the FP64 pipe (26 instructions per reconstruction: the differences, sums
// and splits) with the integer ALUs about as full (16 products, 5 by small
// integers, 3 additions of positive numbers, 4 quotients).  One component per
// thread instead of five in a loop: the range test and the fallback then cover one
// flux, the kernel fits three CTAs per SM (80 registers), and a small box fills the
// chip (256 x 8 x 8 tube: 1040 CTAs instead of 208).  Face kernel of the reference
// order, first with 11 of the products and the quotients on the integer pipe, one
// thread per face: 256^3 54.0 ms, now 29.0 with the viscous averages in it; 64^3
// 874 us, now 464 with them; the tube 78 us, now 39; with 2 CTAs per SM 2% more, with
// 4 (64 registers) 11% more.  The
// positive additions and products by small integers took a step at 256^3 from 103.0
// to 98.3 ms: of the five positive sums, beta_0 and the weights' sums are the ones
// that gain; with none 101.7, only the weights' 99.5, all 101.4.
template <bool REF_ORDER, bool VISC>
__global__ void __launch_bounds__(256, 3)
weno_face_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, int s_in,
                 long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  const int n = blockIdx.y;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const FaceRec& FR = face_rec(tb, ft, f.b);
    const DArr U = R.slot[s_in];
    const DArr PF = FR.pf[f.d];
    const DArr L = FR.lam;
    const long long st = (f.d == 0) ? 1 : (f.d == 1 ? L.js : L.ks);
    const long long su = (f.d == 0) ? 1 : (f.d == 1 ? U.js : U.ks);
    const long long ol = L.off(f.i, f.j, f.k) + f.d * L.ns;
    // lambda = |u| + c > 0: the integer order of the bit patterns is the
    // order of the values, and the maximum (the same value as the
    // reference's chain of rmax) needs no FP64 instruction
    long long m = __double_as_longlong(L.p[ol - 3 * st]);
#pragma unroll
    for (int q = -2; q <= 2; ++q) m = max(m, __double_as_longlong(L.p[ol + q * st]));
    const double me = __longlong_as_double(m);
    const double* u0 = U.p + U.off(f.i, f.j, f.k) + n * U.ns;
    const double* p0 = PF.p + PF.off(f.i, f.j, f.k) + n * PF.ns;
    double p[6], h[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      p[q] = p0[(q - 3) * st];
      h[q] = u0[(q - 3) * su];
    }
    double flx;
    if (!REF_ORDER) {
      flx = weno5js_cd(fma(me, h[0], p[0]), fma(me, h[1], p[1]), fma(me, h[2], p[2]), fma(me, h[3], p[3]),
                       fma(me, h[4], p[4])) +
            weno5js_cd(fma(-me, h[5], p[5]), fma(-me, h[4], p[4]), fma(-me, h[3], p[3]), fma(-me, h[2], p[2]),
                       fma(-me, h[1], p[1]));
    } else {
      // 0.5*(p + me*U) == fma(0.5, p, (0.5*me)*U): halving is exact, so the
      // split stencils round exactly as in the reference (normal range)
      const DWords hme = dwords(0.5 * me);
      bool ok = mid_range(hme.hi);
#pragma unroll
      for (int q = 0; q < 6; ++q) h[q] = weno_mul(hme, weno_fac(h[q], ok));
      flx = weno5js_int(fma(0.5, p[0], h[0]), fma(0.5, p[1], h[1]), fma(0.5, p[2], h[2]), fma(0.5, p[3], h[3]),
                        fma(0.5, p[4], h[4]), ok);
      flx += weno5js_int(fma(0.5, p[5], -h[5]), fma(0.5, p[4], -h[4]), fma(0.5, p[3], -h[3]), fma(0.5, p[2], -h[2]),
                         fma(0.5, p[1], -h[1]), ok);
      if (!ok) flx = weno_llf_plain(p0, st, u0, su, me);
    }
    if (VISC && n > 0) flx = visc_average(R, f, n, flx);
    const DArr Fd = FR.f[f.d];
    Fd.p[Fd.off(f.i, f.j, f.k) + n * Fd.ns] = flx;
  }
}

// ----------------------------------------------------------- Riemann ----
// Quotients, roots and products on the integer pipe without a range test
// each: the caller tests the values that enter (pos, vel), so that every
// operand and result is well inside the normal range, and takes a plain form
// where ok ends up false.
struct IntOps {
  bool ok = true;
  // a quotient of nonzero operands, the same with a dividend that may be
  // zero (positive divisor), a root
  __device__ __forceinline__ double div(double a, double b) const { return dfrom(ddiv_core(dwords(a), dwords(b))); }
  __device__ __forceinline__ double divz(double a, double b) const {
    const DWords w = dwords(a);
    const DWords q = ddiv_core(w, dwords(b));
    const bool zero = ((w.hi & 0x7FFFFFFFu) | w.lo) == 0u;
    return dfrom(zero ? w.hi : q.hi, zero ? w.lo : q.lo);
  }
  __device__ __forceinline__ double root(double a) const { return dfrom(dsqrt_core(dwords(a))); }
  // products of nonzero factors, and of a positive factor a with any x
  __device__ __forceinline__ double mul(double a, double b) const {
    return dfrom(dmul_core(dwords(a), dwords(b)));
  }
  __device__ __forceinline__ double mulz(double a, double x) const {
    const DWords w = dwords(x);
    const DWords r = dmul_core(dwords(a), w);
    const bool zero = ((w.hi & 0x7FFFFFFFu) | w.lo) == 0u;
    return dfrom(zero ? w.hi : r.hi, zero ? w.lo : r.lo);
  }
  // positive, in [2^-150, 2^150); zero or in [2^-400, 2^100); below 2^100
  __device__ __forceinline__ void pos(double x) {
    ok = ok && dwords(x).hi - (873u << 20) < (300u << 20);
  }
  __device__ __forceinline__ void vel(double x) {
    const DWords w = dwords(x);
    ok = ok && (w.hi * 2u - (623u << 21) < (500u << 21) || ((w.hi & 0x7FFFFFFFu) | w.lo) == 0u);
  }
  __device__ __forceinline__ void below(double x) { ok = ok && dwords(x).hi * 2u < (1123u << 21); }
  // max(x, smallp) for a finite x; the result below 2^150
  __device__ __forceinline__ double floor_p(double x, double smallp) {
    const long long b = __double_as_longlong(x), s = __double_as_longlong(smallp);
    const long long m = b < s ? s : b;
    ok = ok && dwords(x).hi * 2u < 0xFFE00000u && (uint32_t)(m >> 32) < (1173u << 20);
    return __longlong_as_double(m);
  }
};

// src/rhs/Riemann.h:9-17, with the hardware's operations.
static __device__ __noinline__ double mc_limiter_plain(double dlft, double drgt) {
  const double dcen = 0.5 * (dlft + drgt);
  const double dsgn = copysign(1.0, dcen);
  const double slop = 2.0 * rmin(fabs(dlft), fabs(drgt));
  const double dlim = (dlft * drgt >= 0.0) ? slop : 0.0;
  return dsgn * rmin(dlim, fabs(dcen));
}

// The same with one FP64 instruction (the sum): the signs, the minima and the
// scalings by 2 and 1/2 on the words.  In range: both slopes zero or in
// [2^-500, 2^500), so that their product's sign is that of the signs and the
// scalings are exact; a sum of two such is zero or above 2^-553.  (Slopes of
// opposite sign, or a zero one: the limited slope is +-0 with the sign of the
// sum.)
__device__ __forceinline__ double mc_limiter(double dlft, double drgt) {
  const DWords l = dwords(dlft), r = dwords(drgt), c = dwords(dlft + drgt);
  const uint32_t lh = l.hi & 0x7FFFFFFFu, rh = r.hi & 0x7FFFFFFFu, ch = c.hi & 0x7FFFFFFFu;
  const bool lz = (lh | l.lo) == 0u, rz = (rh | r.lo) == 0u;
  if (!((lz || lh - (523u << 20) < (1000u << 20)) && (rz || rh - (523u << 20) < (1000u << 20))))
    return mc_limiter_plain(dlft, drgt);
  // 4 min(|l|, |r|) against |l + r|: the smaller half is the limited slope
  const uint64_t al = ((uint64_t)lh << 32) | l.lo, ar = ((uint64_t)rh << 32) | r.lo;
  const uint64_t m = al < ar ? al : ar, ac = ((uint64_t)ch << 32) | c.lo;
  uint64_t d = m + (2ull << 52) < ac ? m + (2ull << 52) : ac;
  d -= 1ull << 52;
  // one zero: product +-0, min(0, .) = 0; opposite signs: dlim = 0; a zero sum
  // comes with one of the two
  if (lz || rz || (int32_t)(l.hi ^ r.hi) < 0) d = 0ull;
  return dfrom((uint32_t)(d >> 32) | (c.hi & 0x80000000u), (uint32_t)d);
}

// Characteristic slopes in direction d (src/rhs/Riemann.h:19-120) and the
// terms of the cell's extrapolations to its two faces (src/rhs/Riemann.h:251-337),
// formed once per cell instead of once per face side: A = (d0+d2)/c + d1
// (density), B = (d2-d0)/rho (normal velocity), C = (d0+d2)*c (pressure), d3,
// d4, with c the cell's sqrt(gamma R T) + 1e-40; for z (`up`) also A and C
// with the sound speed of the cell above the upper face, cell k + 2
// (cns_riemann_z's left state reads q(i,j,k+1), src/rhs/Riemann.h:316).
struct SlopeQ {
  double rho[3], un[3], p[3], t1[3], t2[3], T, Tup;  // cells c-1, c, c+1
};
static __device__ __noinline__ void slope_plain(const SlopeQ& q, double gR, double tiny, bool up, double* o) {
  const double c0 = sqrt(gR * q.T);
  const double cspeed = c0 + tiny;
  const double dpl = q.p[1] - q.p[0], dpr = q.p[2] - q.p[1];
  const double hl = 0.5 * dpl / cspeed, hr = 0.5 * dpr / cspeed;
  const double wl = 0.5 * q.rho[1] * (q.un[1] - q.un[0]), wr = 0.5 * q.rho[1] * (q.un[2] - q.un[1]);
  const double cs2 = cspeed * cspeed;
  const double d0 = mc_limiter_plain(hl - wl, hr - wr);
  const double d1 = mc_limiter_plain((q.rho[1] - q.rho[0]) - dpl / cs2, (q.rho[2] - q.rho[1]) - dpr / cs2);
  const double d2 = mc_limiter_plain(hl + wl, hr + wr);
  const double csr = c0 + 1.e-40, s02 = d0 + d2;
  o[SL_A] = s02 / csr + d1;
  o[SL_B] = (d2 - d0) / q.rho[1];
  o[SL_C] = s02 * csr;
  o[SL_T1] = mc_limiter_plain(q.t1[1] - q.t1[0], q.t1[2] - q.t1[1]);
  o[SL_T2] = mc_limiter_plain(q.t2[1] - q.t2[0], q.t2[2] - q.t2[1]);
  if (up) {
    const double csl = sqrt(gR * q.Tup) + 1.e-40;
    o[SL_AL] = s02 / csl + d1;
    o[SL_CL] = s02 * csl;
  }
}

// The same bits on the integer pipe where the ranges hold.  c0 >= 2^-78 makes
// c0 + 1e-40 = c0 + 2e-40 = c0; the halves of d0 and d2 are taken at the end
// (the limiter and the sums scale exactly), so dp / c and rho du enter whole.
// Normal velocities down to 2^-400: rho du is zero or above 2^-602, the sums of
// limited slopes zero or above 2^-708.  Transverse ones meet only the limiter.
__device__ __forceinline__ void slope_terms(const SlopeQ& q, double gR, double tiny, bool up, double o[NSLOPE]) {
  IntOps I;
#pragma unroll
  for (int n = 0; n < 3; ++n) { I.pos(q.rho[n]); I.pos(q.p[n]); I.vel(q.un[n]); }
  I.pos(gR); I.pos(q.T);
  const double c = I.root(I.mul(gR, q.T));
  I.ok = I.ok && dwords(c).hi >= (945u << 20);
  const double dpl = q.p[1] - q.p[0], dpr = q.p[2] - q.p[1];
  const double hl = I.divz(dpl, c), hr = I.divz(dpr, c);
  const double wl = I.mulz(q.rho[1], q.un[1] - q.un[0]), wr = I.mulz(q.rho[1], q.un[2] - q.un[1]);
  const double cs2 = I.mul(c, c);
  const double d0 = mc_limiter(hl - wl, hr - wr), d2 = mc_limiter(hl + wl, hr + wr);  // doubled
  const double d1 = mc_limiter((q.rho[1] - q.rho[0]) - I.divz(dpl, cs2), (q.rho[2] - q.rho[1]) - I.divz(dpr, cs2));
  const double s02 = d0 + d2;
  o[SL_A] = fma(0.5, I.divz(s02, c), d1);
  o[SL_B] = half_of(I.divz(d2 - d0, q.rho[1]));
  o[SL_C] = half_of(I.mulz(c, s02));
  o[SL_T1] = mc_limiter(q.t1[1] - q.t1[0], q.t1[2] - q.t1[1]);
  o[SL_T2] = mc_limiter(q.t2[1] - q.t2[0], q.t2[2] - q.t2[1]);
  if (up) {
    I.pos(q.Tup);
    const double cl = I.root(I.mul(gR, q.Tup));
    I.ok = I.ok && dwords(cl).hi >= (945u << 20);
    o[SL_AL] = fma(0.5, I.divz(s02, cl), d1);
    o[SL_CL] = half_of(I.mulz(cl, s02));
  }
  if (!I.ok) {
    const SlopeQ a = q;
    double r[NSLOPE];
    slope_plain(a, gR, tiny, up, r);
#pragma unroll
    for (int n = 0; n < SL_AL; ++n) o[n] = r[n];
    if (up) { o[SL_AL] = r[SL_AL]; o[SL_CL] = r[SL_CL]; }
  }
}

// Bound: both pipes (25 FP64 instructions, six quotients, a root and six
// products per cell and direction; the limiters' comparisons and scalings by
// two were 40 further FP64 instructions).  48^3, inviscid: 64 -> 28 us; four CTAs
// per SM 2.5% faster than two over the step.
__global__ void __launch_bounds__(256, 4)
slope_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, const long long* spre0,
             const long long* spre1, const long long* spre2, long long tot0, long long tot1, long long tot2) {
  dep_begin();
  if (list_idle(tb)) return;
  const long long total = tot0 + tot1 + tot2;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    int d;
    long long l;
    const long long* pre;
    if (g < tot0) { d = 0; l = g; pre = spre0; }
    else if (g < tot0 + tot1) { d = 1; l = g - tot0; pre = spre1; }
    else { d = 2; l = g - tot0 - tot1; pre = spre2; }
    const int b = find_box_ll(pre, tb.n, l);
    const BoxRec& R = box_rec(tb, b);
    const int loc = (int)(l - box_base(tb, pre, b));
    const int nx = R.hi[0] - R.lo[0] + 1 + 2 * (d == 0), ny = R.hi[1] - R.lo[1] + 1 + 2 * (d == 1);
    const int i = loc % nx + R.lo[0] - (d == 0);
    const int t = loc / nx;
    const int j = t % ny + R.lo[1] - (d == 1);
    const int k = t / ny + R.lo[2] - (d == 2);
    const DArr q = R.q;
    const DClosures& cl = box_cls(tb, R);
    const long long s = (d == 0) ? 1 : (d == 1 ? q.js : q.ks);
    const double* Q = q.p + q.off(i, j, k);
    const int QN = QU + d, QT1 = (d == 0) ? QV : QU, QT2 = (d == 2) ? QV : QW;
    const bool up = d == 2 && k <= R.hi[2];
    SlopeQ v;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      const double* c = Q + (n - 1) * s;
      v.rho[n] = c[QRHO * q.ns];
      v.un[n] = c[QN * q.ns];
      v.p[n] = c[QPRES * q.ns];
      v.t1[n] = c[QT1 * q.ns];
      v.t2[n] = c[QT2 * q.ns];
    }
    v.T = Q[QT * q.ns];
    v.Tup = up ? Q[2 * s + QT * q.ns] : v.T;
    double o[NSLOPE];
    slope_terms(v, cl.gamma * cl.Rspec, d == 0 ? 2.e-40 : 1.e-40, up, o);
    const DArr S = face_rec(tb, ft, b).slope[d];
    double* so = S.p + S.off(i, j, k);
#pragma unroll
    for (int n = 0; n < SL_AL; ++n) so[n * S.ns] = o[n];
    if (up) {
      so[SL_AL * S.ns] = o[SL_AL];
      so[SL_CL * S.ns] = o[SL_CL];
    }
  }
}

// Two-shock approximate Riemann solver (src/rhs/Riemann.h:123-249) with the
// hardware's operations, out of line: for the faces riemann_prob does not
// cover.  in = (rl, ul, pl, ut1l, ut2l, rr, ur, pr, ut1r, ut2r), out =
// (flxrho, flxu, flxut, flxutt, flxe).
static __device__ __noinline__ void riemann_plain(const double gamma, const double smallp, const double* in,
                                                  double* out) {
  const double rl = in[0], ul = in[1], pl = in[2], ut1l = in[3], ut2l = in[4];
  const double rr = in[5], ur = in[6], pr = in[7], ut1r = in[8], ut2r = in[9];
  const double weakwv = 1.e-3;
  const double small = 1.e-6;
  const double clsql = gamma * pl * rl;
  const double clsqr = gamma * pr * rr;
  double wl = sqrt(clsql);
  double wr = sqrt(clsqr);
  const double cleft = ((wl) / (rl));
  const double cright = ((wr) / (rr));
  const double ccsmall = small * (cleft + cright);
  double pstar = ((wl * pr + wr * pl - wr * wl * (ur - ul)) / (wl + wr));
  pstar = rmax(pstar, smallp);
  double pstnm1 = pstar;
  double wlsq = (0.5 * (gamma - 1.) * (pstar + pl) + pstar) * rl;
  double wrsq = (0.5 * (gamma - 1.) * (pstar + pr) + pstar) * rr;
  wl = sqrt(wlsq);
  wr = sqrt(wrsq);
  double ustarp = ul - ((pstar - pl) / (wl));
  double ustarm = ur + ((pstar - pr) / (wr));
  pstar = ((wl * pr + wr * pl - wr * wl * (ur - ul)) / (wl + wr));
  pstar = rmax(pstar, smallp);
  double ustar = 0.0;
  for (int iter = 0; iter < 3; ++iter) {
    wlsq = (0.5 * (gamma - 1.) * (pstar + pl) + pstar) * rl;
    wrsq = (0.5 * (gamma - 1.) * (pstar + pr) + pstar) * rr;
    wl = ((1.) / (sqrt(wlsq)));
    wr = ((1.) / (sqrt(wrsq)));
    const double ustnm1 = ustarm;
    const double ustnp1 = ustarp;
    ustarm = ur - (pr - pstar) * wr;
    ustarp = ul + (pl - pstar) * wl;
    const double dpditer = fabs(pstnm1 - pstar);
    double zp = fabs(ustarp - ustnp1);
    if (zp - weakwv * cleft < 0.0) zp = dpditer * wl;
    double zm = fabs(ustarm - ustnm1);
    if (zm - weakwv * cright < 0.0) zm = dpditer * wr;
    const double zz = zp + zm;
    const double denom = ((dpditer) / (rmax(zz, ccsmall)));
    pstnm1 = pstar;
    pstar = pstar - denom * (ustarm - ustarp);
    pstar = rmax(pstar, smallp);
    ustar = 0.5 * (ustarm + ustarp);
  }
  double ro, uo, po, sgnm, utrans1, utrans2;
  if (ustar > 0.) {
    ro = rl; uo = ul; po = pl; sgnm = 1.; utrans1 = ut1l; utrans2 = ut2l;
  } else if (ustar < 0.) {
    ro = rr; uo = ur; po = pr; sgnm = -1.; utrans1 = ut1r; utrans2 = ut2r;
  } else {
    uo = 0.5 * (ur + ul);
    po = 0.5 * (pr + pl);
    ro = ((2. * (rl * rr)) / (rl + rr));
    sgnm = 1.;
    utrans1 = 0.5 * (ut1l + ut1r);
    utrans2 = 0.5 * (ut2l + ut2r);
  }
  const double wosq = (0.5 * (gamma - 1.) * (pstar + po) + pstar) * ro;
  const double dpjmp = pstar - po;
  const double suo = sgnm * uo;
  double rgdnv, ugdnv, pgdnv;
  // The reference evaluates every wave speed and the star density before it
  // selects the state; here each is evaluated on the branch that reads it
  // (same operations, same values, same selection, NaN included).
  auto mixed = [&](double spin, double spout, double rstar) {
    const double ss = rmax(spout - spin, spout + spin);
    const double frac = 0.5 * (1. + ((spin + spout) / (rmax(ss, ccsmall))));
    rgdnv = frac * rstar + (1. - frac) * ro;
    ugdnv = frac * ustar + (1. - frac) * uo;
    pgdnv = frac * pstar + (1. - frac) * po;
  };
  if (pstar >= po) {
    // shock: spout == spin, so the side state or the star state
    const double spin = ((sqrt(wosq)) / (ro)) - suo;
    if (spin < 0.) {
      rgdnv = ro; ugdnv = uo; pgdnv = po;
    } else if (spin >= 0.) {
      rgdnv = ((ro) / (1. - ((ro * dpjmp) / (wosq)))); ugdnv = ustar; pgdnv = pstar;
    } else {
      mixed(spin, spin, ((ro) / (1. - ((ro * dpjmp) / (wosq)))));
    }
  } else {
    const double rstar = ((ro) / (1. - ((ro * dpjmp) / (wosq))));
    const double spout = sqrt(((gamma * po) / (ro))) - suo;
    const double spin = sqrt(((gamma * pstar) / (rstar))) - suo;
    if (spout < 0.) {
      rgdnv = ro; ugdnv = uo; pgdnv = po;
    } else if (spin >= 0.) {
      rgdnv = rstar; ugdnv = ustar; pgdnv = pstar;
    } else {
      mixed(spin, spout, rstar);
    }
  }
  out[0] = rgdnv * ugdnv;
  out[1] = rgdnv * ugdnv * ugdnv + pgdnv;
  out[2] = rgdnv * ugdnv * utrans1;
  out[3] = rgdnv * ugdnv * utrans2;
  // (0.5*r)*k + x == fma(0.5, r*k, x): the halving is exact (normal range)
  out[4] = ugdnv * (fma(0.5, rgdnv * (ugdnv * ugdnv + utrans1 * utrans1 + utrans2 * utrans2), ((pgdnv) / (gamma - 1.))) +
                  pgdnv);
}

// The same solver, same bits, with its quotients and roots and most of its
// products on the integer pipe.  The faces whose states are all in the tested
// ranges (densities and pressures in 2^+-150, velocities below 2^100, star
// pressure finite and, after its floor, below 2^150) need no range test in any
// operation: every intermediate then stays well inside the normal range, but for
// the four products of a velocity, which are on the FP64 pipe.  (Velocities as
// small as they come are ordinary: fluid at rest beside moving fluid has them down
// to zero within a few cells.  With a lower bound of 2^-100 a step at 96^3 in such a
// state took 13.4 ms, with every face in riemann_plain, and takes 3.95 now; the FP64
// products cost 0.7% elsewhere.)
// Comparisons of values of known sign are integer comparisons of their bits.
// A transonic fan and a star state outside the ranges take riemann_plain.
// 76 FP64 instructions (sums, the flux products) and 17 quotients, 11 roots and
// 56 products on the integer pipe; with the products on the FP64 pipe the MUSCL
// step at 96^3 takes 3.61 ms instead of 2.94, with any one group of them 2-13%
// more.
__device__ __forceinline__ void riemann_prob(const double gamma, const double smallp, const double in[10],
                                             double out[5]) {
  const double rl = in[0], ul = in[1], pl = in[2], ut1l = in[3], ut2l = in[4];
  const double rr = in[5], ur = in[6], pr = in[7], ut1r = in[8], ut2r = in[9];
  IntOps R;
  R.pos(rl); R.pos(pl); R.pos(rr); R.pos(pr);
  R.below(ul); R.below(ur); R.below(ut1l); R.below(ut2l); R.below(ut1r); R.below(ut2r);
  auto bits = [](double x) { return __double_as_longlong(x); };
  const double hg = 0.5 * (gamma - 1.);
  R.pos(gamma); R.pos(hg);
  double wl = R.root(R.mul(R.mul(gamma, pl), rl));
  double wr = R.root(R.mul(R.mul(gamma, pr), rr));
  const double cleft = R.div(wl, rl), cright = R.div(wr, rr);
  const double wkl = R.mul(1.e-3, cleft), wkr = R.mul(1.e-3, cright);
  const double ccsmall = R.mul(1.e-6, cleft + cright);
  const double du = ur - ul;
  auto star = [&]() {
    const double num = R.mul(wl, pr) + R.mul(wr, pl) - R.mul(wr, wl) * du;
    return R.floor_p(R.divz(num, wl + wr), smallp);
  };
  auto wsq = [&](double ps, double p, double r) { return R.mul(R.mul(hg, ps + p) + ps, r); };
  double pstar = star();
  double pstnm1 = pstar;
  wl = R.root(wsq(pstar, pl, rl));
  wr = R.root(wsq(pstar, pr, rr));
  double ustarp = ul - R.divz(pstar - pl, wl);
  double ustarm = ur + R.divz(pstar - pr, wr);
  pstar = star();
#pragma unroll 1
  for (int iter = 0; iter < 3; ++iter) {
    wl = R.div(1., R.root(wsq(pstar, pl, rl)));
    wr = R.div(1., R.root(wsq(pstar, pr, rr)));
    const double ustnm1 = ustarm, ustnp1 = ustarp;
    ustarm = ur - R.mulz(wr, pr - pstar);
    ustarp = ul + R.mulz(wl, pl - pstar);
    const double dpditer = fabs(pstnm1 - pstar);
    // zp - weakwv * cleft < 0 exactly when zp < weakwv * cleft, both >= 0
    double zp = fabs(ustarp - ustnp1), zm = fabs(ustarm - ustnm1);
    if (bits(zp) < bits(wkl)) zp = R.mulz(wl, dpditer);
    if (bits(zm) < bits(wkr)) zm = R.mulz(wr, dpditer);
    const double zz = zp + zm;
    const double denom = R.divz(dpditer, bits(zz) < bits(ccsmall) ? ccsmall : zz);
    pstnm1 = pstar;
    // (a product with a factor that may be zero on either side: on the FP64 pipe)
    pstar = R.floor_p(pstar - denom * (ustarm - ustarp), smallp);
  }
  const double ustar = 0.5 * (ustarm + ustarp);
  double ro, uo, po, utrans1, utrans2;
  const bool right = bits(ustar) < 0 && (bits(ustar) << 1) != 0;
  double suo;
  if (right) {
    ro = rr; uo = ur; po = pr; utrans1 = ut1r; utrans2 = ut2r;
    suo = -uo;
  } else {
    ro = rl; uo = ul; po = pl; utrans1 = ut1l; utrans2 = ut2l;
    if ((bits(ustar) << 1) == 0) {
      uo = 0.5 * (ur + ul);
      po = 0.5 * (pr + pl);
      ro = R.div(2. * (rl * rr), rl + rr);
      utrans1 = 0.5 * (ut1l + ut1r);
      utrans2 = 0.5 * (ut2l + ut2r);
    }
    suo = uo;
  }
  const double wosq = wsq(pstar, po, ro);
  const double dpjmp = pstar - po;
  const double den = 1. - R.divz(R.mulz(ro, dpjmp), wosq);
  const double rstar = R.div(ro, den);
  R.pos(den); R.pos(rstar);
  double spin, spout;
  if (bits(pstar) >= bits(po)) {
    spin = spout = R.div(R.root(wosq), ro) - suo;
  } else {
    spout = R.root(R.div(R.mul(gamma, po), ro)) - suo;
    spin = R.root(R.div(R.mul(gamma, pstar), rstar)) - suo;
  }
  double rg = rstar, ug = ustar, pg = pstar;
  if (bits(spout) < 0) {
    rg = ro; ug = uo; pg = po;
  } else if (bits(spin) < 0) {
    R.ok = false;  // inside a transonic fan
  }
  const double m = rg * ug;
  out[0] = m;
  out[1] = m * ug + pg;
  out[2] = m * utrans1;
  out[3] = m * utrans2;
  out[4] = ug * (fma(0.5, rg * (ug * ug + utrans1 * utrans1 + utrans2 * utrans2), R.div(pg, gamma - 1.)) + pg);
  if (!R.ok) {
    double a[10], o[5];
#pragma unroll
    for (int n = 0; n < 10; ++n) a[n] = in[n];
    riemann_plain(gamma, smallp, a, o);
#pragma unroll
    for (int n = 0; n < 5; ++n) out[n] = o[n];
  }
}

// MUSCL face states + Riemann flux (src/rhs/Riemann.h:251-337).  Bound: the FP64
// pipe (76% busy at 128^3, 122 instructions a face) behind the solver's serial chain
// of quotients and roots; two CTAs per SM (128 registers) beat three (2.94 against
// 3.10 ms per step at 96^3).  48^3, with the hardware's roots and products and
// checked integer quotients before: 194 -> 86 us.
template <bool VISC>
__global__ void __launch_bounds__(256, 2)
riemann_face_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const int d = f.d;
    const DArr q = R.q;
    const DArr S = face_rec(tb, ft, f.b).slope[d];
    const DClosures& cl = box_cls(tb, R);
    const int QN = QU + d, QT1 = (d == 0) ? QV : QU, QT2 = (d == 2) ? QV : QW;
    const int UN = UMX + d, UT1 = (d == 0) ? UMY : UMX, UT2 = (d == 2) ? UMY : UMZ;
    const int im = f.i - (d == 0), jm = f.j - (d == 1), km = f.k - (d == 2);
    const long long oq = q.off(f.i, f.j, f.k), oqm = q.off(im, jm, km);
    const long long os = S.off(f.i, f.j, f.k), osm = S.off(im, jm, km);
    auto Q = [&](long long off, int n) { return q.p[off + n * q.ns]; };
    auto D = [&](long long off, int n) { return S.p[off + n * S.ns]; };
    const double gam = cl.gamma;
    // left state from cell i-1, right state from cell i, with the terms
    // slope_kernel formed (z: the left terms with the quirk's sound speed);
    // q + 0.5*t == fma(0.5, t, q): the halving is exact (normal range)
    const int cA = (d == 2) ? SL_AL : SL_A, cC = (d == 2) ? SL_CL : SL_C;
    const double in[10] = {rmax(fma(0.5, D(osm, cA), Q(oqm, QRHO)), 1.0e-40),
                           fma(0.5, D(osm, SL_B), Q(oqm, QN)),
                           rmax(fma(0.5, D(osm, cC), Q(oqm, QPRES)), 1.0e-40),
                           fma(0.5, D(osm, SL_T1), Q(oqm, QT1)),
                           fma(0.5, D(osm, SL_T2), Q(oqm, QT2)),
                           rmax(fma(-0.5, D(os, SL_A), Q(oq, QRHO)), 1.0e-40),
                           fma(-0.5, D(os, SL_B), Q(oq, QN)),
                           rmax(fma(-0.5, D(os, SL_C), Q(oq, QPRES)), 1.0e-40),
                           fma(-0.5, D(os, SL_T1), Q(oq, QT1)),
                           fma(-0.5, D(os, SL_T2), Q(oq, QT2))};
    double F[5];
    riemann_prob(gam, 1.0e-40, in, F);
    const DArr Fd = face_rec(tb, ft, f.b).f[d];
    const long long of = Fd.off(f.i, f.j, f.k);
    const int comp_of[5] = {URHO, UN, UT1, UT2, UET};
#pragma unroll
    for (int n = 0; n < 5; ++n)
      Fd.p[of + comp_of[n] * Fd.ns] = VISC && n > 0 ? visc_average(R, f, comp_of[n], F[n]) : F[n];
  }
}

// WENO5-Riemann faces (riemann_weno = 1), an extension with no counterpart in
// the reference (which pairs WENO5 only with the Lax-Friedrichs split and
// the two-shock solver only with MUSCL): rho, u_n, p, u_t1, u_t2 are
// reconstructed to the face from each side with weno5js (left state: cells
// i-3..i+1; right state: the mirror i+2..i-2), rho and p floored at 1e-40
// as the MUSCL states are (src/rhs/Riemann.h:260-272), and riemann_prob
// gives the flux.  One thread per face.
template <bool VISC>
__global__ void __launch_bounds__(256)
weno_riemann_face_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const int d = f.d;
    const DArr q = R.q;
    const DClosures& cl = box_cls(tb, R);
    const int QN = QU + d, QT1 = (d == 0) ? QV : QU, QT2 = (d == 2) ? QV : QW;
    const int UN = UMX + d, UT1 = (d == 0) ? UMY : UMX, UT2 = (d == 2) ? UMY : UMZ;
    const long long sq = (d == 0) ? 1 : (d == 1 ? q.js : q.ks);
    const long long o = q.off(f.i, f.j, f.k);
    const int comp[5] = {QRHO, QN, QPRES, QT1, QT2};
    double lft[5], rgt[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double* p = q.p + o + comp[m] * q.ns;
      double v[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) v[t] = p[(t - 3) * sq];
      lft[m] = weno5js<AMRS_WRREC_IMUL>(v[0], v[1], v[2], v[3], v[4]);
      rgt[m] = weno5js<AMRS_WRREC_IMUL>(v[5], v[4], v[3], v[2], v[1]);
    }
    const double in[10] = {rmax(lft[0], 1.0e-40), lft[1], rmax(lft[2], 1.0e-40), lft[3], lft[4],
                           rmax(rgt[0], 1.0e-40), rgt[1], rmax(rgt[2], 1.0e-40), rgt[3], rgt[4]};
    double F[5];
    riemann_prob(cl.gamma, 1.0e-40, in, F);
    const DArr Fd = face_rec(tb, ft, f.b).f[d];
    const long long of = Fd.off(f.i, f.j, f.k);
    const int comp_of[5] = {URHO, UN, UT1, UT2, UET};
#pragma unroll
    for (int n = 0; n < 5; ++n)
      Fd.p[of + comp_of[n] * Fd.ns] = VISC && n > 0 ? visc_average(R, f, comp_of[n], F[n]) : F[n];
  }
}

// --------------------------------------------------------------- JST ----
__device__ __forceinline__ double discon_sensor(double pp, double pl, double pr) {
  // src/rhs/CNS_hydro_K.h:39-44
  const double pjst = pr + 2.0 * pp + pl;
  const double ptvd = fabs(pr - pp) + fabs(pp - pl);
  return fabs(ddiv_rn(2.0 * (pr - 2.0 * pp + pl), pjst + ptvd + 1.0e-40));
}

// Sensor and spectral radius on the valid box (src/rhs/CNS_hydro_K.h:46-75);
// the arrays are zeroed beforehand, as the reference zeroes its MultiFabs.
__global__ void __launch_bounds__(256)
jst_sensor_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = find_box_ll(ft.vpre, tb.n, g);
    const BoxRec& R = box_rec(tb, b);
    int i, j, k;
    decode_cell(R, (int)(g - box_base(tb, ft.vpre, b)), 0, i, j, k);
    const DArr q = R.q;
    const long long o = q.off(i, j, k);
    auto P = [&](long long off) { return q.p[off + QPRES * q.ns]; };
    const double pp = P(o);
    const FaceRec& FR = face_rec(tb, ft, b);
    const long long os = FR.sen.off(i, j, k);
    FR.sen.p[os] = discon_sensor(pp, P(o - 1), P(o + 1));
    FR.sen.p[os + FR.sen.ns] = discon_sensor(pp, P(o - q.js), P(o + q.js));
    FR.sen.p[os + 2 * FR.sen.ns] = discon_sensor(pp, P(o - q.ks), P(o + q.ks));
    const double ux = q.p[o + QU * q.ns], uy = q.p[o + QV * q.ns], uz = q.p[o + QW * q.ns];
    const double cs = dsqrt_rn(ddiv_rn(box_cls(tb, R).gamma * pp, q.p[o + QRHO * q.ns]));
    FR.lam.p[os] = fabs(ux) + cs;
    FR.lam.p[os + FR.lam.ns] = fabs(uy) + cs;
    FR.lam.p[os + 2 * FR.lam.ns] = fabs(uz) + cs;
  }
}

// JST dissipation subtracted from face fluxes (src/rhs/CNS_hydro_K.h:78-104);
// y and z read component 0 of sensor and lambda, and the z fourth
// difference uses k-1 three times, as in the reference.
__global__ void __launch_bounds__(256)
jst_face_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, int s_in,
                long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const FaceRec& FR = face_rec(tb, ft, f.b);
    const DClosures& cl = box_cls(tb, R);
    const DArr U = R.slot[s_in];
    const long long s = (f.d == 0) ? 1 : (f.d == 1 ? U.js : U.ks);
    const long long sl = (f.d == 0) ? 1 : (f.d == 1 ? FR.sen.js : FR.sen.ks);
    const long long ou = U.off(f.i, f.j, f.k), ol = FR.sen.off(f.i, f.j, f.k);
    const double sen = cl.Cshock * rmax(FR.sen.p[ol - sl], FR.sen.p[ol]);
    const double rr = rmax(FR.lam.p[ol - sl], FR.lam.p[ol]);
    const DArr Fd = FR.f[f.d];
    const long long of = Fd.off(f.i, f.j, f.k);
    for (int n = 0; n < 5; ++n) {
      const long long on = ou + n * U.ns;
      const double dw = (U.p[on] - U.p[on - s]);
      double fdamp;
      if (f.d < 2) fdamp = U.p[on + s] - 3.0 * U.p[on] + 3.0 * U.p[on - s] - U.p[on - 2 * s];
      else fdamp = U.p[on - s] - 3.0 * U.p[on] + 3.0 * U.p[on - s] - U.p[on - s];
      Fd.p[of + n * Fd.ns] -= (sen * dw - rmax(0.0, cl.Cdamp - sen) * fdamp) * rr;
    }
  }
}

// ---------------------------------------------- viscous face average ----
// src/rhs/CNS_hydro_K.h:254-261 (mass component adds zero and is skipped).
__global__ void __launch_bounds__(256)
visc_face_add_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    FaceIdx f;
    if (!decode_face(tb, ft, g, f)) continue;
    const BoxRec& R = box_rec(tb, f.b);
    const DArr V = R.vf;
    const long long s = (f.d == 0) ? 1 : (f.d == 1 ? V.js : V.ks);
    const long long ov = V.off(f.i, f.j, f.k);
    const DArr Fd = face_rec(tb, ft, f.b).f[f.d];
    const long long of = Fd.off(f.i, f.j, f.k);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int c = 4 * f.d + n;
      Fd.p[of + (1 + n) * Fd.ns] = fma(0.5, V.p[ov - s + c * V.ns] + V.p[ov + c * V.ns], Fd.p[of + (1 + n) * Fd.ns]);
    }
  }
}

// --------------------------------------- divergence + stage program ----
// src/tim/CNS_advance.cpp:384-390, then the BLAS-1 program of the stage; one
// thread per cell and component (blockIdx.y), every load issued before the first
// product (their range tests are branches that loads do not cross).  Bound: the
// loads' latency and the FP64 pipe (25 to 35 instructions per cell with every
// product on the integer pipe, 60 to 75 before).  256^3: 2.07 -> 1.46 ms per stage
// (products moved, loads in program order: 1.87; one thread per cell: 2.97).
__global__ void __launch_bounds__(256, 5)
div_stage_kernel(const __grid_constant__ BoxTable tb, const __grid_constant__ FaceTable ft, int s_in, int s_s1,
                 int s_out, DProg prog_in, int rhs_only, long long total) {
  dep_begin();
  if (list_idle(tb)) return;
  const DProg prog = resolve_prog(prog_in);
  const int n = blockIdx.y;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = find_box_ll(ft.vpre, tb.n, g);
    const BoxRec& R = box_rec(tb, b);
    const FaceRec& FR = face_rec(tb, ft, b);
    const int loc = (int)(g - box_base(tb, ft.vpre, b));
    const int nx = R.hi[0] - R.lo[0] + 1, ny = R.hi[1] - R.lo[1] + 1;
    const int t = loc / nx, i = loc - t * nx, k = t / ny, j = t - k * ny;  // in the box
    // face arrays: rows of nx + 1, nx, nx (nodal in their direction)
    const double* px = FR.f[0].p + n * FR.f[0].ns + (loc + t);
    const double* py = FR.f[1].p + n * FR.f[1].ns + (loc + k * nx);
    const double* pz = FR.f[2].p + n * FR.f[2].ns + loc;
    const DArr &Uin = R.slot[s_in], &U1 = R.slot[s_s1], &Uo = R.slot[s_out];
    const int gi = i + R.lo[0], gj = j + R.lo[1], gk = k + R.lo[2];
    const double x0 = px[0], x1 = px[1], y0 = py[0], y1 = py[nx], z0 = pz[0], z1 = pz[nx * ny];
    double s1 = 0.0, s2 = 0.0;
    if (!rhs_only) {
      s1 = U1(gi, gj, gk, n);
      s2 = Uin(gi, gj, gk, n);
    }
    double ds = dmul_rn(R.dxinv[0], x0 - x1) + dmul_rn(R.dxinv[1], y0 - y1) + dmul_rn(R.dxinv[2], z0 - z1);
    const DClosures& cl = box_cls(tb, R);
    if (cl.source) ds = add_source(cl, Uin.p, Uin.off(gi, gj, gk), Uin.ns, n, ds);
    Uo(gi, gj, gk, n) = rhs_only ? ds : apply_prog(prog, s1, s2, ds);
  }
}

// ------------------------------------------------------------ launchers --
cudaError_t launch_keep_faces_plain(int order, const BoxTable& tb, const FaceTable& ft, long long nfaces[3], int nsm,
                                    cudaStream_t st) {
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  const int grid = grid_for(tot, nsm);
  if (order == 2) launch_dep(keep_faces_plain_kernel<2>, grid, 256, 0, st, tb, ft, tot);
  else if (order == 4) launch_dep(keep_faces_plain_kernel<4>, grid, 256, 0, st, tb, ft, tot);
  else launch_dep(keep_faces_plain_kernel<6>, grid, 256, 0, st, tb, ft, tot);
  return cudaGetLastError();
}

cudaError_t launch_weno_point(const BoxTable& tb, const FaceTable& ft, int s_in, long long ngcells, int nsm,
                              cudaStream_t st) {
  launch_dep(weno_flux_lambda_kernel, grid_for(ngcells, nsm), 256, 0, st, tb, ft, s_in, ngcells);
  return cudaGetLastError();
}

cudaError_t launch_weno_faces(const BoxTable& tb, const FaceTable& ft, int s_in, long long nfaces[3], bool ref_order,
                              bool visc, int nsm, cudaStream_t st) {
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  // one face per thread whatever the size: at 256^3 31.0 ms a launch against 31.8
  // with 60 blocks per SM and component
  const dim3 grid(grid_for(tot, nsm, 1 << 18), NCONS);
  if (ref_order && visc) launch_dep(weno_face_kernel<true, true>, grid, 256, 0, st, tb, ft, s_in, tot);
  else if (ref_order) launch_dep(weno_face_kernel<true, false>, grid, 256, 0, st, tb, ft, s_in, tot);
  else if (visc) launch_dep(weno_face_kernel<false, true>, grid, 256, 0, st, tb, ft, s_in, tot);
  else launch_dep(weno_face_kernel<false, false>, grid, 256, 0, st, tb, ft, s_in, tot);
  return cudaGetLastError();
}

cudaError_t launch_weno(const BoxTable& tb, const FaceTable& ft, int s_in, long long ngcells, long long nfaces[3],
                        bool ref_order, bool visc, int nsm, cudaStream_t st) {
  launch_dep(weno_flux_lambda_kernel, grid_for(ngcells, nsm), 256, 0, st, tb, ft, s_in, ngcells);
  return launch_weno_faces(tb, ft, s_in, nfaces, ref_order, visc, nsm, st);
}

cudaError_t launch_slopes(const BoxTable& tb, const FaceTable& ft, const long long* spre_d[3], long long nslope[3],
                          int nsm, cudaStream_t st) {
  const long long ts = nslope[0] + nslope[1] + nslope[2];
  launch_dep(slope_kernel, grid_for(ts, nsm), 256, 0, st, tb, ft, spre_d[0], spre_d[1], spre_d[2], nslope[0], nslope[1],
                                                  nslope[2]);
  return cudaGetLastError();
}

cudaError_t launch_riemann(const BoxTable& tb, const FaceTable& ft, const long long* spre_d[3], long long nslope[3],
                           long long nfaces[3], bool visc, int nsm, cudaStream_t st) {
  const long long ts = nslope[0] + nslope[1] + nslope[2];
  launch_dep(slope_kernel, grid_for(ts, nsm), 256, 0, st, tb, ft, spre_d[0], spre_d[1], spre_d[2], nslope[0], nslope[1],
                                                  nslope[2]);
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  if (visc) launch_dep(riemann_face_kernel<true>, grid_for(tot, nsm, 12), 256, 0, st, tb, ft, tot);
  else launch_dep(riemann_face_kernel<false>, grid_for(tot, nsm, 12), 256, 0, st, tb, ft, tot);
  return cudaGetLastError();
}

cudaError_t launch_weno_riemann(const BoxTable& tb, const FaceTable& ft, long long nfaces[3], bool visc, int nsm,
                                cudaStream_t st) {
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  if (visc) launch_dep(weno_riemann_face_kernel<true>, grid_for(tot, nsm, 12), 256, 0, st, tb, ft, tot);
  else launch_dep(weno_riemann_face_kernel<false>, grid_for(tot, nsm, 12), 256, 0, st, tb, ft, tot);
  return cudaGetLastError();
}

cudaError_t launch_jst_sensor(const BoxTable& tb, const FaceTable& ft, long long nvalid, int nsm, cudaStream_t st) {
  launch_dep(jst_sensor_kernel, grid_for(nvalid, nsm), 256, 0, st, tb, ft, nvalid);
  return cudaGetLastError();
}

cudaError_t launch_jst(const BoxTable& tb, const FaceTable& ft, int s_in, long long ngcells, long long nvalid,
                       long long nfaces[3], int nsm, cudaStream_t st) {
  (void)ngcells;
  launch_dep(jst_sensor_kernel, grid_for(nvalid, nsm), 256, 0, st, tb, ft, nvalid);
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  launch_dep(jst_face_kernel, grid_for(tot, nsm), 256, 0, st, tb, ft, s_in, tot);
  return cudaGetLastError();
}

cudaError_t launch_visc_face_add(const BoxTable& tb, const FaceTable& ft, long long nfaces[3], int nsm,
                                 cudaStream_t st) {
  const long long tot = nfaces[0] + nfaces[1] + nfaces[2];
  launch_dep(visc_face_add_kernel, grid_for(tot, nsm), 256, 0, st, tb, ft, tot);
  return cudaGetLastError();
}

cudaError_t launch_div_stage(const BoxTable& tb, const FaceTable& ft, int s_in, int s_s1, int s_out,
                             const DProg& prog, int rhs_only, long long nvalid, int nsm, cudaStream_t st) {
  launch_dep(div_stage_kernel, dim3(grid_for(nvalid, nsm, 8), NCONS), 256, 0, st, tb, ft, s_in, s_s1, s_out, prog, rhs_only, nvalid);
  return cudaGetLastError();
}

}  // namespace amrs

// Device-side types and point functions of the compressible RHS path.
//
// Every function keeps the floating-point operation order of the reference
// function it cites, and the forward translation units are compiled with
// -fmad=false, so results are bit-identical to the reference's CPU build
// (the reverse-mode units, which recompute linearisation points with these
// functions, allow contraction).
// Explicit fma() appears only where one multiplicand is a power of two
// (exact product), which rounds identically to the separate mul + add.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "ddiv.cuh"

namespace amrs {

constexpr int URHO = 0, UMX = 1, UMY = 2, UMZ = 3, UET = 4, NCONS = 5;
// primitive components; QE = cv*T, stored so KEEP reads it instead of recomputing
constexpr int QRHO = 0, QU = 1, QV = 2, QW = 3, QT = 4, QPRES = 5, QE = 6, NQ = 7;
constexpr int NGHOST = 3;
constexpr int NVF = 12;  // viscous cell fluxes: x,y,z directions x (UMX..UET)
// MUSCL face-state terms per cell and direction (see slope_kernel): the
// Riemann faces' L/R extrapolations read them instead of the raw slopes
constexpr int SL_A = 0, SL_B = 1, SL_C = 2, SL_T1 = 3, SL_T2 = 4, SL_AL = 5, SL_CL = 6, NSLOPE = 7;

// Array4-like view (amrex::Array4<Real>).
struct DArr {
  double* p;
  long long js, ks, ns;
  int b0, b1, b2;
  __host__ __device__ __forceinline__ double& operator()(int i, int j, int k, int n = 0) const {
    return p[(long long)(i - b0) + (long long)(j - b1) * js + (long long)(k - b2) * ks + (long long)n * ns];
  }
  __host__ __device__ __forceinline__ long long off(int i, int j, int k) const {
    return (long long)(i - b0) + (long long)(j - b1) * js + (long long)(k - b2) * ks;
  }
};

// Closures on the device (src/cls/Closures.h:72-182).
struct DClosures {
  double gamma, cv, cp, Rspec;
  int visc_law, cond_law;
  double visc_ref, Tvisc_ref, cond_ref, Tcond_ref;
  double Cshock, Cdamp;
  int source;       // cns.rhs_source with a body force
  double force[3];  // body force per unit mass
};

// compute_rhs's source step (src/tim/CNS_advance.cpp:396-407) with the
// channel problem's user_source (exm/Channel/prob.h:189-193: rhs(UMX) +=
// rho fx, rhs(UET) += m_x fx) for a body force f per unit mass: component n
// of the cell's RHS `ds` gets rho f_d (n = UMX+d) or the m_d f_d in x, y, z
// order (n = UET), for every d with f_d != 0.  U at offset o: the stage input.
__device__ __forceinline__ double add_source(const DClosures& c, const double* U, long long o, long long ns, int n,
                                             double ds) {
  if (n == UET) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (c.force[d] != 0.0) ds = ds + U[o + (UMX + d) * ns] * c.force[d];
  } else if (n != URHO) {
    const double f = c.force[n - UMX];
    if (f != 0.0) ds = ds + U[o + URHO * ns] * f;
  }
  return ds;
}

// visc_const_t::visc / visc_suth_t::visc (src/cls/Closures.h:103-120)
__device__ __forceinline__ double visc(const DClosures& c, double T) {
  if (c.visc_law == 0) return c.visc_ref;
  return ddiv_rn(c.visc_ref * T * dsqrt_rn(T), c.Tvisc_ref + T);
}
// cond_const_t::cond / cond_suth_t::cond (src/cls/Closures.h:130-166)
__device__ __forceinline__ double cond(const DClosures& c, double T) {
  if (c.cond_law == 0) return c.cond_ref;
  return ddiv_rn(c.cond_ref * T * dsqrt_rn(T), c.Tcond_ref + T);
}

// std::max / std::min semantics
__device__ __forceinline__ double rmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double rmin(double a, double b) { return (b < a) ? b : a; }

// A product on the FP64 pipe (a * b) or, with I, the same correctly rounded
// product formed on the integer pipe (dmul_rn).  The kernels of this path
// are bound by the FP64 pipe while their integer pipe idles; the masks below
// (one per routine, chosen by measurement) move part of their products
// across without changing a bit of any result.
template <bool I>
__device__ __forceinline__ double kmul(double a, double b) {
  return I ? dmul_rn(a, b) : a * b;
}

// cons2prim products on the integer pipe: bit 0 the velocities, 1 their
// squares, 2 the kinetic-energy scalings, 3 pressure, rho R and e (a KEEP4 step at
// 128^3: 2996 us without, 2968 with bit 1, 2950 with 1 and 2, 2975 with all four).
#ifndef AMRS_C2P_IMUL
#define AMRS_C2P_IMUL 0x06
#endif
// Viscous cell-flux products on the integer pipe (see viscous_cell_dy).
#ifndef AMRS_VISC_IMUL
#define AMRS_VISC_IMUL 0x3F
#endif

// cons2prim (src/rhs/CNS_hydro_K.h:15-34) plus QE = cv*T.
__device__ __forceinline__ void cons2prim(const double u[5], double q[NQ], const DClosures& c) {
  // max(1e-40, rho) by the bits: larger, and not a NaN
  const long long rb = __double_as_longlong(u[URHO]);
  const double rho = rb > 0x37A16C262777579Cll && rb <= 0x7FF0000000000000ll ? u[URHO] : 1e-40;
  constexpr int M = AMRS_C2P_IMUL;
  double rhoinv = ddiv_rn(1.0, rho);
  double ux = kmul<M & 1>(u[UMX], rhoinv);
  double uy = kmul<M & 1>(u[UMY], rhoinv);
  double uz = kmul<M & 1>(u[UMZ], rhoinv);
  double rhoke = kmul<(M >> 2) & 1>(kmul<(M >> 2) & 1>(0.5, rho),
                                    kmul<(M >> 1) & 1>(ux, ux) + kmul<(M >> 1) & 1>(uy, uy) +
                                        kmul<(M >> 1) & 1>(uz, uz));
  double rhoei = (u[UET] - rhoke);
  double p = kmul<(M >> 3) & 1>(c.gamma - 1.0, rhoei);
  q[QRHO] = rho;
  q[QU] = ux;
  q[QV] = uy;
  q[QW] = uz;
  q[QPRES] = p;
  q[QT] = ddiv_rn(p, kmul<(M >> 3) & 1>(rho, c.Rspec));
  q[QE] = kmul<(M >> 3) & 1>(c.cv, q[QT]);
}

// Ranges in which keep_pair<D, true> holds, tested once per cell where the
// primitives are formed: density, pressure and energy in [2^-100, 2^100),
// velocities zero or in [2^-200, 2^100).  Every product of a pair then stays well
// inside the normal range (the smallest, P times the velocity products' sum,
// above 2^-810).
__device__ __forceinline__ bool keep_range(const double q[NQ]) {
  bool ok = true;
#pragma unroll
  for (int n = 0; n < NQ; ++n) {
    const DWords w = dwords(q[n]);
    if (n == QU || n == QV || n == QW)
      ok = ok && (w.hi * 2u - (823u << 21) < (300u << 21) || ((w.hi & 0x7FFFFFFFu) | w.lo) == 0u);
    else if (n != QT)
      ok = ok && w.hi - (923u << 20) < (200u << 20);
  }
  return ok;
}

__device__ __forceinline__ bool is_zero(double x) {
  const DWords w = dwords(x);
  return ((w.hi & 0x7FFFFFFFu) | w.lo) == 0u;
}
// 0.5 x for a zero or normal x well above the smallest
__device__ __forceinline__ double half_of(double x) {
  const DWords w = dwords(x);
  return dfrom(((w.hi & 0x7FFFFFFFu) | w.lo) == 0u ? w.hi : w.hi - (1u << 20), w.lo);
}

// a * b on the integer pipe without range tests, +-0 where `zero`.
__device__ __forceinline__ double mul_core(double a, double b) { return dfrom(dmul_core(dwords(a), dwords(b))); }
__device__ __forceinline__ double mul_zero(double a, double b, bool zero) {
  const DWords x = dwords(a), y = dwords(b);
  const DWords r = dmul_core(x, y);
  return dfrom(zero ? (x.hi ^ y.hi) & 0x80000000u : r.hi, zero ? 0u : r.lo);
}

// The same with the sign bit of `sg` for a zero (the words of a product with a
// zero factor are not a zero's, so nothing can be read from them).
__device__ __forceinline__ double mul_zero(double a, double b, bool zero, uint32_t sg) {
  const DWords r = dmul_core(dwords(a), dwords(b));
  return dfrom(zero ? sg & 0x80000000u : r.hi, zero ? 0u : r.lo);
}

// One KEEP pair term (src/rhs/CentralKEEP.h:19-36 helpers, :76-83 body),
// already multiplied by its coefficient: the contribution of pair
// (point 1 = larger index, point 2 = smaller index) to the face flux in
// direction d.  q1/q2 give rho,u,v,w,T,p,e.  FAST: both points are in the ranges
// of keep_range, and the sixteen products run on the integer pipe (the same
// correctly rounded products); otherwise every operation on the FP64 pipe.
template <int D, bool FAST = false>
__device__ __forceinline__ void keep_pair(const double* q1, const double* q2, double coef, double T[5]) {
  constexpr int QN = QU + D;
  const double rhoS = q1[QRHO] + q2[QRHO];
  const double unS = q1[QN] + q2[QN];
  // Binary scalings commute with rounding (normal range), so every power of
  // two in the reference's expressions moves into the pair's constant
  // coefficient, to the bit:
  //   fghCubic: 0.125*rhoS*unS*h == 0.125*(P*h), P = rhoS*unS;
  //   fgQuad massflx 0.25*rhoS*unS == 0.25*P, and massflx*ke with
  //   ke = 0.5*(u1u2+v1v2+w1w2) == 0.125*(P*s3);
  //   fDiv 0.5*(p1+p2) and fgDiv 0.5*(p1*un2+p2*un1) added to an eighth:
  //   x/8 + s/2 == (x + 4s)/8 == fma(4, s, x)/8.
  // So coef*(...) == (coef/8)*(...) with the eighths taken out, and no
  // FP64 instruction is spent on a power-of-two scaling.
  const double c8 = 0.125 * coef, c4 = 0.25 * coef;
  const double psum = q1[QPRES] + q2[QPRES], eS = q1[QE] + q2[QE];
  if (FAST) {
    // P is zero exactly when unS is, and with it every term but the pressure's;
    // D's own momentum term P unS + 4 psum is positive
    const bool zP = is_zero(unS);
    const double P = mul_core(rhoS, unS);  // not read where zP; its sign is that of unS
    const uint32_t gP = dwords(unS).hi, gT = gP ^ dwords(c8).hi;
    double vS[3], s[3];
    bool z[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double a = q1[QU + c], b = q2[QU + c];
      s[c] = mul_zero(a, b, is_zero(a) || is_zero(b));
      vS[c] = a + b;
      z[c] = zP || is_zero(vS[c]);
    }
    const double s3 = s[0] + s[1] + s[2];
    T[URHO] = mul_zero(c4, P, zP, gT);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (c == D) T[UMX + c] = mul_core(c8, fma(4.0, psum, mul_zero(P, vS[c], zP, 0u)));
      else T[UMX + c] = mul_zero(c8, mul_core(P, vS[c]), z[c], gT ^ dwords(vS[c]).hi);
    }
    const double pu = mul_zero(q1[QPRES], q2[QN], is_zero(q2[QN])) + mul_zero(q2[QPRES], q1[QN], is_zero(q1[QN]));
    const double en =
        fma(4.0, pu, mul_zero(P, s3, zP || is_zero(s3), gP ^ dwords(s3).hi) + mul_zero(P, eS, zP, gP));
    T[UET] = mul_zero(c8, en, is_zero(en));
  } else {
    const double P = rhoS * unS;
    const double s3 = q1[QU] * q2[QU] + q1[QV] * q2[QV] + q1[QW] * q2[QW];
    const double cx = P * (q1[QU] + q2[QU]);
    const double cy = P * (q1[QV] + q2[QV]);
    const double cz = P * (q1[QW] + q2[QW]);
    const double ce = P * eS;
    const double pu = q1[QPRES] * q2[QN] + q2[QPRES] * q1[QN];
    T[URHO] = c4 * P;
    T[UMX] = c8 * (D == 0 ? fma(4.0, psum, cx) : cx);
    T[UMY] = c8 * (D == 1 ? fma(4.0, psum, cy) : cy);
    T[UMZ] = c8 * (D == 2 ? fma(4.0, psum, cz) : cz);
    T[UET] = c8 * fma(4.0, pu, P * s3 + ce);
  }
}

// Cell-centred viscous fluxes (src/rhs/CNS_hydro_K.h:108-172) from the
// primitive values at the cell and its six neighbours.  Output: x, y, z
// blocks of (UMX..UET); the mass entries are zero in the reference.
// `qc` centre, `qxm/qxp`, `qym/qyp`, `qzm/qzp` neighbours (u,v,w,T read).
// The same with the four y derivatives (u, v, w, T) given: the body shared
// by the interior form and the wall rows' one-sided form.
__device__ __forceinline__ void viscous_cell_dy(const double* qc, const double* qxm, const double* qxp,
                                                const double dy[4], const double* qzm, const double* qzp,
                                                const double dxinv[3], const DClosures& c, double f[NVF]) {
  // (a-b)*0.5*dxinv == (a-b)*(0.5*dxinv) exactly: the 0.5 scalings are exact.
  // Products on the integer pipe (AMRS_VISC_IMUL): bit 0 the x derivative
  // scalings, 1 the y ones (formed by viscous_cell), 2 the z ones, 3 the
  // r1_3*div terms, 4 the stress scalings by mu, 5 the energy-flux products.
  constexpr int M = AMRS_VISC_IMUL;
  const double hx = 0.5 * dxinv[0], hz = 0.5 * dxinv[2];
  const double ux = qc[QU];
  const double dudx = kmul<M & 1>(qxp[QU] - qxm[QU], hx);
  const double dvdx = kmul<M & 1>(qxp[QV] - qxm[QV], hx);
  const double dwdx = kmul<M & 1>(qxp[QW] - qxm[QW], hx);
  const double dTdx = kmul<M & 1>(qxp[QT] - qxm[QT], hx);
  const double uy = qc[QV];
  const double dudy = dy[0], dvdy = dy[1], dwdy = dy[2], dTdy = dy[3];
  const double uz = qc[QW];
  const double dudz = kmul<(M >> 2) & 1>(qzp[QU] - qzm[QU], hz);
  const double dvdz = kmul<(M >> 2) & 1>(qzp[QV] - qzm[QV], hz);
  const double dwdz = kmul<(M >> 2) & 1>(qzp[QW] - qzm[QW], hz);
  const double dTdz = kmul<(M >> 2) & 1>(qzp[QT] - qzm[QT], hz);
  const double div = dudx + dvdy + dwdz;
  const double mu = visc(c, qc[QT]);
  const double lambda = cond(c, qc[QT]);
  const double r1_3 = 1.0 / 3.0;
  // The fluxes are stored negated (-tau, -lambda dT - tau.u).  Negation is
  // exact, so (-2mu)*d == -(2mu*d) and a + (-t)*u == a - t*u to the bit:
  // the negated stresses n.. are formed directly and the sums add them,
  // with no separate negations.
  constexpr bool MD = (M >> 3) & 1, MS = (M >> 4) & 1, ME = (M >> 5) & 1;
  const double nmu = -mu, nmu2 = -2.0 * mu, nlam = -lambda;
  const double nxx = kmul<MS>(nmu2, dudx - kmul<MD>(r1_3, div));
  const double nxy = kmul<MS>(nmu, dudy + dvdx);
  const double nxz = kmul<MS>(nmu, dudz + dwdx);
  const double nyy = kmul<MS>(nmu2, dvdy - kmul<MD>(r1_3, div));
  const double nyz = kmul<MS>(nmu, dvdz + dwdy);
  const double nzz = kmul<MS>(nmu2, dwdz - kmul<MD>(r1_3, div));
  f[0] = nxx;
  f[1] = nxy;
  f[2] = nxz;
  f[3] = kmul<ME>(nlam, dTdx) + kmul<ME>(nxx, ux) + kmul<ME>(nxy, uy) + kmul<ME>(nxz, uz);
  f[4] = nxy;
  f[5] = nyy;
  f[6] = nyz;
  f[7] = kmul<ME>(nlam, dTdy) + kmul<ME>(nxy, ux) + kmul<ME>(nyy, uy) + kmul<ME>(nyz, uz);
  f[8] = nxz;
  f[9] = nyz;
  f[10] = nzz;
  f[11] = kmul<ME>(nlam, dTdz) + kmul<ME>(nxz, ux) + kmul<ME>(nyz, uy) + kmul<ME>(nzz, uz);
}

__device__ __forceinline__ void viscous_cell(const double* qc, const double* qxm, const double* qxp,
                                             const double* qym, const double* qyp, const double* qzm,
                                             const double* qzp, const double dxinv[3], const DClosures& c,
                                             double f[NVF]) {
  constexpr bool MY = (AMRS_VISC_IMUL >> 1) & 1;
  const double hy = 0.5 * dxinv[1];
  const double dy[4] = {kmul<MY>(qyp[QU] - qym[QU], hy), kmul<MY>(qyp[QV] - qym[QV], hy),
                        kmul<MY>(qyp[QW] - qym[QW], hy), kmul<MY>(qyp[QT] - qym[QT], hy)};
  viscous_cell_dy(qc, qxm, qxp, dy, qzm, qzp, dxinv, c, f);
}

// ViscousWallFluxes (src/rhs/CNS_hydro_K.h:177-251): the cell viscous fluxes
// of the ghost row next to a y wall with second-order one-sided y
// derivatives; loc 0 (lower wall) reads rows j, j+1, j+2 as (q0, q1, q2),
// loc 1 (upper wall) rows j, j-1, j-2.  -a + 4b and 3c - 4b are single fmas
// (the factor 4 is exact).
__device__ __forceinline__ void viscous_wall_cell(int loc, const double* qc, const double* qxm, const double* qxp,
                                                  const double* q1, const double* q2, const double* qzm,
                                                  const double* qzp, const double dxinv[3], const DClosures& c,
                                                  double f[NVF]) {
  const double hy = 0.5 * dxinv[1];
  double dy[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int m = QU + n;
    dy[n] = (loc == 0) ? (fma(4.0, q1[m], -q2[m]) - 3.0 * qc[m]) * hy
                       : (fma(-4.0, q1[m], 3.0 * qc[m]) + q2[m]) * hy;
  }
  viscous_cell_dy(qc, qxm, qxp, dy, qzm, qzp, dxinv, c, f);
}

// RK stage program (AMReX BLAS-1 semantics), registers S1, S2, dS.
// fa/fb: 0 the coefficient is a / b; 1 it is dt * a / dt * b; 2 it is
// dt / a / dt / b, with dt read from device memory (dtp) when the kernel
// starts: the device-resident time loop changes dt without new launches.
struct DOp {
  int kind, dst, x, y;
  double a, b;
  int fa, fb;
};
struct DProg {
  int nops;
  DOp ops[3];
  const double* dtp;
};

__device__ __forceinline__ double dt_coef(int form, double c, double dt) {
  return form == 1 ? dt * c : (form == 2 ? dt / c : c);
}
// The program with its dt-dependent coefficients evaluated (dt * c and
// dt / c round exactly as the host's CNS::advance arithmetic).
__device__ __forceinline__ DProg resolve_prog(DProg p) {
  if (p.dtp) {
    const double dt = *p.dtp;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      p.ops[o].a = dt_coef(p.ops[o].fa, p.ops[o].a, dt);
      p.ops[o].b = dt_coef(p.ops[o].fb, p.ops[o].b, dt);
    }
  }
  return p;
}

// Its products on the integer pipe (dmul_rn), or no product where the factor is
// one.  The registers are picked by selects (an indexed array would live in
// local memory).
__device__ __forceinline__ double prog_mul(double a, double x) {
  return __double_as_longlong(a) == 0x3FF0000000000000ll ? x : dmul_rn(a, x);
}
__device__ __forceinline__ double prog_pick(int r, double s1, double s2, double ds) {
  return r == 0 ? s1 : (r == 1 ? s2 : ds);
}
// the program on registers S1, S2 and dS; the stage result is S2
__device__ __forceinline__ double apply_prog(const DProg& p, double s1, double s2, double ds) {
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    if (o >= p.nops) break;
    const DOp& q = p.ops[o];
    const double x = prog_pick(q.x, s1, s2, ds);
    double r = x;
    if (q.kind == 0) r = prog_mul(q.a, x) + prog_mul(q.b, prog_pick(q.y, s1, s2, ds));
    else if (q.kind == 1) r = prog_pick(q.dst, s1, s2, ds) + prog_mul(q.a, x);
    else if (q.kind == 2) r = x + prog_mul(q.a, prog_pick(q.dst, s1, s2, ds));
    if (q.dst == 0) s1 = r;
    else if (q.dst == 1) s2 = r;
    else ds = r;
  }
  return s2;
}

}  // namespace amrs

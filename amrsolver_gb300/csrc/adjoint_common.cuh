// Pieces shared by the reverse-mode kernels.
#pragma once
#include "amrs_boxes.cuh"
#include "weno_int.cuh"

namespace amrs {

constexpr int NQA = 6;  // primitive cotangents: rho, u, v, w, T, p (e = cv*T folded into T)

// Reverse of cons2prim (src/rhs/CNS_hydro_K.h:15-34) at cell (i,j,k) of box R:
// given the primitive cotangents qb (NQA order), the cotangents of the
// conserved state U = R.slot[0] there.  max(1e-40, rho) passes the density
// cotangent only where rho > 1e-40 (the forward's branch).
__device__ __forceinline__ void cons2prim_vjp(const BoxRec& R, const DClosures& cl, int i, int j, int k,
                                              const double qb[NQA], double ub5[5]) {
  const DArr Q = R.q;
  const long long oq = Q.off(i, j, k);
  const double rho = Q.p[oq + QRHO * Q.ns], u = Q.p[oq + QU * Q.ns], v = Q.p[oq + QV * Q.ns],
               w = Q.p[oq + QW * Q.ns], T = Q.p[oq + QT * Q.ns];
  const double rinv = ddiv_rn(1.0, rho);
  const double eib = (cl.gamma - 1.0) * (qb[QPRES] + ddiv_rn(qb[QT], rho * cl.Rspec));  // d/d rhoei
  // d/d rhoke = -eib
  const double reib = dmul_rn(rho, -eib);
  const double ub = qb[QU] + reib * u, vb = qb[QV] + reib * v, wb = qb[QW] + reib * w;
  const double rb = qb[QRHO] - 0.5 * (u * u + v * v + w * w) * eib -
                    (qb[QT] * T + (ub * u + vb * v + wb * w)) * rinv;
  const DArr U = R.slot[0];
  const double rho_raw = U(i, j, k, URHO);
  ub5[0] = (rho_raw > 1e-40) ? rb : 0.0;
  ub5[1] = dmul_rn(ub, rinv);
  ub5[2] = dmul_rn(vb, rinv);
  ub5[3] = dmul_rn(wb, rinv);
  ub5[4] = eib;
}

// Gradient and value of weno5js (src/rhs/High_resolution.h:124-159):
//   W = sum_k w_k v_k / 6,  w_k = a_k / A,  a_k = c_k / e_k^2,  e_k = beta_k + eps
//   dW/ds = sum_k (w_k/6) grad v_k + sum_k ebar_k grad beta_k,
//   ebar_k = -2 w_k (v_k/6 - W) / e_k.
// With q_k the product of the other two e's, P = e0 e1 e2 and
// D = sum_k c_k q_k^2: w_k = c_k q_k^2 / D and w_k / e_k = c_k q_k^3 / (D P),
// so one division 1/(D P) serves the weights and the e_k quotients (D P ~ e^7
// stays in range for e in [1e-40, 1e40]; outside it the four-division form).
//
// Everything is a function of the differences t_q = s_{q+1} - s_q: the smoothness
// differences, and y_k = v_k/6 - s2 (y0 = d1/12 + d2/4, y1 = d3/12 - g/4,
// y2 = d4/12 - d5/4), with W = s2 + sum_k w_k y_k because the weights sum to one.
// The entries of the gradient then sum to one as well, which gives the middle
// one.  (The reverse pass has no bit-exact counterpart.)
struct WenoDiffs {
  double d1, d2, d3, g, d4, d5;
  __device__ __forceinline__ explicit WenoDiffs(const double t[4])
      : d1(t[1] - t[0]), d2(2.0 * t[1] + d1), d3(t[2] - t[1]), g(-t[1] - t[2]), d4(t[3] - t[2]),
        d5(-2.0 * t[2] + d4) {}
};
__device__ __forceinline__ void weno_grad_sums(double x0, double x1, double x2, double p1, double p2, double p3,
                                               double p4, double p5, double p6, double gr[5]) {
  gr[0] = (1.0 / 3.0) * x0 + (p1 + p2);
  gr[1] = (-7.0 / 6.0) * x0 + ((-1.0 / 6.0) * x1 + (-2.0 * p1 + (-4.0 * p2 + (p3 + p4))));
  gr[3] = (1.0 / 3.0) * x1 + ((5.0 / 6.0) * x2 + (-2.0 * p5 + (-4.0 * p6 + (p3 - p4))));
  gr[4] = (-1.0 / 6.0) * x2 + (p5 + p6);
  gr[2] = ((1.0 - gr[0]) - gr[4]) - (gr[1] + gr[3]);
}

// With the hardware's operations, out of line; Wy = W - s2.
static __device__ __noinline__ void weno5js_grad_plain(const double* t, double* gr, double* Wy) {
  constexpr double eps = 1e-40;
  const WenoDiffs d(t);
  const double g2 = d.g * d.g;
  const double e0 = eps + ((13.0 / 12.0) * d.d1 * d.d1 + 0.25 * d.d2 * d.d2);
  const double e1 = eps + ((13.0 / 12.0) * d.d3 * d.d3 + 0.25 * g2 * g2);
  const double e2 = eps + ((13.0 / 12.0) * d.d4 * d.d4 + 0.25 * d.d5 * d.d5);
  const double q0 = e1 * e2, q1 = e0 * e2, q2 = e0 * e1;
  const double t0 = 0.1 * q0 * q0, t1 = 0.6 * q1 * q1, t2 = 0.3 * q2 * q2;
  const double P = e0 * q0, DP = (t0 + t1 + t2) * P;
  double w0, w1, w2, we0, we1, we2;  // w_k and w_k / e_k
  if (DP > 1e-300 && DP < 1e300) {
    const double r = 1.0 / DP, rP = r * P;
    w0 = t0 * rP; w1 = t1 * rP; w2 = t2 * rP;
    we0 = t0 * q0 * r; we1 = t1 * q1 * r; we2 = t2 * q2 * r;
  } else {
    const double i0 = 1.0 / e0, i1 = 1.0 / e1, i2 = 1.0 / e2;
    const double a0 = 0.1 * i0 * i0, a1 = 0.6 * i1 * i1, a2 = 0.3 * i2 * i2;
    const double iA = 1.0 / (a0 + a1 + a2);
    w0 = a0 * iA; w1 = a1 * iA; w2 = a2 * iA;
    we0 = w0 * i0; we1 = w1 * i1; we2 = w2 * i2;
  }
  const double y0 = d.d1 * (1.0 / 12.0) + 0.25 * d.d2, y1 = d.d3 * (1.0 / 12.0) - 0.25 * d.g,
               y2 = d.d4 * (1.0 / 12.0) - 0.25 * d.d5;
  const double W = w0 * y0 + w1 * y1 + w2 * y2;
  *Wy = W;
  const double b0 = -2.0 * (y0 - W) * we0, b1 = -2.0 * (y1 - W) * we1, b2 = -2.0 * (y2 - W) * we2;
  weno_grad_sums(w0, w1, w2, b0 * (13.0 / 6.0) * d.d1, b0 * 0.5 * d.d2, b1 * (13.0 / 6.0) * d.d3, b1 * g2 * d.g,
                 b2 * (13.0 / 6.0) * d.d4, b2 * 0.5 * d.d5, gr);
}

// The same with its products and the division on the integer pipe (38 FP64
// instructions are left of about 110): behind one range test per smoothness
// difference and per y_k - Wy no product tests its own.  Differences are below 2^60,
// s1 - s3 below 2^35 (its fourth power enters e), so e lies in [2^-133, 2^143) and D P
// in the normal range.  A zero y_k - Wy gives zero terms, and so does a difference
// below 2^-240: its terms are below 2^-170, beside entries that sum to one (ebar_k is
// at most 2^134 |y_k - Wy|, and that at most 2^-66 where e_k is about eps).  The y_k
// are twelvefold, Y0 = d1 + 3 d2 and so on, and 1/12 goes with 1/(D P).  t: the four
// differences; Wy = W - s2.
__device__ __forceinline__ void weno5js_grad(const double t[4], double gr[5], double& Wy) {
  bool ok = true, slow;
  const WenoDiffs d(t);
  const DWords D1 = weno_diff(d.d1, ok), D2 = weno_diff(d.d2, ok), D3 = weno_diff(d.d3, ok), G = weno_diff(d.g, ok),
               D4 = weno_diff(d.d4, ok), D5 = weno_diff(d.d5, ok);
  ok = ok && (G.hi & 0x7FFFFFFFu) < (1058u << 20);
  const bool z1 = weno_tiny(d.d1), z2 = weno_tiny(d.d2), z3 = weno_tiny(d.d3), zg = weno_tiny(d.g), z4 = weno_tiny(d.d4),
             z5 = weno_tiny(d.d5);
  auto term = [](DWords a, DWords b, bool zero) {
    const DWords x = dmul_core(a, b);
    return zero ? 0.0 : dfrom(x);
  };
  const DWords c1312{0x3FF15555u, 0x55555555u}, c112{0x3FB55555u, 0x55555555u};  // 13/12, 1/12
  const DWords g2 = dmul_core(G, G);
  const DWords e0 = weno_e(fma(0.25, dfrom(dmul_core(D2, D2)), dfrom(dmul_core(dmul_core(c1312, D1), D1))));
  const DWords e1 = weno_e(fma(0.25, dfrom(dmul_core(g2, g2)), dfrom(dmul_core(dmul_core(c1312, D3), D3))));
  const DWords e2 = weno_e(fma(0.25, dfrom(dmul_core(D5, D5)), dfrom(dmul_core(dmul_core(c1312, D4), D4))));
  const DWords q0 = dmul_core(e1, e2), q1 = dmul_core(e0, e2), q2 = dmul_core(e0, e1);
  const DWords t0 = dmul_core(dmul_core(DWords{0x3FB99999u, 0x9999999Au}, q0), q0);
  const DWords t1 = dmul_core(dmul_core(DWords{0x3FE33333u, 0x33333333u}, q1), q1);
  const DWords t2 = dmul_core(dmul_core(DWords{0x3FD33333u, 0x33333333u}, q2), q2);
  const DWords P = dmul_core(e0, q0);
  const DWords r = ddiv_core(DWords{0x3FF00000u, 0u}, dmul_core(dwords(dfrom(t0) + dfrom(t1) + dfrom(t2)), P), &slow);
  ok = ok && !slow;
  const DWords rP = dmul_core(r, P), r12 = dmul_core(r, c112);
  const double x0 = dfrom(dmul_core(t0, rP)), x1 = dfrom(dmul_core(t1, rP)), x2 = dfrom(dmul_core(t2, rP));
  const double y0 = fma(3.0, d.d2, d.d1), y1 = fma(-3.0, d.g, d.d3), y2 = fma(-3.0, d.d5, d.d4);
  const double S = x0 * y0 + x1 * y1 + x2 * y2;
  Wy = S * (1.0 / 12.0);
  // b_k = w_k / e_k (y_k - Wy) = -ebar_k / 2; the terms ebar_k grad beta_k:
  // p1 = -(13/3) b0 d1, p2 = -b0 d2, p4 = -2 b1 g^3, ...
  const ZWords f0 = weno_fac(y0 - S, ok), f1 = weno_fac(y1 - S, ok), f2 = weno_fac(y2 - S, ok);
  auto negated = [](DWords a) { return DWords{a.hi ^ 0x80000000u, a.lo}; };
  const DWords b0 = negated(dmul_core(dmul_core(t0, dmul_core(q0, r12)), f0.w));
  const DWords b1 = negated(dmul_core(dmul_core(t1, dmul_core(q1, r12)), f1.w));
  const DWords b2 = negated(dmul_core(dmul_core(t2, dmul_core(q2, r12)), f2.w));
  const DWords c133{0x40115555u, 0x55555555u};  // 13/3
  const DWords gb{b1.hi + (1u << 20), b1.lo};   // 2 b1
  weno_grad_sums(x0, x1, x2, term(dmul_core(c133, b0), D1, f0.zero || z1), term(b0, D2, f0.zero || z2),
                 term(dmul_core(c133, b1), D3, f1.zero || z3), term(dmul_core(gb, g2), G, f1.zero || zg),
                 term(dmul_core(c133, b2), D4, f2.zero || z4), term(b2, D5, f2.zero || z5), gr);
  if (!ok) {
    double a[4], o[5], w;
#pragma unroll
    for (int n = 0; n < 4; ++n) a[n] = t[n];
    weno5js_grad_plain(a, o, &w);
#pragma unroll
    for (int n = 0; n < 5; ++n) gr[n] = o[n];
    Wy = w;
  }
}

}  // namespace amrs

// Pieces of WENO5-JS on the integer pipe, shared by the forward reconstruction
// (weno5js_int) and its gradient (weno5js_grad): values enter through one range
// test each (`ok`), and every product and quotient behind them goes without.
#pragma once
#include "amrs_device.cuh"

namespace amrs {

// A smoothness difference below 2^60, for its square or fourth power.  One below
// 2^-240, zero or subnormal too, enters as 2^-200: either way its part of beta is below
// 2^-399, so less than half a last place of the other part from 2^-346 up, and with
// that below 2^-346 beta is less than half a last place of eps; no bit of eps + beta
// depends on it.  (Fluid at rest beside moving fluid has differences of momentum of
// any small size.  With a lower bound of 2^-100 and the plain form below it such a step
// at 64^3 took 3.17 ms, 2.76 now, and noise of 1e-35 around rest 2.73, 1.70 now.  Of nine
// ways to write the two tests this one is as fast as that bound, the others 1-2% slower.)
__device__ __forceinline__ bool weno_tiny(double x) { return (dwords(x).hi & 0x7FFFFFFFu) < (783u << 20); }
__device__ __forceinline__ DWords weno_diff(double x, bool& ok) {
  DWords w = dwords(x);
  const bool tiny = weno_tiny(x);
  ok = ok && (tiny || w.hi * 2u - (783u << 21) < (300u << 21));
  w.hi = tiny ? (823u << 20) : w.hi;
  return w;
}
static __device__ __noinline__ double dadd_hw(double a, double b) { return a + b; }
// eps + beta: beta from 2^-78 up (eps is below half its last place), eps below
// 2^-187 (the other way round); in between the hardware adds them, out of line.
__device__ __forceinline__ DWords weno_e(double beta) {
  DWords w = dwords(beta);
  const bool big = w.hi >= (945u << 20), tiny = w.hi < (836u << 20);
  if (!big) {
    w = DWords{0x37A16C26u, 0x2777579Cu};  // 1e-40
    if (!tiny) w = dwords(dadd_hw(1e-40, beta));
  }
  return w;
}
// A factor that may be zero: its words, and whether it is.
struct ZWords {
  DWords w;
  bool zero;
};
__device__ __forceinline__ ZWords weno_fac(double x, bool& ok) {
  ZWords z;
  z.w = dwords(x);
  z.zero = ((z.w.hi & 0x7FFFFFFFu) | z.w.lo) == 0u;
  ok = ok && (z.zero || mid_range(z.w.hi));
  return z;
}
// a * x for a nonzero a of the middle range.
__device__ __forceinline__ double weno_mul(DWords a, const ZWords& x) {
  const DWords r = dmul_core(a, x.w);
  return dfrom(x.zero ? ((a.hi ^ x.w.hi) & 0x80000000u) : r.hi, x.zero ? 0u : r.lo);
}

}  // namespace amrs

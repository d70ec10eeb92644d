// Correctly rounded FP64 division a / b, multiplication a * b and square
// root sqrt(x) (IEEE round to nearest, ties to even) computed on the integer
// pipe.
//
// Why: on this GPU the FP64 pipe issues 2 lanes per clock per SM and every
// kernel of the path is bound by it; a hardware-style FP64 division
// (reciprocal seed plus Newton steps in DFMA) costs several FP64 issue slots.
// The same correctly rounded results can be formed from the operands' bits
// with 32-bit integer instructions, which run on units with far more lanes
// and overlap with the FP64 work of other warps.  The results are the same
// numbers (IEEE division, square root and multiplication are correctly
// rounded, so any correct method gives the same bits): kernels that must
// match the reference bit for bit may use them.
//
// All three work on 32-bit words and multiply with 32 x 32 -> 64 bit
// multiply-adds, and every exponent and sign is formed by adding the words'
// upper 12 bits (the significand's carry then moves into the exponent by
// itself).
//
// Product: the exact 106-bit product from four multiply-adds, the 53-bit
// significand, rounding word and sticky bit by funnel shifts.
//
// Division and square root (long division in digits of 28-29 bits with a
// 32-bit reciprocal estimate, Knuth, The Art of Computer Programming vol. 2,
// 4.3.1, and the rounding test of Ziv, ACM TOMS 17(3), 1991): an FP32
// reciprocal (reciprocal square root) seed of 22 bits and one Newton step in
// 32-bit integers give v with a relative error below 2^-29, rounded down;
// the first digit is a high product with v, the exact remainder follows in
// 64-bit arithmetic, the second digit and remainder likewise, and a third
// high product extends the quotient (root) to more than 80 bits.  Neither
// operation has results half way between two doubles, so the truncated
// 84-bit value decides the rounding unless it lies within a few units of
// 2^-84 of a midpoint; there the sign of the exact remainder at the midpoint
// does, again in 64-bit arithmetic.  That is one random operand pair in 2^28,
// but every 1/x for x an odd number of units in the last place below a power of
// two, and every root of an odd number of units above one: a uniform state with
// rho = 1 and gamma p = 1 up to rounding is full of them.
//
// Domain: operands with exponents in the middle half of the range (about
// 2^-503 .. 2^504), for the product +-0 too; anything else (subnormal,
// infinite, NaN, results that could overflow or underflow) takes the
// hardware operation, so each function equals its operator for every input.
//
// Bound: the integer pipes' issue rate.  Cycles per warp operation and SM with
// 16 warps resident and nothing else running (GB300), against the earlier
// form (64-bit fixed-point Newton iterations and a 128-bit product) and the
// hardware operation: product 14 (28, 19), division 27 (76, 137), square root
// 29 (77, 143); without the range checks (the *_core functions) 10, 20 and 25, a
// division that leaves undecided roundings to its caller 17.
// Beside a saturated FP64 stream of 16 FMAs, four products cost 4% (hardware
// products 30%) and four divisions 6% (earlier form 41%).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define AMRS_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#include <string.h>
#define AMRS_HD inline
#endif

namespace amrs {

struct DWords {
  uint32_t hi, lo;
};

// The words of x.  On the device an opaque move: the compiler would otherwise
// turn integer tests on a reinterpreted double (an exponent field equal to
// 0x7FF, (bits << 1) == 0) back into FP64 compares, each of which takes an
// FP64 issue slot -- the very resource these functions exist to spare.
AMRS_HD DWords dwords(double x) {
  DWords w;
#ifdef __CUDA_ARCH__
  asm("mov.b64 {%0, %1}, %2;" : "=r"(w.lo), "=r"(w.hi) : "d"(x));
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  w.hi = (uint32_t)(u >> 32);
  w.lo = (uint32_t)u;
#endif
  return w;
}

AMRS_HD double dfrom(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  double x;
  asm("mov.b64 %0, {%1, %2};" : "=d"(x) : "r"(lo), "r"(hi));
  return x;
#else
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

AMRS_HD double dfrom(DWords w) { return dfrom(w.hi, w.lo); }

AMRS_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
AMRS_HD uint64_t madw(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
// the upper word of (hi:lo) << s and the lower word of (hi:lo) >> s, 0 <= s < 32
AMRS_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)((((uint64_t)hi << 32 | lo) << s) >> 32);
#endif
}
AMRS_HD uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (uint32_t)(((uint64_t)hi << 32 | lo) >> s);
#endif
}
// (hi:lo) plus the carry of r + k, plus E in the upper word
AMRS_HD DWords round_pack(uint32_t r, uint32_t k, uint32_t hi, uint32_t lo, uint32_t E) {
#ifdef __CUDA_ARCH__
  uint32_t l, h;
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
      : "=r"(l), "=r"(h)
      : "r"(r), "r"(k), "r"(lo), "r"(hi), "r"(E));
  return DWords{h, l};
#else
  const uint64_t c = ((uint64_t)r + k) >> 32;
  const uint64_t u = ((((uint64_t)hi << 32) | lo) + c) + ((uint64_t)E << 32);
  return DWords{(uint32_t)(u >> 32), (uint32_t)u};
#endif
}

// The operations for inputs outside the integer paths' domains (dmul_hw here,
// ddiv_rest and dsqrt_rest below) are out of line: a call is a real branch taken
// only by lanes that need it, where an inlined fallback is predicated by the
// compiler and issues its FP64 instruction on every call.
#ifdef __CUDA_ARCH__
#define AMRS_OUT_OF_LINE static __device__ __noinline__
#define AMRS_SQRT(x) sqrt(x)
AMRS_OUT_OF_LINE double dmul_hw(double a, double b) { return __dmul_rn(a, b); }
#else
#define AMRS_OUT_OF_LINE inline
#define AMRS_SQRT(x) ::sqrt(x)
inline double dmul_hw(double a, double b) { return a * b; }
#endif

// Seeds of the Newton steps.  They need about 22 correct bits, not correct
// rounding: on the device the approximate FP32 reciprocal and reciprocal
// square root (rcp.approx / rsqrt.approx, within 1 ulp and 2^-22.9 relative),
// which run on the special-function unit and use no FP64 slot.  The host
// build perturbs the correctly rounded value by up to +-2 ulps, so the host
// checks cover seeds at least that far off.
AMRS_HD uint32_t seed_perturb(uint32_t rb, uint32_t v) {
#ifdef __CUDA_ARCH__
  (void)v;
  return rb;
#else
  return rb + (uint32_t)((int)((v ^ (v >> 7) ^ (v >> 13)) % 5u) - 2);
#endif
}
// a seed in (0.5, 1] (its bits, possibly an ulp or two outside) as a 32-bit
// fraction: 2^32 times the value clamped to [0.5, 1)
AMRS_HD uint32_t seed_fraction(uint32_t rb) {
  rb = rb < 0x3F000000u ? 0x3F000000u : rb;
  rb = rb > 0x3F7FFFFFu ? 0x3F7FFFFFu : rb;
  return rb * 256u + 0x80000000u;
}
// 2^32 / f for the float f in [1, 2) with these bits, to 22 bits
AMRS_HD uint32_t seed_rcp(uint32_t fb) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  return seed_fraction(__float_as_uint(r));
#else
  float f, r;
  memcpy(&f, &fb, 4);
  r = 1.0f / f;
  uint32_t rb;
  memcpy(&rb, &r, 4);
  return seed_fraction(seed_perturb(rb, fb));
#endif
}
// 2^32 / sqrt(f) for the float f in [1, 4) with these bits, to 22 bits
AMRS_HD uint32_t seed_rsqrt(uint32_t fb) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  return seed_fraction(__float_as_uint(r));
#else
  float f;
  memcpy(&f, &fb, 4);
  const float r = (float)(1.0 / sqrt((double)f));
  uint32_t rb;
  memcpy(&rb, &r, 4);
  return seed_fraction(seed_perturb(rb, fb));
#endif
}
// the Newton correction v e / 2^31 for |e| < 2^11
AMRS_HD uint32_t seed_corr(uint32_t v, int32_t e) { return (uint32_t)(((int32_t)(v >> 12) * e) >> 19); }

// exponent of the word in [520, 1528)
AMRS_HD bool mid_range(uint32_t hi) { return hi * 2u - 0x41000000u < 0x7E000000u; }

// a / b for words in the domain.  ma/mb in (1/2, 2), digits q1, q2, q3 of
// ma 2^86 / mb = q1 2^58 + q2 2^29 + q3, each rounded down (v is):
//   q1 <= ma 2^28 / mb,   R1 = ma 2^28 - q1 mb in [0, 2.3 mb)
//   q2 <= R1 2^29 / mb,   R2 = R1 2^29 - q2 mb in [0, 3.8 mb)
//   q3 <= R2 2^29 / mb    within 5 units
// Where that leaves the rounding open, m is the last digit with which the
// quotient would be the midpoint, and R2 2^29 - m mb (below 2^60) has the sign.
struct DDiv {
  uint32_t q3, rl, rh, nl, nh, Tl, Wh, Wl, s, r, E;  // R2 = (rh:rl), -mb = (nh:nl)
  AMRS_HD DDiv(DWords a, DWords b) {
    const uint32_t mah = (a.hi & 0xFFFFFu) | 0x100000u, mbh = (b.hi & 0xFFFFFu) | 0x100000u;
    // v ~ 2^63 / dh, dh = the top 32 bits of mb 2^11; one Newton step
    const uint32_t dh = shl_hi(b.lo, mbh, 11);
    const uint32_t v0 = seed_rcp(((dh >> 8) & 0x7FFFFFu) | 0x3F800000u);
    const int32_t e = (int32_t)(0x7FFFFFFFu - mulhi32(v0, dh));
    const uint32_t v = v0 + seed_corr(v0, e) - 3u;  // < 2^95 / (mb 2^11)
    const uint64_t nmb = 0ull - (((uint64_t)mbh << 32) | b.lo);
    nl = (uint32_t)nmb;
    nh = (uint32_t)(nmb >> 32);
    const uint32_t q1 = mulhi32(shl_hi(a.lo, mah, 11), v) >> 3;
    uint64_t R = madw(q1, nl, ((uint64_t)shl_hi(a.lo, mah, 28) << 32) | (a.lo << 28));
    rl = (uint32_t)R;
    rh = (uint32_t)(R >> 32) + q1 * nh;
    const uint32_t q2 = mulhi32(shr_lo(rl, rh, 23), v);
    R = madw(q2, nl, ((uint64_t)shl_hi(rl, rh, 29) << 32) | (rl << 29));
    rl = (uint32_t)R;
    rh = (uint32_t)(R >> 32) + q2 * nh;
    q3 = mulhi32(shr_lo(rl, rh, 23), v);
    const uint64_t T = madw(q2, 1u << 29, q3);
    const uint64_t W = madw(q1, 1u << 26, T >> 32);  // in (2^53, 2^55)
    Tl = (uint32_t)T;
    Wh = (uint32_t)(W >> 32);
    Wl = (uint32_t)W;
    const uint32_t top = Wh >> 22;
    s = 1u + top;
    r = shr_lo(Tl, Wl, s);
    E = (a.hi & 0xFFF00000u) - (b.hi & 0xFFF00000u) + (1021u << 20) + (top << 20);
  }
  AMRS_HD bool undecided() const { return r - 0x7FFFFFF8u < 8u; }
  AMRS_HD void decide() {
    const uint32_t m = q3 + ((0x80000000u - r) << s) - (Tl & ((1u << s) - 1u));
    const uint64_t D = madw(m, nl, ((uint64_t)shl_hi(rl, rh, 29) << 32) | (rl << 29)) + ((uint64_t)(m * nh) << 32);
    r = (int64_t)D < 0 ? 0x7FFFFFFFu : 0x80000000u;
  }
  AMRS_HD DWords pack() const { return round_pack(r, 0x80000000u, Wh >> s, shr_lo(Wl, Wh, s), E); }
};
AMRS_HD DWords ddiv_core(DWords a, DWords b) {
  DDiv q(a, b);
  if (__builtin_expect(q.undecided(), 0)) q.decide();
  return q.pack();
}
// The same without the decision: *slow is set where it is needed.  For callers
// whose operands reach it by chance only and that have a fallback anyway.
AMRS_HD DWords ddiv_core(DWords a, DWords b, bool* slow) {
  const DDiv q(a, b);
  *slow = q.undecided();
  return q.pack();
}

// What ddiv_rn leaves: an undecided rounding, or an operand outside the domain.
AMRS_OUT_OF_LINE double ddiv_rest(double a, double b) {
  const DWords A = dwords(a), B = dwords(b);
  return mid_range(A.hi) && mid_range(B.hi) ? dfrom(ddiv_core(A, B)) : a / b;
}

// a / b, correctly rounded; the integer path where its domain holds.
AMRS_HD double ddiv_rn(double a, double b) {
  const DWords A = dwords(a), B = dwords(b);
  bool slow;
  double x = dfrom(ddiv_core(A, B, &slow));
  if (!mid_range(A.hi) || !mid_range(B.hi) || slow) {
    // +-0 / b with b in range is +-0
    if (((A.hi << 1) | A.lo) == 0u && mid_range(B.hi)) x = dfrom((A.hi ^ B.hi) & 0x80000000u, 0u);
    else x = ddiv_rest(a, b);
  }
  return x;
}

// K a for K = 3, 5, 7 or 11 and normal a with K a finite, correctly rounded: the
// product has one or two bits more than the floor of log2 K, and rounds at them.
template <uint32_t K>
AMRS_HD DWords dmul_small(DWords a) {
  constexpr uint32_t s0 = K < 4 ? 1 : (K < 8 ? 2 : 3);
  const uint32_t mh = (a.hi & 0xFFFFFu) | 0x100000u;
  uint64_t P = (uint64_t)a.lo * K + ((uint64_t)(mh * K) << 32);
  const uint32_t c = (uint32_t)(P >> (53 + s0)), s = s0 + c;
  P += (c ? (1u << s0) - 1u : (1u << (s0 - 1u)) - 1u) + ((uint32_t)(P >> s) & 1u);
  P >>= s;
  return DWords{(a.hi & 0xFFF00000u) + (uint32_t)(P >> 32) + ((s - 1u) << 20), (uint32_t)P};
}

// x + y of two positive normal numbers whose sum stays finite, correctly rounded:
// significands aligned in 64 bits with ten guard bits and a sticky bit; beyond 62
// places the smaller one is only the sticky bit.
AMRS_HD DWords dadd_pos(DWords x, DWords y) {
  const bool sw = y.hi > x.hi;
  const uint32_t ah = sw ? y.hi : x.hi, al = sw ? y.lo : x.lo, bh = sw ? x.hi : y.hi, bl = sw ? x.lo : y.lo;
  const uint32_t e = ah >> 20;
  uint32_t d = e - (bh >> 20);
  d = d < 62u ? d : 62u;
  const uint64_t A = ((uint64_t)((ah & 0xFFFFFu) | 0x100000u) << 32 | al) << 10;
  const uint64_t B = ((uint64_t)((bh & 0xFFFFFu) | 0x100000u) << 32 | bl) << 10;
  uint64_t S = A + (B >> d);
  S |= ((B << 1) << (63u - d)) != 0u;
  const uint32_t c = (uint32_t)(S >> 63);
  S = (S >> c) | (S & c);
  S = (S + (0x1FFu + ((uint32_t)(S >> 10) & 1u))) >> 10;
  return DWords{(uint32_t)(S >> 32) + ((e - 1u + c) << 20), (uint32_t)S};
}

// a * b for words in the domain (any exponents whose sum gives a normal
// product).  v:t:p is the 106-bit product ma mb, p3 its upper word in
// [2^8, 2^10); the rounding word r holds the bits below the significand with
// the last word's sticky bit or-ed in, and r + 0x7FFFFFFF + lsb carries
// exactly when rounding to nearest even goes up.
AMRS_HD DWords dmul_core(DWords a, DWords b) {
  const uint32_t mah = (a.hi & 0xFFFFFu) | 0x100000u, mbh = (b.hi & 0xFFFFFu) | 0x100000u;
  const uint64_t p = madw(a.lo, b.lo, 0ull);
  const uint64_t t = madw(mah, b.lo, madw(a.lo, mbh, p >> 32));
  const uint64_t v = madw(mah, mbh, t >> 32);
  const uint32_t p3 = (uint32_t)(v >> 32), p2 = (uint32_t)v, p1 = (uint32_t)t, p0 = (uint32_t)p;
  const uint32_t top = p3 >> 9, s = 12u - top;
  const uint32_t r = shl_hi(p0, p1, s) | (p0 < 1u ? p0 : 1u);
  const uint32_t lo = shl_hi(p1, p2, s);
  return round_pack(r, 0x7FFFFFFFu + (lo & 1u), shl_hi(p2, p3, s), lo,
                    (a.hi & 0xFFF00000u) + (b.hi & 0xFFF00000u) - 0x40000000u + (top << 20));
}

// a * b, correctly rounded; the integer path where its domain holds.
AMRS_HD double dmul_rn(double a, double b) {
  const DWords A = dwords(a), B = dwords(b);
  double x = dfrom(dmul_core(A, B));
  if (!mid_range(A.hi) || !mid_range(B.hi)) {
    const bool za = ((A.hi << 1) | A.lo) == 0u, zb = ((B.hi << 1) | B.lo) == 0u;
    if ((za && (zb || mid_range(B.hi))) || (zb && mid_range(A.hi))) x = dfrom((A.hi ^ B.hi) & 0x80000000u, 0u);
    else x = dmul_hw(a, b);
  }
  return x;
}

// sqrt(x) for words in the domain (positive).  x = M 2^(2k), n' = M 2^60 in
// [2^60, 2^62); digits S1 (31 bits), s2, s3 of sqrt(n') 2^54 = S1 2^54 +
// s2 2^27 + s3 with v ~ 2^62 / sqrt(n') a few units below:
//   S1 < sqrt(n') by 0.5 .. 8,    R1 = n' - S1^2 > 0
//   s2 < R1 2^27 / (2 sqrt(n')) by 2 .. 9 (the 3 outweighs the omitted
//   second-order term),           R2 = R1 2^54 - s2 (S1 2^28 + s2) in (0, 2^63)
//   s3 ~ R2 / (2 sqrt(n')) within 4 units.
// Where that leaves the rounding open, m is the last digit with which the root
// would be the midpoint A 2^27 + m, A = S1 2^27 + s2, and the sign is that of
// n' 2^108 - (A 2^27 + m)^2 = 2^28 (R2 2^26 - m A) - m^2.
struct DSqrt {
  uint32_t S1, s2, s3, r, E;
  uint64_t R2, W;
  AMRS_HD explicit DSqrt(DWords x) {
    const uint32_t odd = (~x.hi >> 20) & 1u;  // the unbiased exponent is odd
    const uint32_t mxh = (x.hi & 0xFFFFFu) | 0x100000u;
    const uint32_t nh = shl_hi(x.lo, mxh, 10u + odd);  // top word of 4 n'
    const uint32_t v0 = seed_rsqrt((shl_hi(x.lo, x.hi, 3) & 0x7FFFFFu) | (0x3F800000u + (odd << 23)));
    const int32_t e = (int32_t)(0x3FFFFFFFu - mulhi32(mulhi32(v0, v0), nh));
    const uint32_t v = v0 + seed_corr(v0, e) - 4u;
    S1 = mulhi32(nh, v);
    const uint64_t n4 = ((uint64_t)shl_hi(x.lo, mxh, 8u + odd) << 32) | (x.lo << (8u + odd));
    const uint64_t R1 = n4 - (uint64_t)S1 * S1;
    s2 = mulhi32((uint32_t)(R1 >> 4), v) - 3u;
    const uint64_t M = madw(S1, 1u << 28, s2);
    const uint64_t P = madw(s2, (uint32_t)M, (uint64_t)(s2 * (uint32_t)(M >> 32)) << 32);
    R2 = ((uint64_t)((uint32_t)R1 << 22) << 32) - P;
    s3 = mulhi32((uint32_t)(R2 >> 31), v);
    const uint64_t T = madw(s2, 1u << 27, s3);
    W = madw(S1, 1u << 22, T >> 32);
    r = (uint32_t)T;
    E = (((x.hi + 0x100000u) >> 1) & 0x7FF00000u) + (510u << 20);
  }
  AMRS_HD bool undecided() const { return r - 0x7FFFFFF8u < 16u; }
  AMRS_HD void decide() {
    const uint32_t m = s3 + (0x80000000u - r);
    const uint64_t A = madw(S1, 1u << 27, s2);
    const int64_t Y = (int64_t)((R2 << 26) - (madw(m, (uint32_t)A, 0ull) + ((uint64_t)(m * (uint32_t)(A >> 32)) << 32)));
    r = Y > (int64_t)(((uint64_t)m * m) >> 28) ? 0x80000000u : 0x7FFFFFFFu;
  }
  AMRS_HD DWords pack() const { return round_pack(r, 0x80000000u, (uint32_t)(W >> 32), (uint32_t)W, E); }
};
AMRS_HD DWords dsqrt_core(DWords x) {
  DSqrt q(x);
  if (__builtin_expect(q.undecided(), 0)) q.decide();
  return q.pack();
}

AMRS_HD bool dsqrt_range(uint32_t hi) { return hi - (520u << 20) < (1008u << 20); }
AMRS_OUT_OF_LINE double dsqrt_rest(double x) {
  const DWords X = dwords(x);
  return dsqrt_range(X.hi) ? dfrom(dsqrt_core(X)) : AMRS_SQRT(x);
}

// sqrt(x), correctly rounded; the integer path for positive x in its domain,
// +-0 directly, anything else by the hardware square root.
AMRS_HD double dsqrt_rn(double x) {
  const DWords X = dwords(x);
  const DSqrt q(X);
  double y = dfrom(q.pack());
  if (!dsqrt_range(X.hi) || q.undecided()) {
    if (((X.hi << 1) | X.lo) == 0u) y = x;
    else y = dsqrt_rest(x);
  }
  return y;
}

}  // namespace amrs

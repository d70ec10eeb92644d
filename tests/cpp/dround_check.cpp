// Host check of the quotients and roots whose 84-bit truncation cannot decide the
// rounding (amrsolver_gb300/csrc/ddiv.cuh: ddiv_core, dsqrt_core), against the host's
// IEEE operations: 1/x and sqrt(x) for x a few units in the last place from a power
// of two, quotients of such numbers, and quotients and roots built to lie next to a
// midpoint q (54 bits, odd) on either side: q b or q^2 is d more or less than a number
// of 53 bits, d small, from q = d / b and q = sqrt(d) modulo 2^55.  The cores are called
// themselves, so nothing else can stand in.  Prints "mismatches N checked M".
//   dround_check <count> <seed>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../amrsolver_gb300/csrc/ddiv.cuh"

static uint64_t s_state;
static uint64_t rnd() {  // splitmix64
  uint64_t z = (s_state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static double from_bits(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static uint64_t to_bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }

static long long bad = 0, checked = 0;
static void say(const char* op, double a, double b, double ref, double got) {
  ++checked;
  if (to_bits(ref) == to_bits(got)) return;
  if (bad < 10) printf("MISMATCH %s a=%a b=%a ref=%a got=%a\n", op, a, b, ref, got);
  ++bad;
}
static void quot(double a, double b) { say("div", a, b, a / b, amrs::dfrom(amrs::ddiv_core(amrs::dwords(a), amrs::dwords(b)))); }
static void root(double a) { say("sqrt", a, 0, std::sqrt(a), amrs::dfrom(amrs::dsqrt_core(amrs::dwords(a)))); }
static double near(int e, long long k) { return from_bits(((uint64_t)(1023 + e) << 52) + (uint64_t)k); }

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
  s_state = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1;
  for (long long k = -3000; k <= 3000; ++k)
    for (int e = -3; e <= 3; ++e) {
      quot(1.0, near(e, k));
      quot(-3.0, near(e, k));
      root(near(e, k));
      for (long long j = -4; j <= 4; ++j) quot(near(0, j), near(e, k));
    }
  for (long long i = 0; i < n; ++i) {
    const uint64_t d = (rnd() >> (39 + rnd() % 24)) | 1ull;  // up to 2^25
    const uint64_t sd = (rnd() & 1) ? d : 0ull - d;
    {  // quotient: q b = d mod 2^54, b odd
      const uint64_t mb = (1ull << 52) | (rnd() >> 12) | 1ull;
      uint64_t inv = mb;  // Newton: correct to 3, 6, .. 96 bits
      for (int k = 0; k < 5; ++k) inv *= 2ull - mb * inv;
      const uint64_t q = (sd * inv) & ((1ull << 54) - 1);
      const unsigned __int128 p = (unsigned __int128)q * mb - (unsigned __int128)(__int128)(int64_t)sd;
      const int sh = (p >> 106) ? 54 : 53;
      const uint64_t ma = (uint64_t)(p >> sh);
      if (q >> 53 && ma >> 52 == 1ull)
        quot(from_bits((ma & 0xFFFFFFFFFFFFFull) | (1020ull << 52)), from_bits((mb & 0xFFFFFFFFFFFFFull) | (1023ull << 52)));
    }
    {  // root: q^2 = s mod 2^55, s = 1 mod 8
      const uint64_t s = (sd & ~7ull) | 1ull;
      uint64_t q = 1ull | (rnd() & 4ull);  // one of the roots, lifted bit by bit
      q = ((q * q - s) & 15ull) ? q ^ 4ull : q;
      for (int k = 4; k < 56; ++k)
        if (((q * q - s) >> k) & 1ull) q ^= 1ull << (k - 1);
      if (rnd() & 1) q = 0ull - q;
      q = (q & ((1ull << 54) - 1)) | (1ull << 53);
      const unsigned __int128 p = (unsigned __int128)q * q;
      for (int sh = 53; sh <= 55; ++sh) {
        const uint64_t m = (uint64_t)((p + ((unsigned __int128)1 << (sh - 1))) >> sh);  // the nearest
        if (m >> 52 == 1ull) root(from_bits((m & 0xFFFFFFFFFFFFFull) | ((uint64_t)(1023 + sh + 52 - 106) << 52)));
      }
    }
    // a 54-bit odd q (a midpoint) and b: a nearest to q b / 2 and its neighbours, then all sizes of the error
    const uint64_t q = (1ull << 53) | (rnd() >> 11) | 1ull;
    const uint64_t mb = (1ull << 52) | (rnd() >> (12 + rnd() % 52));  // short significands too
    const unsigned __int128 p = (unsigned __int128)q * mb;            // in [2^105, 2^107)
    const int sh = (p >> 106) ? 54 : 53;
    const uint64_t ma = (uint64_t)(p >> sh);
    const double b = from_bits((mb & 0xFFFFFFFFFFFFFull) | ((uint64_t)(1000 + rnd() % 40) << 52));
    for (int d = -1; d <= 2; ++d) {
      const uint64_t m = ma + (uint64_t)(int64_t)d;
      if (m >> 52 == 1ull) quot(from_bits((m & 0xFFFFFFFFFFFFFull) | (1020ull << 52)), b);
    }
    // the squares of midpoints
    const double x = (double)q;
    const double s = x * x;
    for (int d = -1; d <= 1; ++d) root(from_bits(to_bits(s) + (uint64_t)(int64_t)d));
    const uint64_t low = (rnd() >> (11 + rnd() % 53)) | 1ull;  // an odd number of units above one, two
    root(near((int)(rnd() & 1), (long long)(low & 0xFFFFFFFFFFFFFull)));
    quot(1.0, near(0, -(long long)(low & 0xFFFFFFFFFFFFFull)));
  }
  printf("mismatches %lld checked %lld\n", bad, checked);
  return bad ? 1 : 0;
}

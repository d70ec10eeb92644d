// Positive addition and products by small integers (dadd_pos, dmul_small) against
// the host's, bit for bit:
// dadd_check COUNT SEED.
#include <stdio.h>
#include <stdlib.h>

#include <random>

#include "../../amrsolver_gb300/csrc/ddiv.cuh"

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
  std::mt19937_64 r(argc > 2 ? strtoull(argv[2], nullptr, 10) : 1);
  long long bad = 0;
  auto check = [&](double x, double y) {
    const double got = amrs::dfrom(amrs::dadd_pos(amrs::dwords(x), amrs::dwords(y)));
    volatile double want = x + y;
    const double w = want;
    if (memcmp(&got, &w, 8) != 0 && bad++ < 5) printf("%a + %a: %a, not %a\n", x, y, got, w);
  };
  auto times = [&](double x, double k, amrs::DWords w) {
    const double got = amrs::dfrom(w);
    volatile double want = k * x;
    const double e = want;
    if (memcmp(&got, &e, 8) != 0 && bad++ < 5) printf("%a * %a: %a, not %a\n", k, x, got, e);
  };
  auto make = [](uint64_t e, uint64_t m) {
    const uint64_t u = e << 52 | (m & 0xFFFFFFFFFFFFFull);
    double x;
    memcpy(&x, &u, 8);
    return x;
  };
  // exponents over the whole range, differences around 0, 53 and 63, and
  // significands random, short, all ones and with long runs of zeros
  for (long long i = 0; i < n; ++i) {
    const uint64_t e = 70 + r() % 1900, d = r() % 4 ? r() % 70 : r() % (e - 1);
    uint64_t m[2] = {r(), r()};
    for (auto& v : m) {
      const unsigned k = r() % 8;
      if (k == 0) v = 0;
      else if (k == 1) v = ~0ull;
      else if (k == 2) v = ~0ull << (r() % 53);
      else if (k == 3) v = 1ull << (r() % 52);
      else if (k == 4) v = ~0ull >> (12 + r() % 52);
    }
    const double x = make(e, m[0]), y = make(d < e ? e - d : 1, m[1]);
    check(x, y);
    check(y, x);
    const double v = r() % 2 ? x : -x;
    const amrs::DWords a = amrs::dwords(v);
    times(v, 3, amrs::dmul_small<3>(a));
    times(v, 5, amrs::dmul_small<5>(a));
    times(v, 7, amrs::dmul_small<7>(a));
    times(v, 11, amrs::dmul_small<11>(a));
  }
  printf("mismatches %lld checked %lld\n", bad, 6 * n);
  return bad != 0;
}

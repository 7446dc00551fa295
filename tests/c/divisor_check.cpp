// Checks invariant_divisor (csrc/host_common.h): for random divisors, those of
// the uniform grids 1/2 .. 1/4096 and short significands, the two-instruction
// quotient fma(x, zh, x zl) against the division on random numerators and on
// the numerators whose quotient lies nearest to a midpoint of two doubles
// (found here by a search over convergents, not by the function's own list).
// Prints: divisors, divisors without a pair, wrong quotients, and wrong
// quotients of the single product x zh (which must be many).
#include <cstdio>
#include <cstring>
#include <random>

#include "host_common.h"

int main() {
  std::mt19937_64 g(20260301);
  long none = 0, total = 0, wrong = 0, naive = 0;
  auto try_x = [&](double x, double y, double zh, double zl) {
    const double q = x / y;
    wrong += std::fma(x, zh, x * zl) != q;
    naive += x * zh != q;
  };
  for (int k = 0; k < 6000; k++) {
    double y;
    uint64_t b = (g() >> 12) | 0x3f50000000000000ull;
    std::memcpy(&y, &b, 8);
    if (k % 3 == 1) y = 1.0 / (2 + k % 4096);
    if (k % 3 == 2) {
      b &= ~((1ull << (k % 50)) - 1);
      std::memcpy(&y, &b, 8);
    }
    double zh, zl;
    total++;
    if (!sns::invariant_divisor(y, &zh, &zl)) {
      none++;
      continue;
    }
    for (int j = 0; j < 200; j++) {
      double x;
      uint64_t c = (g() >> 12) | 0x3ff0000000000000ull;
      std::memcpy(&x, &c, 8);
      try_x(x, y, zh, zl);
      try_x(-x * 1e-30, y, zh, zl);
    }
    // numerators next to y times a midpoint, whose quotient rounds by its last bits
    for (int j = 0; j < 200; j++) {
      double m;
      uint64_t c = (g() >> 12) | 0x3ff0000000000000ull;
      std::memcpy(&m, &c, 8);
      const double x0 = std::fma(m, y, y * 1.1102230246251565e-16);
      try_x(x0, y, zh, zl);
      try_x(std::nextafter(x0, 0.0), y, zh, zl);
      try_x(std::nextafter(x0, 1e9), y, zh, zl);
    }
    try_x(0.0, y, zh, zl);
  }
  std::printf("%ld %ld %ld %ld\n", total, none, wrong, naive);
  return 0;
}

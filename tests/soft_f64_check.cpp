// soft_product (csrc/ntk_soft_f64.cuh) against the host's IEEE product:
// prints "checked wrong refused" over random operands of every magnitude,
// short mantissas and operands next to powers of two.
#include <cstdio>
#include <random>

#include "ntk_soft_f64.cuh"

static double from(uint64_t u) {
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}

int main() {
  std::mt19937_64 r(7);
  long checked = 0, wrong = 0, refused = 0;
  for (long i = 0; i < 4000000; ++i) {
    uint64_t a = r(), g = r();
    if (i % 4 == 1) a &= 0xfffff80000000000ull, g &= 0xfffff00000000000ull;  // exact products
    if (i % 4 == 2) a = (a & 0xfff0000000000000ull) | (r() % 3 ? 0 : 0x000fffffffffffffull);
    if (i % 4 == 3) g = (g & 0xfff0000000000000ull) | (r() % 3 ? 1 : 0x000fffffffffffffull);
    if (i % 8) g = (g & 0x800fffffffffffffull) | ((uint64_t)(1023 - 60 + r() % 121) << 52);
    const double x = from(a), y = from(g);
    const ntk::SoftFactor f = ntk::soft_factor(y);
    if (!ntk::soft_in_range(x, f)) {
      ++refused;
      continue;
    }
    ++checked;
    if (ntk::soft_product(x, f) != x * y) ++wrong;
  }
  for (double x : {0.0, -0.0, 5e-324, 1e-308, 1e300 * 1e10, -(1e300 * 1e10), 1e308})  // never taken
    if (ntk::soft_in_range(x, ntk::soft_factor(1.5))) ++wrong;
  for (double y : {0.0, 1e-20, 1e20, 5e-324})
    if (ntk::soft_in_range(1.0, ntk::soft_factor(y))) ++wrong;
  std::printf("%ld %ld %ld\n", checked, wrong, refused);
  return 0;
}

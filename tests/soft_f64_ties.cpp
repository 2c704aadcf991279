// soft_product and, where it serves, soft_product_untied
// (csrc/ntk_soft_f64.cuh) against the host's IEEE product where the exact
// product may lie halfway between two doubles: short factors times full
// operands and the reverse.  Factors within
// 2^+-SOFT_SPAN, the kernels' range, with operands of every exponent.  Prints
// "checked ties wrong untied wrong wide wrong".
#include <cstdio>
#include <random>

#include "ntk_soft_f64.cuh"

static double from(uint64_t u) {
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}

int main() {
  std::mt19937_64 r(11);
  long checked = 0, ties = 0, wrong = 0, untied = 0, wrong2 = 0, wide = 0, wrong3 = 0;
  auto check = [&](double a, double g) {
    const ntk::SoftFactor f = ntk::soft_factor(g), f2 = ntk::soft_factor_untied(g);
    if (!ntk::soft_in_range(a, f)) return;
    uint64_t ma, mg;
    std::memcpy(&ma, &a, 8);
    std::memcpy(&mg, &g, 8);
    ma = (ma & ((1ull << 52) - 1)) | 1ull << 52;
    mg = (mg & ((1ull << 52) - 1)) | 1ull << 52;
    const unsigned __int128 p = (unsigned __int128)ma * mg;  // [2^104, 2^106)
    const int drop = p >> 105 ? 53 : 52;
    const unsigned __int128 rest = p & (((unsigned __int128)1 << drop) - 1);
    ties += rest == (unsigned __int128)1 << (drop - 1);
    ++checked;
    if (ntk::soft_product(a, f) != a * g) ++wrong;
    if (!ntk::soft_untied(a, f2)) return;
    ++untied;
    if (ntk::soft_product_untied(a, f2) != a * g) ++wrong2;
  };
  const double shorts[] = {1.5, .75, 3., .375, 1.25, 5.5, 381.75, -1.5, -.625, 1. + 1. / 1024};
  for (int i = 0; i < 400000; ++i) {
    // operands of 53 - 3 * (i % 18) significant bits, exponents within the range
    const uint64_t bits = (r() & ~(((uint64_t)1 << (3 * (i % 18))) - 1) & 0x800fffffffffffffull);
    const double a = from(bits | (uint64_t)(1023 - 200 + r() % 400) << 52);
    for (double g : shorts) check(a, g);
    // a factor of full length and one of any length beside it
    check(a, from(r() & 0x800fffffffffffffull | (uint64_t)(1023 - 60 + r() % 121) << 52));
    const uint64_t gb = r() & ~(((uint64_t)1 << (r() % 53)) - 1) & 0x800fffffffffffffull;
    check(a, from(gb | (uint64_t)(1023 - 60 + r() % 121) << 52));
  }
  for (int i = 0; i < 2000000; ++i) {
    const double a = from(r()), g = from((r() & 0x800fffffffffffffull) | (uint64_t)(1023 - 260 + r() % 521) << 52);
    const ntk::SoftFactor f = ntk::soft_factor(g, ntk::SOFT_SPAN), f2 = ntk::soft_factor_untied(g, ntk::SOFT_SPAN);
    if (ntk::soft_in_range(a, f, ntk::SOFT_SPAN)) {
      ++wide;
      wrong3 += ntk::soft_product(a, f) != a * g;
    }
    if (ntk::soft_untied(a, f2, ntk::SOFT_SPAN)) wrong3 += ntk::soft_product_untied(a, f2) != a * g;
  }
  for (double g : {1e76, -1e-76, 0.0})  // beyond the span
    wrong3 += ntk::soft_in_range(1.0, ntk::soft_factor(g, ntk::SOFT_SPAN), ntk::SOFT_SPAN);
  std::printf("%ld %ld %ld %ld %ld %ld %ld\n", checked, ties, wrong, untied, wrong2, wide, wrong3);
  return 0;
}

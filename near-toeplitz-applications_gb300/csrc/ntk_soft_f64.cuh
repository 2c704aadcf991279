// ntk_soft_f64.cuh -- FP64 products by tabulated factors on the integer pipes.
//
// A warp-wide FP64 instruction holds a GB300 sub-partition's FP64 pipe for
// ~76 clocks, while its integer and FP32 pipes idle: an FP64 operation that
// takes fewer than 76 issue slots in integer arithmetic, off the dependent
// chain, is cheaper there, and runs beside the FP64 instructions that stay.
// soft_product (~45 clocks) is such an operation: the exact 106-bit product
// rounded to 53 bits, ties to even, i.e. the IEEE product bit for bit.  Ties
// are common where an operand is short (one product in six for 1.5 or 0.75).
// Operands outside the range where neither overflow nor underflow can occur
// (subnormal, inf and nan among them) take the FP64 pipe's product; zeros,
// which are out of that range too, a path of their own (rare_rows).
// soft_product_untied (41 clocks) rounds half up and serves operands whose
// product cannot be a tie; the one-thread sweeps, which both pipes bound, take
// it and leave the others to the FP64 pipe (a 512^3 gradient 2817 -> 2919 us
// with soft_product, 2836 so).  Kernels with few rows a thread take
// soft_product: a block of rows with a boundary value of 1 or a factor of 1.5
// beside the FP64 product costs them more (a 256 x 256 derivative 8.2 -> 10.2
// us, ADI steps 5%).
// Compiles for the host too, where tests/soft_f64_check.cpp and
// tests/soft_f64_ties.cpp compare it with the host's IEEE product.
#pragma once
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

#ifdef __CUDACC__
#define SOFT_HD __host__ __device__ __forceinline__
#else
#define SOFT_HD inline
#endif

namespace ntk {

// A factor prepared for soft_product: mantissa with its leading one in bit
// 63, and what to add to the other operand's upper word (exponent, and the
// sign by wrapping).  lim: how many exponents of the other operand, from span
// + 4 on and in units of its upper word, are served; 0: none (a factor that is
// zero, not finite or beyond 2^+-span).  The kernels serve factors within
// 2^+-SOFT_SPAN (coefficients in any units: 1 / dx^2 is beyond 2^60 from dx =
// 1e-9 on) times operands within 1e+-229.
struct SoftFactor {
  uint64_t mant;
  uint32_t eadd;
  uint32_t lim;
};

SOFT_HD uint32_t soft_hi(double a) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(a);
#else
  uint64_t u;
  std::memcpy(&u, &a, 8);
  return (uint32_t)(u >> 32);
#endif
}
SOFT_HD uint32_t soft_lo(double a) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(a);
#else
  uint64_t u;
  std::memcpy(&u, &a, 8);
  return (uint32_t)u;
#endif
}
SOFT_HD double soft_double(uint64_t r) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double x;
  std::memcpy(&x, &r, 8);
  return x;
#endif
}

constexpr int SOFT_SPAN = 250;

SOFT_HD SoftFactor soft_factor(double g, int span = 60) {
  const uint64_t u = (uint64_t)soft_hi(g) << 32 | soft_lo(g);
  const int e = (int)((u >> 52) & 0x7ff) - 1023;
  SoftFactor f;
  f.mant = (u << 11) | (1ull << 63);
  // the leading one of the rounded mantissa adds one to the exponent field
  f.eadd = ((uint32_t)e << 20) + (uint32_t)(u >> 63 << 31);
  f.lim = (e >= -span && e <= span) ? (uint32_t)(2036 - 2 * span) << 20 : 0u;
  return f;
}

// The factor for soft_product_untied: factors of 2 .. 33 significant bits are
// not served (a product by one of 34 or more bits is no tie unless the
// operand's lower word is zero, a product by a power of two is exact).
SOFT_HD SoftFactor soft_factor_untied(double g, int span = 60) {
  SoftFactor f = soft_factor(g, span);
  if ((f.mant & 0x7fffffffull) == 0 && f.mant << 1 != 0) f.lim = 0;
  return f;
}

SOFT_HD uint64_t soft_umul64hi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// FP64 work that few rows need, as calls: ptxas turns a short conditional
// body (an `if`, a loop of at most one turn, a bra.uni) into predicated
// instructions, and a predicated-off FP64 instruction holds the FP64 pipe like
// an executed one (soft_product beside a DFMA: 76 clocks a warp; with its
// range check as an `if` around an FP64 product 149, around a call 76).
#ifdef __CUDACC__
static __device__ __noinline__ double rare_mul(double a, double b) { return a * b; }
// the compact scheme's one-sided boundary stencils (compact/rhs.py:21-31)
static __device__ __noinline__ double one_sided(double sigma, double f0, double f1, double f2) {
  return sigma * ((-5.0 * f0 + 4.0 * f1) + f2);
}
#endif

// whether soft_product serves operand a
SOFT_HD bool soft_in_range(double a, const SoftFactor& f, int span = 60) {
  return (soft_hi(a) & 0x7fffffffu) - ((uint32_t)(span + 4) << 20) < f.lim;
}

// a times the factor, a in range
SOFT_HD double soft_product(double a, const SoftFactor& f) {
  const uint32_t ah = soft_hi(a), al = soft_lo(a);
  const uint32_t mh = (ah << 11 | al >> 21) | 0x80000000u, ml = al << 11;
  const uint32_t gh = (uint32_t)(f.mant >> 32), gl = (uint32_t)f.mant;
  // the 128-bit product: t, and its lower words as a sticky word
  const uint64_t p = (uint64_t)ml * gl;
  const uint64_t q = (uint64_t)mh * gl + (p >> 32);
  const uint64_t s = (uint64_t)ml * gh + (uint32_t)q;
  uint64_t t = (uint64_t)mh * gh + (q >> 32) + (s >> 32);  // [2^62, 2^64)
  const uint32_t low = (uint32_t)s | (uint32_t)p;
  uint32_t e = (ah & 0xfff00000u) + f.eadd;
  if (t >> 63 == 0) {
    t <<= 1;
    e -= 1u << 20;
  }
  uint64_t r = ((uint64_t)e << 32) + (t >> 11) + ((t >> 10) & 1u);
  if (((((uint32_t)t ^ 0x400u) & 0x7ffu) | low) == 0) r &= ~(uint64_t)1;  // a tie, rounded up: the even neighbour
  return soft_double(r);
}

// whether soft_product_untied is the IEEE product of a and a soft_factor_untied
SOFT_HD bool soft_untied(double a, const SoftFactor& f, int span = 60) {
  return soft_in_range(a, f, span) && soft_lo(a) != 0;
}

SOFT_HD double soft_product_untied(double a, const SoftFactor& f) {
  const uint32_t ah = soft_hi(a), al = soft_lo(a);
  const uint64_t m = (((uint64_t)ah << 32 | al) << 11) | (1ull << 63);
  uint64_t t = soft_umul64hi(m, f.mant);  // [2^62, 2^64)
  uint32_t e = (ah & 0xfff00000u) + f.eadd;
  if (t >> 63 == 0) {
    t <<= 1;
    e -= 1u << 20;
  }
  return soft_double(((uint64_t)e << 32) + (t >> 11) + ((t >> 10) & 1u));
}

#ifdef __CUDACC__
__device__ __forceinline__ SoftFactor load_factor(const SoftFactor* p) {
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
  return SoftFactor{(uint64_t)q.y << 32 | q.x, q.z, q.w};
}
#endif

// whether a is +-0, without an FP64 comparison
SOFT_HD bool soft_zero(double a) { return (soft_hi(a) << 1 | soft_lo(a)) == 0; }

// the zero a times g, g finite
SOFT_HD double soft_zero_times(double a, double g) {
  return soft_double((uint64_t)((soft_hi(a) ^ soft_hi(g)) & 0x80000000u) << 32);
}
SOFT_HD bool soft_finite(double g) { return (soft_hi(g) & 0x7ff00000u) != 0x7ff00000u; }

#ifdef __CUDACC__
// y[k] = a[k] g(k) where some of a block's rows are not served(k).  Zeros, of
// which fields with quiet regions are full, keep off the FP64 pipe here too: a
// block whose other rows are served keeps their products.
template <int N, class G, class S>
__device__ __forceinline__ void rare_rows(const double (&a)[N], double (&y)[N], G g, S served) {
  bool zeros = true;
#pragma unroll
  for (int k = 0; k < N; ++k) zeros = zeros && (served(k) || (soft_zero(a[k]) && soft_finite(g(k))));
  if (zeros) {
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (soft_zero(a[k])) y[k] = soft_zero_times(a[k], g(k));
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = rare_mul(a[k], g(k));
  }
}
#endif

}  // namespace ntk

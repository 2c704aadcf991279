// ntk_soft_f64.cuh -- FP64 products by tabulated factors on the integer pipes.
//
// A warp-wide FP64 instruction holds a GB300 sub-partition's FP64 pipe for
// ~76 clocks, while its integer and FP32 pipes idle: an FP64 operation that
// takes fewer than 76 issue slots in integer arithmetic, off the dependent
// chain, is cheaper there, and runs beside the FP64 instructions that stay.
// soft_product (41 clocks) is such an operation: the exact 106-bit product's upper 64 bits,
// rounded to 53, i.e. the IEEE product except that a result within 2^-62 of a
// rounding boundary may round to its other neighbour.  Operands outside the
// range where neither overflow nor underflow can occur (zero, subnormal, inf
// and nan among them) take the FP64 pipe's product.
// Compiles for the host too, where tests/soft_f64_check.cpp compares it with
// the host's IEEE product.
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
// sign by wrapping).  lim: how many exponents of the other operand, from 64
// on and in units of its upper word, are served; 0: none (a factor that is
// zero, not finite or beyond 2^+-60).
struct SoftFactor {
  uint64_t mant;
  uint32_t eadd;
  uint32_t lim;
};

SOFT_HD SoftFactor soft_factor(double g) {
#ifdef __CUDA_ARCH__
  const uint64_t u = (uint64_t)__double_as_longlong(g);
#else
  uint64_t u;
  std::memcpy(&u, &g, 8);
#endif
  const int e = (int)((u >> 52) & 0x7ff) - 1023;
  SoftFactor f;
  f.mant = (u << 11) | (1ull << 63);
  // the leading one of the rounded mantissa adds one to the exponent field
  f.eadd = ((uint32_t)e << 20) + (uint32_t)(u >> 63 << 31);
  f.lim = (e >= -60 && e <= 60) ? (1980u - 64u) << 20 : 0u;
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
SOFT_HD bool soft_in_range(double a, const SoftFactor& f) {
#ifdef __CUDA_ARCH__
  const uint32_t ah = (uint32_t)__double2hiint(a);
#else
  uint64_t ua;
  std::memcpy(&ua, &a, 8);
  const uint32_t ah = (uint32_t)(ua >> 32);
#endif
  return (ah & 0x7fffffffu) - (64u << 20) < f.lim;
}

// a times the factor, a in range
SOFT_HD double soft_product(double a, const SoftFactor& f) {
#ifdef __CUDA_ARCH__
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
#else
  uint64_t ua;
  std::memcpy(&ua, &a, 8);
  const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua;
#endif
  const uint64_t m = (((uint64_t)ah << 32 | al) << 11) | (1ull << 63);
  uint64_t t = soft_umul64hi(m, f.mant);  // [2^62, 2^64)
  uint32_t e = (ah & 0xfff00000u) + f.eadd;
  if (t >> 63 == 0) {
    t <<= 1;
    e -= 1u << 20;
  }
  const uint64_t r = ((uint64_t)e << 32) + (t >> 11) + ((t >> 10) & 1u);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double x;
  std::memcpy(&x, &r, 8);
  return x;
#endif
}

}  // namespace ntk

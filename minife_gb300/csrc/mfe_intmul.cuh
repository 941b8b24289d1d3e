// FP64 multiplication, correctly rounded, on the integer pipe.
//
// GB300's FP64 pipe takes 1.9 operations per clock and SM, its integer pipe 64.
// A multiplication of two normal numbers whose product is normal takes 18
// integer instructions, so moving multiplications there frees the FP64 pipe
// for the additions (the element matrices, mfe_hex8.cuh).  The result is the
// IEEE 754 product rounded to nearest even, bit for bit.
//
// With the operands' 53-bit mantissas shifted left by 6, the 118-bit product is
// h 2^64 + (m.lo, t.lo) with h in [2^52, 2^54): h holds the result's mantissa,
// or twice it (s = 1).  Rounding adds half a unit of the last place kept (at
// bit 63 below h, or at bit 0 of h) and clears the last bit on a tie, which is
// when every bit below the one added is then zero.
#pragma once

#include <cstdint>

namespace mfe {

// A normal FP64 number taken apart: mantissa 2^6 (h 2^32 + l) and the sign and
// exponent field less 512, so that two of them add to the product's.
struct IntMul {
  uint32_t l, h, se;
};

__host__ __device__ __forceinline__ IntMul intmul_split(uint32_t hi, uint32_t lo)
{
  const uint32_t m = (hi & 0xfffffu) | 0x100000u;
  IntMul a;
  a.l = lo << 6;
#ifdef __CUDA_ARCH__
  a.h = __funnelshift_l(lo, m, 6);
#else
  a.h = (m << 6) | (lo >> 26);
#endif
  a.se = (hi & 0xfff00000u) - (512u << 20);
  return a;
}

// hi and lo words of a b, for normal a and b whose product is normal
__host__ __device__ __forceinline__ void intmul(const IntMul& a, const IntMul& b, uint32_t& hi, uint32_t& lo)
{
#ifdef __CUDA_ARCH__
  uint64_t t, m, h;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(t) : "r"(a.l), "r"(b.l));
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(m) : "r"(a.l), "r"(b.h), "l"(t >> 32));
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(m) : "r"(a.h), "r"(b.l), "l"(m));
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(h) : "r"(a.h), "r"(b.h), "l"(m >> 32));
#else
  const uint64_t t = (uint64_t)a.l * b.l;
  uint64_t m = (uint64_t)a.l * b.h + (t >> 32);
  m += (uint64_t)a.h * b.l;
  const uint64_t h = (uint64_t)a.h * b.h + (m >> 32);
#endif
  const uint32_t s = (uint32_t)(h >> 53);
  const uint32_t half = (s << 31) ^ 0x80000000u;  // the half below h, where s = 0
  uint32_t r0, r1, r2;                            // h and the word below it, the half added
#ifdef __CUDA_ARCH__
  asm("{\n\tadd.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;\n\t}"
      : "=r"(r0), "=r"(r1), "=r"(r2)
      : "r"((uint32_t)m), "r"(half), "r"((uint32_t)h), "r"(s), "r"((uint32_t)(h >> 32)));
#else
  r0 = (uint32_t)m + half;
  const uint64_t r = h + s + (r0 < half ? 1u : 0u);
  r1 = (uint32_t)r;
  r2 = (uint32_t)(r >> 32);
#endif
  const bool tie = ((r1 & s) | r0 | (uint32_t)t) == 0u;
#ifdef __CUDA_ARCH__
  lo = __funnelshift_r(r1, r2, s);
#else
  lo = s ? (r1 >> 1) | (r2 << 31) : r1;
#endif
  if (tie) lo &= ~1u;
  hi = (r2 >> s) + a.se + b.se + (s << 20);
}

#ifdef __CUDACC__
__device__ __forceinline__ IntMul intmul_split(double a)
{
  return intmul_split((uint32_t)__double2hiint(a), (uint32_t)__double2loint(a));
}

__device__ __forceinline__ double intmul(const IntMul& a, const IntMul& b)
{
  uint32_t hi, lo;
  intmul(a, b, hi, lo);
  return __hiloint2double((int)hi, (int)lo);
}

// 2^-R <= |a| < 2^(R + 1)
template <int R>
__device__ __forceinline__ bool intmul_range(double a)
{
  const uint32_t m = (uint32_t)__double2hiint(a) & 0x7fffffffu;
  return m - ((uint32_t)(1023 - R) << 20) < ((uint32_t)(2 * R + 1) << 20);
}
#endif

}  // namespace mfe

// Mersenne twister of the McICA generator (mcica_random_numbers.f90:77-306),
// device side.  The reference's int32 arithmetic with logical ishft is uint32
// arithmetic; getRandomReal is u32 / (2^32 - 1) in double precision.
#pragma once
#include <stdint.h>

namespace gbmt {

__device__ __forceinline__ uint32_t temper(uint32_t y) {
  uint32_t x = y ^ (y >> 11);
  x ^= (x << 7) & 0x9d2c5680u;
  x ^= (x << 15) & 0xefc60000u;
  return x ^ (x >> 18);
}
__device__ __forceinline__ uint32_t twist(uint32_t u, uint32_t v) {
  return (((u & 0x80000000u) | (v & 0x7fffffffu)) >> 1) ^ ((v & 1u) ? 0x9908b0dfu : 0u);
}
// u / (2^32 - 1) rounded to nearest, in integer arithmetic (a conversion and a
// division in fp64 are some fifteen instructions at 1/64 of the integer rate).
// In base 2^32 the quotient is 0.uuu..., so its bits from the first set one on are r r r ...
// with r = u rotated left by its leading zeros z: the significand is the first
// 53 of them, rounded by the next one (never a tie: the bits go on with another
// r), and all ones carry over into 1.
__device__ __forceinline__ double real(uint32_t u) {
  const int z = __clz(u);
  const uint32_t r = __funnelshift_l(u, u, z);
  const unsigned long long m = ((unsigned long long)(r >> 11) << 32 | (r << 21 | r >> 11)) + (r >> 10 & 1u);
  return u ? __longlong_as_double((long long)(m + ((unsigned long long)(uint32_t)(1021 - z) << 52))) : 0.0;
}

}  // namespace gbmt

// A 32-bit number as three bfloat16 parts, x = high + middle + low exactly (numbers above 2^-110): each part is the next eight bits of the
// mantissa, cut off, so all have the sign of x and none is larger than x.  Products of the parts with a bfloat16 number are exact in 32 bit,
// so three warp-level MMAs give a product with a 32-bit operand.  An infinite x is its high part, with zeros behind it, and a NaN stays one.
// Pairs of neighbours, as MMA fragments hold them.
#pragma once
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

__device__ __forceinline__ float bf16_low(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_high(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ void split3(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low) {
  const auto upper = [](float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); };
  const auto rest = [](float a) { return a - __uint_as_float(__float_as_uint(a) & 0xffff0000u); };
  high = upper(x, y);
  x = fabsf(x) == INFINITY ? 0.f : rest(x);
  y = fabsf(y) == INFINITY ? 0.f : rest(y);
  middle = upper(x, y);
  low = upper(rest(x), rest(y));
}

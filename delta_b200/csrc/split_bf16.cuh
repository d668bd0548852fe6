// A 32-bit number as three bfloat16 parts, x = high + middle + low up to 2^-24 of it: products of the parts with a bfloat16 number are
// exact in 32 bit, so three warp-level MMAs give a product with a 32-bit operand.  Pairs of neighbours, as MMA fragments hold them.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

__device__ __forceinline__ float bf16_low(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_high(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ void split3(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low) {
  __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
  high = *reinterpret_cast<uint32_t*>(&p);
  x -= bf16_low(high);
  y -= bf16_high(high);
  p = __floats2bfloat162_rn(x, y);
  middle = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(x - bf16_low(middle), y - bf16_high(middle));
  low = *reinterpret_cast<uint32_t*>(&p);
}

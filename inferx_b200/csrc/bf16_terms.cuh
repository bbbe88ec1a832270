// An fp32 number as the sum of three bfloat16 terms, each the rounding of what the ones before left
// over: 3 x 8 bits, and bfloat16 has fp32's range.  (No normal third term below 2^-102; infinities and
// numbers that round up to them leave NaN.)
#pragma once
#include "common.cuh"

// The three terms of two numbers, packed.
__device__ __forceinline__ void bf16_terms2(float a, float b, unsigned& t1, unsigned& t2,
                                            unsigned& t3) {
  __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  t1 = *reinterpret_cast<unsigned*>(&p);
  a -= __uint_as_float(t1 << 16);
  b -= __uint_as_float(t1 & 0xffff0000u);
  p = __floats2bfloat162_rn(a, b);
  t2 = *reinterpret_cast<unsigned*>(&p);
  a -= __uint_as_float(t2 << 16);
  b -= __uint_as_float(t2 & 0xffff0000u);
  p = __floats2bfloat162_rn(a, b);
  t3 = *reinterpret_cast<unsigned*>(&p);
}

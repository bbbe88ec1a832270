// What the recurrences that are walked in segments share (delta_segments.cu, linear_segments.cu):
// packed fp32 arithmetic, asynchronous copies of 16 and 4 bytes, and how a column of the state is
// laid over lanes.
#pragma once
#include "common.cuh"

#define DS_CHUNK 16           // tokens staged at a time
#define DS_THREADS 128
#define DS_WARPS (DS_THREADS / 32)

typedef unsigned long long ds_pair;       // two fp32 numbers

__device__ __forceinline__ ds_pair ds_pack(float a, float b) {
  ds_pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 ds_unpack(ds_pair p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ ds_pair ds_mul2(ds_pair a, ds_pair b) {
  ds_pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ ds_pair ds_fma2(ds_pair a, ds_pair b, ds_pair c) {
  ds_pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ void ds_async(void* dst, const void* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Lanes a column, float4 of it a lane, by the key's size.
#define DS_BY_K(K, GO)          \
  do {                          \
    if ((K) <= 16) GO(4, 1);    \
    else if ((K) <= 32) GO(4, 2);  \
    else if ((K) <= 64) GO(4, 4);  \
    else if ((K) <= 128) GO(4, 8); \
    else if ((K) <= 256) GO(16, 4);  \
    else GO(16, 8);             \
  } while (0)

static inline int ds_cols(int K) { return DS_WARPS * (K <= 128 ? 8 : 2); }
static inline int ds_pitch(int K) {
  return K <= 16 ? 16 : K <= 32 ? 32 : K <= 64 ? 64 : K <= 128 ? 128 : K <= 256 ? 256 : 512;
}

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

// How the state lies over a warp: DS_LANES neighbouring lanes share C neighbouring columns, and
// each holds KQ float4 of every one of them, entries 4 (lane + DS_LANES i) + {0..3}, so that a
// float4 of k, q or a decay from shared memory serves C columns of a thread.  (A warp's 16-byte
// read takes four cycles of shared memory, also where its lanes share addresses: with one column a
// thread and four lanes a column those reads, and not the arithmetic, bounded the walks: 2,048
// tokens of 16 heads of 64 x 128 took 330 us in the delta rule and 203 us in the linear
// recurrence.)
#define DS_LANES 8
#define DS_GROUPS (DS_WARPS * (32 / DS_LANES))    // of columns, a block

// Where segment `seg` of sequence s lies in scratch, for head h: tokens before the sequence /
// tokens a segment + the sequence's number + the segment's.  No two meet, and T / seg_len + S + 1
// hold all, also where one sequence of many is long.
__device__ __forceinline__ size_t ds_cell(const int* cu_q, int s, int seg_len, int seg, int H,
                                          int h) {
  return (size_t)(cu_q[s] / seg_len + s + seg) * H + h;
}
static inline long long ds_cells(int T, int S, int seg_len, int H) {
  return ((long long)T / seg_len + S + 1) * H;
}

// float4 a lane, columns a thread, by the key's size
#define DS_BY_K(K, GO)           \
  do {                           \
    if ((K) <= 32) GO(1, 4);     \
    else if ((K) <= 64) GO(2, 4);   \
    else if ((K) <= 128) GO(4, 4);  \
    else if ((K) <= 256) GO(8, 2);  \
    else GO(16, 1);              \
  } while (0)

static inline int ds_cols(int K) { return DS_GROUPS * (K <= 128 ? 4 : K <= 256 ? 2 : 1); }
static inline int ds_pitch(int K) {
  return K <= 32 ? 32 : K <= 64 ? 64 : K <= 128 ? 128 : K <= 256 ? 256 : 512;
}
// Blocks of a pass that an SM holds at once: by registers what the launch bounds ask for, by shared
// memory (228 KB, 1 KB of it for each block) three at keys of 128, two at 256, one beyond.
template <int KQ> constexpr int ds_min_blocks() {
  return KQ <= 2 ? 5 : KQ <= 4 ? 3 : KQ <= 8 ? 2 : 1;
}
static inline int ds_resident(int K, size_t smem) {
  const int by_registers = K <= 64 ? 5 : K <= 128 ? 3 : K <= 256 ? 2 : 1;
  const int by_smem = (int)(228 * 1024 / (smem + 1024));
  return by_smem < by_registers ? by_smem : by_registers;
}
// Blocks of such a pass that the device holds at once (without a device, a B200's).
static inline long long ds_blocks_at_once(int K, size_t smem) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    sms = 148;
  }
  return (long long)ds_resident(K, smem) * sms;
}

// The sums of C columns over the DS_LANES lanes that share them; lane l of them gets column
// ds_own<C>(l)'s.
template <int C> __device__ __forceinline__ int ds_own(int l) {
  return C == 4 ? (l >> 1) & 3 : C == 2 ? (l >> 2) & 1 : 0;
}
template <int C> __device__ __forceinline__ float ds_sum(const float* v, int l) {
  float r;
  if (C == 4) {
    const bool up = l & 4, up2 = l & 2;
    const float s0 = up ? v[0] : v[2], s1 = up ? v[1] : v[3];
    const float r0 = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, s0, 4);
    const float r1 = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, s1, 4);
    r = (up2 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, up2 ? r0 : r1, 2);
  } else if (C == 2) {
    const bool up = l & 4;
    r = (up ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[1], 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
  } else {
    r = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
  }
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
// The other way round: every lane gets the C columns' values.
template <int C> __device__ __forceinline__ void ds_share(float own, float* v, int l) {
  if (C == 4) {
    const float o = __shfl_xor_sync(0xffffffffu, own, 2);
    const float p0 = l & 2 ? o : own, p1 = l & 2 ? own : o;
    const float q0 = __shfl_xor_sync(0xffffffffu, p0, 4), q1 = __shfl_xor_sync(0xffffffffu, p1, 4);
    v[0] = l & 4 ? q0 : p0;
    v[1] = l & 4 ? q1 : p1;
    v[2] = l & 4 ? p0 : q0;
    v[3] = l & 4 ? p1 : q1;
  } else if (C == 2) {
    const float o = __shfl_xor_sync(0xffffffffu, own, 4);
    v[0] = l & 4 ? o : own;
    v[1] = l & 4 ? own : o;
  } else {
    v[0] = own;
  }
}

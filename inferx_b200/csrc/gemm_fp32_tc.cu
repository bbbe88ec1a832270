// fp32 product y = x . w^T on the 5th-generation tensor cores, for the 32-bit mode's prompts.
//
// An fp32 number is the sum of three bfloat16 terms, a = a1 + a2 + a3, each the rounding of what
// the ones before left over (3 x 8 bits, and bfloat16 has fp32's range).  The product is formed
// from six products of terms that bfloat16 MMAs add up in fp32 accumulators:
//
//   a b = a2 b2 + a1 b3 + a3 b1  +  a1 b2 + a2 b1  +  a1 b1       (in this order, small ones first)
//
// what is left out is below 2^-25 of |a b| and of either sign.  The tensor cores' accumulation is
// not fp32's rounding to nearest, so an accumulator holds 64 entries of k only and is then added
// to an fp32 register.  Both together are closer to 64 bits than a chain of K fused multiply-adds
// (relative error of normal x against normal w: 1.3e-7 against 8.1e-7 at K 2048, 1.3e-7 against
// 1.3e-6 at K 5632, 1.7e-7 against 1.9e-6 at K 11008).
//
// A block makes 128 x 128 results.  Warps 0-7 read the next 64 entries of k of its 128 + 128 rows
// into registers (a step ahead), split them into the three terms, write w's as swizzled tiles in
// shared memory and x's into tensor memory (two stages of either), and add up the accumulators of
// the step before the last; one thread of warp 8 issues the 24 MMAs of a step.  The MMAs of a step
// take 1,536 cycles (128 x 128 x 64, six times); the splitting warps, two a scheduler, about
// 1,350 issue slots and twice that in time, which is what bounds it (tensor pipe half busy).
// Measured against that: x in shared memory as well, 10 % slower (the MMAs would read all that
// shared memory gives); 16 splitting warps, 10 % slower (96 registers a thread spill); packed
// fp32 subtractions, 15 % slower.  The terms are made in the kernel, from operands read as they
// are, and not by a pass of their own: the weights' terms would be 1.5 times the weights, written
// and read again.
//
// With fewer tiles than SMs, or a last wave that is nearly empty, k is cut into `splits` runs whose
// partial sums a second kernel adds in ascending order.
//
// Infinities and NaN, and sums that overflow on the way, come out of the terms as infinities or
// NaN; bfloat16 holds no third term of numbers below 2^-110.  A sum that is not finite, or below
// 2^-64 and not 0, is computed again from the operands, fp32 multiply-adds, a warp per element.
// (What is left: operands below 2^-110 that meet others above 2^40 lose last bits.)  That code
// stands at the end of the block, unrolled: made a function on sums in shared memory, it costs the
// loop over steps 10 %, by other registers.
//
// Every mbarrier wait is bounded (codes 41: splitting warps, 42: MMA).  Requires K a multiple of
// 8 and bases on 32-byte marks.
#include <cfloat>

#include "common.cuh"
#include "tma_common.cuh"
#include "tcgen05_common.cuh"

#define F3_BM 128
#define F3_BN 128
#define F3_BK 64
#define F3_WARPS 8                                // that split and add up; one more issues MMAs
#define F3_THREADS (F3_WARPS * 32 + 32)
#define F3_PART (128 * F3_BK * 2)                 // one term of w: 16 KB
#define F3_STAGE (3 * F3_PART)

enum { F3_ERR_SPLIT = 41, F3_ERR_MMA = 42 };

struct F3Bars {
  unsigned long long full[2], done[2];
  unsigned tmem_holder;
  int abort_flag;
};

// eight consecutive k of one row
__device__ __forceinline__ void f3_load8(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
// sixteen columns of this thread's row
__device__ __forceinline__ void f3_ld16(unsigned taddr, float* v) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// The three terms of two numbers, packed.
__device__ __forceinline__ void f3_split2(float a, float b, unsigned& t1, unsigned& t2,
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
// Of eight numbers, 16 bytes each, into the same place of three tiles.
__device__ __forceinline__ void f3_split8(const float* v, unsigned char* at) {
  unsigned t1[4], t2[4], t3[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) f3_split2(v[2 * i], v[2 * i + 1], t1[i], t2[i], t3[i]);
  *reinterpret_cast<uint4*>(at) = make_uint4(t1[0], t1[1], t1[2], t1[3]);
  *reinterpret_cast<uint4*>(at + F3_PART) = make_uint4(t2[0], t2[1], t2[2], t2[3]);
  *reinterpret_cast<uint4*>(at + 2 * F3_PART) = make_uint4(t3[0], t3[1], t3[2], t3[3]);
}
// 16 lanes x 16 columns of tensor memory from a warp's registers: thread T holds columns
// 8 b + 2 (T % 4) + {0, 1} of row T / 4 in r[4 b + {0, 1}] and of row 8 + T / 4 in r[4 b + {2, 3}].
__device__ __forceinline__ void f3_st16x16(unsigned taddr, const unsigned* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}

// Whether a sum has to be made again: not finite, or so small that operands without a third term
// may have gone into it.
__device__ __forceinline__ bool f3_again(float s) {
  const float a = fabsf(s);
  return !(a <= FLT_MAX) || (a < 5.421010862427522e-20f && a > 0.f);
}

__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_fp32_tc_kernel(const float* __restrict__ x, const float* __restrict__ w,
                    float* __restrict__ out, float* __restrict__ part, int M, int N, int K,
                    int steps_per_split, int act, int* __restrict__ status) {
  constexpr unsigned IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((F3_BN >> 3) << 17) |
                             ((F3_BM >> 4) << 24);
  // two accumulators from columns 0 and 128; x's terms, 32 columns each, from 256 and 352
  constexpr unsigned TMEM_COLS = 512, X_COL = 2 * F3_BN, X_STAGE = 96;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) F3Bars bars;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // neighbouring blocks share a tile of weights
  const int m0 = blockIdx.x * F3_BM, n0 = blockIdx.y * F3_BN;
  const int k_begin = blockIdx.z * steps_per_split * F3_BK;
  const int k_end = min(K, k_begin + steps_per_split * F3_BK);
  const int n_steps = (k_end - k_begin + F3_BK - 1) / F3_BK;      // at least 1

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.full[i], F3_WARPS);
      mbar_init(&bars.done[i], 1);
    }
    bars.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == F3_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&bars.tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = bars.tmem_holder;
  volatile int* abortp = &bars.abort_flag;

  if (warp == F3_WARPS) {
    if (lane == 0) {
      bool ok = true;
      for (int j = 0; j < n_steps; ++j) {
        const int st = j & 1;
        ok = mbar_wait(&bars.full[st], (j >> 1) & 1, abortp);
        if (!ok) break;
        tc_fence_after();
        unsigned char* at = smem + st * F3_STAGE;
        const unsigned sums = tmem_base + st * F3_BN;
        // (term of x, term of w)
        constexpr int TX[6] = {1, 0, 2, 0, 1, 0}, TW[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
        for (int p = 0; p < 6; ++p) {
          const unsigned xt = tmem_base + X_COL + st * X_STAGE + TX[p] * 32;
          const unsigned long long wd = umma_desc(at + TW[p] * F3_PART);
#pragma unroll
          for (int k4 = 0; k4 < F3_BK / 16; ++k4)
            tc_mma_ts(sums, xt + 8 * k4, wd + 2 * k4, IDESC, p + k4 > 0 ? 1u : 0u);
        }
        tc_commit(&bars.done[st]);
      }
      if (!ok && !*abortp) { atomicExch(status, F3_ERR_MMA); *abortp = 1; }
    }
  } else {
    // w: rows r + 32 i, 16-byte chunk c of a tile's row
    const int r = tid >> 3, c = tid & 7;
    const float* ws = w + (size_t)(n0 + r) * K + c * 8;
    const size_t w_down = (size_t)32 * K;
    const int w_left = N - n0 - r;                           // rows from here to the end
    // row r + 32 i keeps r's place in its group of eight, so the swizzle is the same
    unsigned char* at0 = smem + r * 128 + ((c ^ (r & 7)) << 4);
    const int quarter = warp & 3, half = warp >> 2;
    // x: rows xr + 8 i of this warp's 32, four k from xk and from xk + 16 of its 32 k
    const int xr = quarter * 32 + (lane >> 2), xk = half * 32 + (lane & 3) * 4;
    const float* xs = x + (size_t)(m0 + xr) * K + xk;
    const size_t x_down = (size_t)8 * K;
    const int x_left = M - m0 - xr;
    float wv[4][8];
    float4 xv[8];                                            // [2 * (row / 8) + (k / 16)]
    auto fetch_w = [&](int i, int k0) {
      if (k0 + c * 8 < k_end && 32 * i < w_left) {
        f3_load8(ws + i * w_down + k0, wv[i]);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[i][u] = 0.f;
      }
    };
    auto fetch_x = [&](int i, int k0) {
      const int kk = (i & 1) * 16;
      xv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k0 + xk + kk < k_end && 8 * (i >> 1) < x_left)
        xv[i] = *reinterpret_cast<const float4*>(xs + (i >> 1) * x_down + k0 + kk);
    };
    // this thread's part of the result: row `quarter * 32 + lane`, 64 columns
    const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    auto add_up = [&](int st) {
      tc_fence_after();
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 16) {
        float t[16];
        f3_ld16(lane_addr + st * F3_BN + half * 64 + c0, t);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c0 + i] += t[i];
      }
    };
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) fetch_x(i, k_begin);
#pragma unroll
    for (int i = 0; i < 4; ++i) fetch_w(i, k_begin);
    for (int j = 0; j < n_steps; ++j) {
      const int st = j & 1;
      if (j >= 2) {      // the MMAs of step j - 2: their operands are read, their sums stand
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.done[st], ((j >> 1) - 1) & 1, abortp));
        if (!ok) break;
        tc_fence_after();
      }
      // registers are filled for the next step as soon as they are split, so that a load has
      // the whole step to arrive (past the last step it is out of range and reads nothing)
      const int k_next = k_begin + (j + 1) * F3_BK;
      const unsigned xt = lane_addr + X_COL + st * X_STAGE + half * 16;
#pragma unroll
      for (int g = 0; g < 2; ++g) {          // 16 rows
        unsigned t1[8], t2[8], t3[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {        // (row / 8, k / 16)
          const int i = 4 * g + q, at = (q & 1) * 4 + (q >> 1) * 2;
          f3_split2(xv[i].x, xv[i].y, t1[at], t2[at], t3[at]);
          f3_split2(xv[i].z, xv[i].w, t1[at + 1], t2[at + 1], t3[at + 1]);
          fetch_x(i, k_next);
        }
        const unsigned to = xt + ((unsigned)(g * 16) << 16);
        f3_st16x16(to, t1);
        f3_st16x16(to + 32, t2);
        f3_st16x16(to + 64, t3);
      }
      unsigned char* at = at0 + st * F3_STAGE;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f3_split8(wv[i], at + i * 32 * 128);
        fetch_w(i, k_next);
      }
      if (j >= 2) add_up(st);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.full[st]);
    }
    for (int j = max(0, n_steps - 2); ok && j < n_steps; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.done[j & 1], (j >> 1) & 1, abortp));
      if (ok) add_up(j & 1);
    }
    if (!ok) {
      if (lane == 0 && !*abortp) { atomicExch(status, F3_ERR_SPLIT); *abortp = 1; }
    } else {
      const int row = m0 + quarter * 32 + lane, col0 = n0 + half * 64;
      // sums that have to be, again from the operands: a warp per element
#pragma unroll
      for (int i = 0; i < 64; ++i) {
        unsigned bad = __ballot_sync(0xffffffffu, row < M && col0 + i < N && f3_again(acc[i]));
        while (bad) {
          const int l = __ffs(bad) - 1;
          bad &= bad - 1;
          const float* xr_bad = x + (size_t)(m0 + quarter * 32 + l) * K;
          const float* wr_bad = w + (size_t)(col0 + i) * K;
          float s = 0.f;
          for (int k = k_begin + lane; k < k_end; k += 32) s = fmaf(xr_bad[k], wr_bad[k], s);
          s = warp_sum(s);
          if (lane == l) acc[i] = s;
        }
      }
      if (row < M) {
        float* dst = (part ? part + (size_t)blockIdx.z * M * N : out) + (size_t)row * N + col0;
        if (!part) {
#pragma unroll
          for (int i = 0; i < 64; ++i) acc[i] = ix_act<float>(acc[i], act);
        }
        if (col0 + 64 <= N && N % 4 == 0) {
#pragma unroll
          for (int i = 0; i < 64; i += 4)
            *reinterpret_cast<float4*>(dst + i) =
                make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (col0 + i < N) dst[i] = acc[i];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == F3_WARPS) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  }
}

// The runs' partial sums, in ascending order.
__global__ void gemm_fp32_tc_sum_kernel(const float* __restrict__ part, float* __restrict__ out,
                                        long long n, int splits, int act) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float s = part[i];
    for (int z = 1; z < splits; ++z) s += part[(long long)z * n + i];
    out[i] = ix_act<float>(s, act);
  }
}

// Runs to cut k into: the number for which waves x steps of a block, and what the partial sums
// cost to write and read, is least.  A step is some 1.6 us; partial sums 0.35 us a MB both ways,
// their kernel's launch 3 us (M 600, N 2048, K 5632: 3 runs 120 us, one 145; M 64, N 11264,
// K 2048: one run 60 us, 3 runs 70; M 64, N 2048, K 5632: 9 runs 35.5 us, one 140).  Runs are 4
// steps at least on average; the last may be shorter.  A row's last bits follow the number of runs,
// and so the number of rows.
IX_API int ix_gemm_fp32_tc_splits(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 1;
  const long long tiles = ((M + F3_BM - 1) / F3_BM) * (long long)((N + F3_BN - 1) / F3_BN);
  const int steps = (K + F3_BK - 1) / F3_BK;
  int best = 1;
  double best_us = 1e30;
  for (int s = 1; s <= 16 && steps / s >= 4; ++s) {
    const int per = (steps + s - 1) / s;
    if ((long long)per * (s - 1) >= steps) continue;       // an empty last run
    const double waves = (double)((tiles * s + 147) / 148);
    const double us = waves * (per * 1.6 + 3.0) +
                      (s > 1 ? 3.0 + 0.35 * s * (double)M * N * 4e-6 : 0.0);
    if (us < 0.97 * best_us) { best_us = us; best = s; }
  }
  return best;
}

// x: [M, K], w: [N, K], out: [M, N], all fp32.  splits > 1: part [splits, M, N] fp32 scratch.
IX_API int ix_gemm_fp32_tc(const float* x, const float* w, float* out, float* part, int M, int N,
                           int K, int splits, int act, int* status, cudaStream_t stream) {
  if (M <= 0) return IX_OK;
  if (N <= 0 || K <= 0 || splits < 1 || splits > 16 || status == nullptr || (splits > 1 && !part))
    return IX_ERR_SIZE;
  if (K % 8) return IX_ERR_UNSUPPORTED;
  if ((((uintptr_t)x | (uintptr_t)w) & 31) || (((uintptr_t)out | (uintptr_t)part) & 15))
    return IX_ERR_ALIGN;
  const int steps = (K + F3_BK - 1) / F3_BK;
  const int per = (steps + splits - 1) / splits;
  if ((long long)per * (splits - 1) >= steps) return IX_ERR_SIZE;
  const long long gy = (N + F3_BN - 1) / F3_BN;
  if (gy > 65535) return IX_ERR_SIZE;
  const int smem = 2 * F3_STAGE + 1024;
  // one block an SM: a second one could not have tensor memory (smem is under half of an SM's)
  const int ask = smem < 120 * 1024 ? 120 * 1024 : smem;
  cudaError_t e = cudaFuncSetAttribute(gemm_fp32_tc_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, ask);
  if (e != cudaSuccess) return (int)e;
  gemm_fp32_tc_kernel<<<dim3((M + F3_BM - 1) / F3_BM, (unsigned)gy, splits), F3_THREADS, ask,
                        stream>>>(x, w, out, splits > 1 ? part : nullptr, M, N, K, per, act,
                                  status);
  int rc = ix_launch_status();
  if (rc != IX_OK || splits == 1) return rc;
  const long long n = (long long)M * N;
  const long long blocks = (n + 255) / 256;
  gemm_fp32_tc_sum_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream>>>(
      part, out, n, splits, act);
  return ix_launch_status();
}

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
// Two SMs make 256 features of up to 160 rows (cta_group::2): a block holds 128 rows of w, the M
// side, and half of the rows of x, the N side.  Warps 0-15 read the next 64 entries of k of both
// into registers (a step ahead), split them into the three terms and write those as swizzled tiles
// in shared memory (two stages), and add up the accumulators of the step before the last; the first
// block's last warp issues the 24 MMAs of a step for both.  A row of w is split for 160 rows of x and
// a row of x for 256 of w, where a block on its own split either for 128.  What bounds a step is the
// splitting warps' chain of loads, splits, writes and sums: 1.5 us up to 96 rows, 1.65 at 128, 1.9 at
// 160 (all pairs busy, K 4,096 to 16,384), with the tensor pipe 44 % busy and 1.4 instructions a cycle
// of 4 at 600 rows of 11264 x 2048.  Against a block on its own: 600 rows of 11264 x 2048 176 us, was
// 186; of 2048 x 5632 98, was 127; 800 rows of 22016 x 4096 788, was 1,019; 40 rows of 11264 x 2048 49,
// was 74.  It is slower where one wave of blocks of 128 x 128 filled the device: 800 rows of 2048 x
// 5632 140 us, was 125, 1,000 rows 146 and 134, 2,048 rows of 1024 x 2816 84 and 78.  Operands brought
// as they are into shared memory by TMA, a step ahead, were slower too (194 us for the first).  The
// terms are made in the kernel, and not by a pass of their own: the weights' terms would be 1.5 times
// the weights, written and read again.
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

#include "bf16_terms.cuh"
#include "common.cuh"
#include "tma_common.cuh"
#include "tcgen05_common.cuh"

#define F3_BF 128                                 // features of a block (two blocks a tile)
#define F3_MAX_ROWS 160                           // rows of a tile
#define F3_BK 64
#define F3_WARPS 16                               // that split and add up; one more issues MMAs
#define F3_THREADS (F3_WARPS * 32 + 32)
#define F3_PART (F3_BF * F3_BK * 2)               // one term of w: 16 KB

enum { F3_ERR_SPLIT = 41, F3_ERR_MMA = 42 };

struct F3Bars {
  unsigned long long ready[2], full[2], done[2];
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
// eight columns of this thread's lane
__device__ __forceinline__ void f3_ld8(unsigned taddr, float* v) {
  unsigned r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// Of eight numbers, 16 bytes each, into the same place of three tiles PART bytes apart.
template <int PART>
__device__ __forceinline__ void f3_split8(const float* v, unsigned char* at) {
  unsigned t1[4], t2[4], t3[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) bf16_terms2(v[2 * i], v[2 * i + 1], t1[i], t2[i], t3[i]);
  *reinterpret_cast<uint4*>(at) = make_uint4(t1[0], t1[1], t1[2], t1[3]);
  *reinterpret_cast<uint4*>(at + PART) = make_uint4(t2[0], t2[1], t2[2], t2[3]);
  *reinterpret_cast<uint4*>(at + 2 * PART) = make_uint4(t3[0], t3[1], t3[2], t3[3]);
}

// Whether a sum has to be made again: not finite, or so small that operands without a third term
// may have gone into it.
__device__ __forceinline__ bool f3_again(float s) {
  const float a = fabsf(s);
  return !(a <= FLT_MAX) || (a < 5.421010862427522e-20f && a > 0.f);
}

// ROWS: rows of x that the tile has room for; `rows` (a multiple of 32, at most ROWS) are used.
template <int ROWS>
__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_fp32_tc_kernel(const float* __restrict__ x, const float* __restrict__ w,
                    float* __restrict__ out, float* __restrict__ part, int M, int N, int K,
                    int rows, int steps_per_split, int act, int* __restrict__ status) {
  constexpr int X_PART = ROWS / 2 * F3_BK * 2, STAGE = 3 * (F3_PART + X_PART);
  constexpr int COLS = ROWS / 4;                    // rows of the tile a warp adds up
  constexpr unsigned TMEM_COLS = 2 * ROWS <= 128 ? 128 : 2 * ROWS <= 256 ? 256 : 512;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) F3Bars bars;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // neighbouring pairs share a tile of weights
  const int rank = (int)tc_rank();
  const int m0 = (blockIdx.x >> 1) * rows, n0 = (blockIdx.y * 2 + rank) * F3_BF;
  const int k_begin = blockIdx.z * steps_per_split * F3_BK;
  const int k_end = min(K, k_begin + steps_per_split * F3_BK);
  const int n_steps = (k_end - k_begin + F3_BK - 1) / F3_BK;      // at least 1

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.ready[i], F3_WARPS);            // a block's own tiles are written
      mbar_init(&bars.full[i], 2);                    // both blocks' are (the first block's is used)
      mbar_init(&bars.done[i], 1);
    }
    bars.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == F3_WARPS) tc_alloc<true>(&bars.tmem_holder, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_cluster_sync();
  tc_fence_after();
  const unsigned tmem_base = __shfl_sync(0xffffffffu, bars.tmem_holder, 0);
  volatile int* abortp = &bars.abort_flag;

  if (warp == F3_WARPS) {
    // The whole warp walks the steps and one lane issues: descriptors that are the warp's and not
    // a thread's stay in uniform registers (one lane on its own takes some 130 cycles an MMA).
    // A block's tiles are reported to the first block by this warp, which waits for its own block's
    // warps: sixteen arrivals a step at the other block's barrier would be as many releases for the
    // cluster.
    const unsigned full = tc_of_rank(&bars.full[0], 0);
    if (rank == 1) {
      bool ok = true;
      for (int j = 0; j < n_steps; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.ready[j & 1], (j >> 1) & 1, abortp));
        if (!ok) break;
        if (lane == 0) tc_arrive_at(full + (j & 1) * 8);
        __syncwarp();
      }
      if (!ok && lane == 0 && !*abortp) { atomicExch(status, F3_ERR_MMA); *abortp = 1; }
    } else {
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(rows >> 3) << 17) |
                             ((unsigned)(2 * F3_BF >> 4) << 24);
      bool ok = true;
      for (int j = 0; j < n_steps; ++j) {
        const int st = j & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.ready[st], (j >> 1) & 1, abortp));
        if (!ok) break;
        if (lane == 0) mbar_arrive(&bars.full[st]);
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.full[st], (j >> 1) & 1, abortp));
        if (!ok) break;
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        tc_fence_after();
        unsigned char* at = smem + st * STAGE;
        const unsigned sums = tmem_base + st * ROWS;
        // (term of x, term of w)
        constexpr int TX[6] = {1, 0, 2, 0, 1, 0}, TW[6] = {1, 2, 0, 1, 0, 0};
        if (lane == 0) {
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const unsigned long long wd = umma_desc(at + TW[p] * F3_PART);
            const unsigned long long xd = umma_desc(at + 3 * F3_PART + TX[p] * X_PART);
#pragma unroll
            for (int k4 = 0; k4 < F3_BK / 16; ++k4)
              tc_mma_pair(sums, wd + 2 * k4, xd + 2 * k4, idesc, p + k4 > 0 ? 1u : 0u);
          }
          tc_commit_pair(&bars.done[st]);
        }
        __syncwarp();
      }
      if (!ok && lane == 0 && !*abortp) { atomicExch(status, F3_ERR_MMA); *abortp = 1; }
    }
  } else {
    // rows r + 64 i of the block's tiles, 16-byte chunk c of a tile's row
    constexpr int XI = (ROWS / 2 + 63) / 64;
    const int r = tid >> 3, c = tid & 7;
    const int x0 = m0 + rank * (rows / 2);                   // this block's half of x's rows
    const float* ws = w + (size_t)(n0 + r) * K + c * 8;
    const float* xs = x + (size_t)(x0 + r) * K + c * 8;
    const size_t down = (size_t)64 * K;
    const int w_left = N - n0 - r;                           // rows from here to the end
    const int x_left = min(rows / 2, M - x0) - r;
    // row r + 64 i keeps r's place in its group of eight, so the swizzle is the same
    unsigned char* at0 = smem + r * 128 + ((c ^ (r & 7)) << 4);
    const int quarter = warp & 3, col0 = (warp >> 2) * COLS;
    float wv[2][8], xv[XI][8];
    auto fetch_w = [&](int i, int k0) {
      if (k0 + c * 8 < k_end && 64 * i < w_left) {
        f3_load8(ws + i * down + k0, wv[i]);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[i][u] = 0.f;
      }
    };
    auto fetch_x = [&](int i, int k0) {
      if (k0 + c * 8 < k_end && 64 * i < x_left) {
        f3_load8(xs + i * down + k0, xv[i]);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) xv[i][u] = 0.f;
      }
    };
    // this thread's part of the result: feature `quarter * 32 + lane`, COLS rows
    const unsigned sums_addr = tmem_base + ((unsigned)(quarter * 32) << 16) + col0;
    float acc[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
    auto add_up = [&](int st) {
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < COLS; q += 8) {        // more at a time would cost registers that spill
        float t[8];
        f3_ld8(sums_addr + st * ROWS + q, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[q + i] += t[i];
      }
    };
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 2; ++i) fetch_w(i, k_begin);
#pragma unroll
    for (int i = 0; i < XI; ++i) fetch_x(i, k_begin);
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
      unsigned char* at = at0 + st * STAGE;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        f3_split8<F3_PART>(wv[i], at + i * 64 * 128);
        fetch_w(i, k_next);
      }
#pragma unroll
      for (int i = 0; i < XI; ++i)
        if (r + 64 * i < ROWS / 2) {
          f3_split8<X_PART>(xv[i], at + 3 * F3_PART + i * 64 * 128);
          fetch_x(i, k_next);
        }
      if (j >= 2) add_up(st);
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.ready[st]);
    }
    for (int j = max(0, n_steps - 2); ok && j < n_steps; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.done[j & 1], (j >> 1) & 1, abortp));
      if (ok) add_up(j & 1);
    }
    if (!ok) {
      if (lane == 0 && !*abortp) { atomicExch(status, F3_ERR_SPLIT); *abortp = 1; }
    } else {
      const int f = n0 + quarter * 32 + lane, row0 = m0 + col0;
      const int there = min(rows - col0, M - row0);          // rows of this warp's that exist
      // sums that have to be, again from the operands: a warp per element
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        unsigned bad = __ballot_sync(0xffffffffu, i < there && f < N && f3_again(acc[i]));
        while (bad) {
          const int l = __ffs(bad) - 1;
          bad &= bad - 1;
          const float* xr_bad = x + (size_t)(row0 + i) * K;
          const float* wr_bad = w + (size_t)(n0 + quarter * 32 + l) * K;
          float s = 0.f;
          for (int k = k_begin + lane; k < k_end; k += 32) s = fmaf(xr_bad[k], wr_bad[k], s);
          s = warp_sum(s);
          if (lane == l) acc[i] = s;
        }
      }
      if (f < N) {         // a warp's threads hold neighbouring features of a row
        float* dst = (part ? part + (size_t)blockIdx.z * M * N : out) + (size_t)row0 * N + f;
#pragma unroll
        for (int i = 0; i < COLS; ++i)
          if (i < there) dst[(size_t)i * N] = part ? acc[i] : ix_act<float>(acc[i], act);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // neither block ends while the other can still reach its barriers, tiles or accumulators
  tc_cluster_sync();
  if (warp == F3_WARPS) tc_dealloc<true>(tmem_base, TMEM_COLS);
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

// Microseconds of a call in `splits` runs of k with tiles of `rows` rows: waves of pairs of blocks, a
// step of which counts 0.75 us and 8.1 ns a row (1.3 us at 64 rows, 1.8 at 128, 2.05 at 160, a steeper
// line than the steps' own times above), and what partial sums cost to write and read, 0.35 us a MB both
// ways and 3 us for their kernel's launch.  Of 32 products of 400 to 3,000 rows, each timed in 1 to 6
// runs, the number that this chooses was the fastest or within 6 % of it.
static double f3_cost(int M, int N, int K, int rows, int splits) {
  const int steps = (K + F3_BK - 1) / F3_BK, per = (steps + splits - 1) / splits;
  const long long tiles = ((M + rows - 1) / rows) * (long long)((N + 2 * F3_BF - 1) / (2 * F3_BF));
  const double waves = (double)((tiles * splits + 73) / 74);
  return waves * (per * (0.75 + 0.0081 * rows) + 4.0) +
         (splits > 1 ? 3.0 + 0.35 * splits * (double)M * N * 4e-6 : 0.0);
}

// Rows of a tile (a multiple of 32, at most F3_MAX_ROWS): those for which the call takes least.  Wide
// tiles do most per step, narrower ones fill a last wave (600 rows of 11264 x 2048: four tiles of
// 160 200 us, five of 128 176).
static int f3_tile_rows(int M, int N, int K, int splits) {
  int best = F3_MAX_ROWS;
  double best_us = 1e30;
  for (int rows = F3_MAX_ROWS; rows >= 32; rows -= 32) {
    const int tiles = (M + rows - 1) / rows;
    const int even = ((M + tiles - 1) / tiles + 31) / 32 * 32;
    const double us = f3_cost(M, N, K, even, splits);
    if (us < 0.99 * best_us) { best_us = us; best = even; }
  }
  return best;
}

// Runs to cut k into: the number for which the call takes least.  Runs are 4 steps at least on
// average; the last may be shorter.  A row's last bits follow the number of runs, and so the number
// of rows.
IX_API int ix_gemm_fp32_tc_splits(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 1;
  const int steps = (K + F3_BK - 1) / F3_BK;
  int best = 1;
  double best_us = 1e30;
  for (int s = 1; s <= 16 && steps / s >= 4; ++s) {
    const int per = (steps + s - 1) / s;
    if ((long long)per * (s - 1) >= steps) continue;       // an empty last run
    const double us = f3_cost(M, N, K, f3_tile_rows(M, N, K, s), s);
    if (us < 0.97 * best_us) { best_us = us; best = s; }
  }
  return best;
}

template <int ROWS>
static int f3_launch(const float* x, const float* w, float* out, float* part, int M, int N, int K,
                     int rows, int per, int splits, int act, int* status, cudaStream_t stream) {
  int smem = 2 * 3 * (F3_PART + ROWS / 2 * F3_BK * 2) + 1024;
  // one block an SM: a second one could not have tensor memory
  if (smem < 120 * 1024) smem = 120 * 1024;
  auto kern = gemm_fp32_tc_kernel<ROWS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * ((M + rows - 1) / rows), (N + 2 * F3_BF - 1) / (2 * F3_BF), splits);
  cfg.blockDim = dim3(F3_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, x, w, out, part, M, N, K, rows, per, act, status);
  return ix_launch_status();
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
  if ((N + F3_BF - 1LL) / F3_BF > 65535) return IX_ERR_SIZE;
  const int rows = f3_tile_rows(M, N, K, splits);
  auto go = rows <= 64 ? f3_launch<64> : rows <= 128 ? f3_launch<128> : f3_launch<160>;
  const int rc = go(x, w, out, splits > 1 ? part : nullptr, M, N, K, rows, per, splits, act, status,
                    stream);
  if (rc != IX_OK || splits == 1) return rc;
  const long long n = (long long)M * N;
  const long long blocks = (n + 255) / 256;
  gemm_fp32_tc_sum_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream>>>(
      part, out, n, splits, act);
  return ix_launch_status();
}

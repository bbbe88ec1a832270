// The state-space recurrence of delta_parts.cu over portions of prompts, in chunks on the tensor
// cores (bfloat16 x, B, C; scalar decay per head):
//
//   S_t = exp(-exp(A) dt_t) S_(t-1) + dt_t B_t x_t^T,    y_t = S_t^T C_t + D x_t
//
// Inside a chunk of 64 tokens, with G_t the sum of the log decays up to and with token t:
//
//   y_t   = exp(G_t) S_start^T C_t + sum_(s <= t) exp(G_t - G_s) dt_s (C_t . B_s) x_s + D x_t
//   S_end = exp(G_end) S_start + sum_s exp(G_end - G_s) dt_s B_s x_s^T
//
// Three passes: own (every chunk's sum into S_end, to scratch), join (per entry of the state, along
// a sequence's chunks: the scratch entry becomes the chunk's start state), out (every token's y).
// The walk takes a token's 3 K V multiply-adds a head one token after the other, and its segments
// side by side are bound by the FFMA and shared-memory rate (2,048 tokens, 32 heads of 128 x 64:
// 144 + 311 us for its two passes, 92 us for these three).  Chunks do the same sums as products.
// What bounds them is how few warps an SM holds (8 in out, by shared memory) between stages that
// wait for one another: tensor pipe 16 %, L2 at 9 to 26 % with the chunks' states (K V fp32 a head,
// written twice and read twice).
//
// Nothing of 32 bits is narrowed: x, B and C enter the products as they are (bfloat16), and what is
// fp32 (weighted inputs, weighted scores, start states) as three bfloat16 terms, 24 bits, small
// terms first into fp32 accumulators.  The tensor cores do not round those sums to nearest, so sums
// over the state's entries are taken 64 at a time and added in fp32.  G is summed in 64 bits,
// because exp(G_t - G_s) of close tokens far down a chunk would lose the bits that their difference
// cancels.
//
// Products take numbers: a later token's weight of 0 times an infinite x is not a number, nor is
// the second term of an infinite one.  So a block whose results are not all finite makes them again
// token by token (walk_column): tokens ahead of an infinity keep their results, and what is
// infinite in the walk is infinite here.
//
// Requires K and V multiples of 8, K at most 256, rows on 16-byte marks.
#include "bf16_terms.cuh"
#include "common.cuh"

#define SC_L 64               // tokens a chunk
#define SC_VT 64              // value columns a block
#define SC_THREADS 128
#define SC_MAX_K 256

__device__ __forceinline__ unsigned sc_smem(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void sc_ldm4(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void sc_ldm4t(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void sc_mma(float* c, const unsigned* a, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void sc_async16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sc_smem(dst)), "l"(src),
               "r"(bytes) : "memory");
}
__device__ __forceinline__ void sc_async_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
// `rows` of SC_L rows and `cols` of `padded` columns into shared rows of `pitch`, the rest zero
__device__ __forceinline__ void sc_load(bf16* dst, int pitch, const bf16* src, long long ld,
                                        int rows, int cols, int padded) {
  const int per = padded >> 3;
  for (int i = threadIdx.x; i < SC_L * per; i += SC_THREADS) {
    const int r = i / per, c = (i - r * per) * 8;
    const bool ok = r < rows && c < cols;
    sc_async16(dst + r * pitch + c, ok ? src + (size_t)r * ld + c : src, ok ? 16 : 0);
  }
}

struct ScIn {
  const bf16* xbc;            // rows x | B | C
  long long ld;
  const bf16* dt_raw;
  long long ld_dt;
  const float *dt_bias, *a_log, *d_skip;
  const int* cu_q;
  int H, V, K, G, s0;
};
struct ScWhere {              // a block's chunk
  int t0, n, entry;           // first token of the step, tokens, scratch number
};
// A chunk's number is tokens before the sequence / 64 + the sequence's number + the chunk's: no
// two meet.
__device__ __forceinline__ ScWhere sc_where(const int* cu_q, int s, int s0, int chunk) {
  const int begin = cu_q[s], end = cu_q[s + 1], base = cu_q[s0];
  ScWhere w;
  w.t0 = begin + chunk * SC_L;
  w.n = min(SC_L, end - w.t0);
  w.entry = (begin - base) / SC_L + (s - s0) + chunk;
  return w;
}
__device__ __forceinline__ float sc_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// G and dt of the chunk's tokens by one warp; tokens past the end: G of the last, dt 0.
__device__ __forceinline__ void sc_gates(double* G, float* dt, const ScIn& in, int h, int t0,
                                         int n) {
  const int lane = threadIdx.x & 31;
  const float neg_a = -expf(in.a_log[h]), bias = in.dt_bias[h];
  double carry = 0.0;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int t = half * 32 + lane;
    float d = 0.f;
    double g = 0.0;
    if (t < n) {
      d = sc_softplus(__bfloat162float(in.dt_raw[(size_t)(t0 + t) * in.ld_dt + h]) + bias);
      g = (double)neg_a * (double)d;
      if (g < -1e6) g = -1e6;    // a decay of 0 either way; differences of sums stay numbers
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double p = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) g += p;
    }
    g += carry;
    carry = __shfl_sync(0xffffffffu, g, 31);
    G[t] = g;
    dt[t] = d;
  }
}

// One value column of the chunk token by token, with the walk's operations: S, the column's state
// with `pitch` floats from entry to entry, becomes the state behind the chunk; `y` (null: none)
// takes the tokens' outputs, y_pitch floats apart.
__device__ __noinline__ void walk_column(float a_log, float dsk, const float* dt, int n, int K,
                                         int pk, const bf16* b_s, const bf16* c_s, const bf16* x,
                                         long long ld, float* S, int pitch, float* y,
                                         size_t y_pitch) {
  const float neg_a = -expf(a_log);
  for (int t = 0; t < n; ++t) {
    const float d = dt[t], a = expf(neg_a * d), xv = __bfloat162float(x[(size_t)t * ld]);
    float acc = 0.f;
    for (int k = 0; k < K; ++k) {
      const float kk = __fmul_rn(d, __bfloat162float(b_s[t * pk + k]));
      const float s = __fmaf_rn(a, S[(size_t)k * pitch], __fmul_rn(kk, xv));
      S[(size_t)k * pitch] = s;
      if (y) acc = __fmaf_rn(s, __bfloat162float(c_s[t * pk + k]), acc);
    }
    if (y) y[t * y_pitch] = __fmaf_rn(dsk, xv, acc);
  }
}

// ---------------------------------------------------------------------------
// own: grid (value tiles, chunks, heads * sequences)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SC_THREADS)
ssd_chunk_own_kernel(ScIn in, float* __restrict__ scr_s, float* __restrict__ scr_p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double G[SC_L];
  __shared__ float dt[SC_L];
  const int K = in.K, V = in.V, Kp = (K + 15) & ~15, pk = Kp + 8;
  constexpr int pv = SC_VT + 8;
  bf16* b_s = reinterpret_cast<bf16*>(smem_raw);        // [SC_L][pk]
  bf16* x_s = b_s + SC_L * pk;                          // three terms of [SC_L][pv]
  const int h = blockIdx.z % in.H, s = in.s0 + blockIdx.z / in.H, v0 = blockIdx.x * SC_VT;
  const ScWhere at = sc_where(in.cu_q, s, in.s0, blockIdx.y);
  if (at.n <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bf16* row = in.xbc + (size_t)at.t0 * in.ld;
  sc_load(b_s, pk, row + (size_t)in.H * V + (size_t)(h / (in.H / in.G)) * K, in.ld, at.n, K, Kp);
  sc_load(x_s, pv, row + (size_t)h * V + v0, in.ld, at.n, min(SC_VT, V - v0), SC_VT);
  if (warp == 0) sc_gates(G, dt, in, h, at.t0, at.n);
  sc_async_wait();
  __syncthreads();
  const double g_end = G[SC_L - 1];
  for (int i = tid; i < SC_L * (SC_VT / 2); i += SC_THREADS) {
    const int t = i / (SC_VT / 2), c = (i % (SC_VT / 2)) * 2;
    const float w = expf((float)(g_end - G[t])) * dt[t];
    const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(x_s + t * pv + c);
    unsigned terms[3];
    bf16_terms2(__low2float(x) * w, __high2float(x) * w, terms[0], terms[1], terms[2]);
#pragma unroll
    for (int u = 0; u < 3; ++u)
      *reinterpret_cast<unsigned*>(x_s + (u * SC_L + t) * pv + c) = terms[u];
  }
  __syncthreads();
  const size_t cell = (size_t)at.entry * in.H + h;
  if (blockIdx.x == 0 && tid == 0) scr_p[cell] = expf((float)g_end);
  float* out = scr_s + cell * K * V;
  bool bad = false;
  for (int mt = warp; mt < Kp >> 4; mt += SC_THREADS / 32) {
    float acc[SC_VT / 8][4];
#pragma unroll
    for (int j = 0; j < SC_VT / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    const int steps = (at.n + 15) >> 4;
    for (int u = 2; u >= 0; --u) {
      for (int kk = 0; kk < steps; ++kk) {
        unsigned a[4];
        sc_ldm4t(a, sc_smem(b_s + (kk * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * pk + mt * 16 +
                            ((lane >> 3) & 1) * 8));
        const int brow = u * SC_L + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int j = 0; j < SC_VT / 8; j += 2) {
          unsigned b[4];
          sc_ldm4t(b, sc_smem(x_s + brow * pv + j * 8 + ((lane >> 4) & 1) * 8));
          sc_mma(acc[j], a, b[0], b[1]);
          sc_mma(acc[j + 1], a, b[2], b[3]);
        }
      }
    }
    const int r = mt * 16 + (lane >> 2), t2 = (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < SC_VT / 8; ++j) {
      const int c = v0 + j * 8 + t2;
#pragma unroll
      for (int e = 0; e < 4; ++e) bad |= !isfinite(acc[j][e]);
      if (c >= V) continue;
      float* at_r = out + (size_t)r * V + c;
      if (r < K) *reinterpret_cast<float2*>(at_r) = make_float2(acc[j][0], acc[j][1]);
      if (r + 8 < K)
        *reinterpret_cast<float2*>(at_r + (size_t)8 * V) = make_float2(acc[j][2], acc[j][3]);
    }
  }
  if (__syncthreads_or(bad) && tid < SC_VT && v0 + tid < V) {
    float* S = out + v0 + tid;
    for (int k = 0; k < K; ++k) S[(size_t)k * V] = 0.f;
    walk_column(in.a_log[h], 0.f, dt, at.n, K, pk, b_s, nullptr, row + (size_t)h * V + v0 + tid,
                in.ld, S, V, nullptr, 0);
  }
}

// ---------------------------------------------------------------------------
// join: grid (groups of entries, heads, sequences); a thread owns four neighbouring entries of the
// state along the sequence's chunks, eight of which it fetches at a time
// ---------------------------------------------------------------------------
#define SJ_THREADS 128
#define SJ_AHEAD 8

__global__ void __launch_bounds__(SJ_THREADS)
ssd_chunk_join_kernel(float* __restrict__ scr_s, const float* __restrict__ scr_p,
                      float* __restrict__ state, const int* __restrict__ cu_q,
                      const int* __restrict__ state_slot, int H, int KV, int s0) {
  const int h = blockIdx.y, s = s0 + blockIdx.z;
  const int n = cu_q[s + 1] - cu_q[s];
  const int i = blockIdx.x * SJ_THREADS + threadIdx.x;
  if (n <= 0 || i * 4 >= KV) return;
  const ScWhere first = sc_where(cu_q, s, s0, 0);
  const int chunks = (n + SC_L - 1) / SC_L;
  float4* st = reinterpret_cast<float4*>(state + ((size_t)state_slot[s] * H + h) * KV) + i;
  float4 x = *st;
  for (int c0 = 0; c0 < chunks; c0 += SJ_AHEAD) {
    float4 own[SJ_AHEAD];
    float p[SJ_AHEAD];
#pragma unroll
    for (int j = 0; j < SJ_AHEAD; ++j)
      if (c0 + j < chunks) {
        const size_t cell = (size_t)(first.entry + c0 + j) * H + h;
        own[j] = reinterpret_cast<const float4*>(scr_s + cell * KV)[i];
        p[j] = scr_p[cell];
      }
#pragma unroll
    for (int j = 0; j < SJ_AHEAD; ++j)
      if (c0 + j < chunks) {
        const size_t cell = (size_t)(first.entry + c0 + j) * H + h;
        reinterpret_cast<float4*>(scr_s + cell * KV)[i] = x;
        x.x = fmaf(p[j], x.x, own[j].x);
        x.y = fmaf(p[j], x.y, own[j].y);
        x.z = fmaf(p[j], x.z, own[j].z);
        x.w = fmaf(p[j], x.w, own[j].w);
      }
  }
  *st = x;
}

// ---------------------------------------------------------------------------
// out: grid (value tiles, chunks, heads * sequences); warp w owns the chunk's tokens 16 w .. + 15
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SC_THREADS)
ssd_chunk_out_kernel(ScIn in, const float* __restrict__ scr_s, float* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double G[SC_L];
  __shared__ float dt[SC_L];
  const int K = in.K, V = in.V, Kp = (K + 15) & ~15, pk = Kp + 8;
  constexpr int pv = SC_VT + 8;
  bf16* c_s = reinterpret_cast<bf16*>(smem_raw);        // [SC_L][pk]
  bf16* b_s = c_s + SC_L * pk;                          // [SC_L][pk]
  bf16* x_s = b_s + SC_L * pk;                          // [SC_L][pv]
  bf16* s_s = x_s + SC_L * pv;                          // three terms of [Kp][pv]
  const int h = blockIdx.z % in.H, s = in.s0 + blockIdx.z / in.H, v0 = blockIdx.x * SC_VT;
  const ScWhere at = sc_where(in.cu_q, s, in.s0, blockIdx.y);
  if (at.n <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bf16* row = in.xbc + (size_t)at.t0 * in.ld;
  const bf16* b_row = row + (size_t)in.H * V + (size_t)(h / (in.H / in.G)) * K;
  sc_load(b_s, pk, b_row, in.ld, at.n, K, Kp);
  sc_load(c_s, pk, b_row + (size_t)in.G * K, in.ld, at.n, K, Kp);
  sc_load(x_s, pv, row + (size_t)h * V + v0, in.ld, at.n, min(SC_VT, V - v0), SC_VT);
  const float* start = scr_s + ((size_t)at.entry * in.H + h) * K * V;
  for (int i = tid; i < Kp * (SC_VT / 4); i += SC_THREADS) {
    const int r = i / (SC_VT / 4), c = (i % (SC_VT / 4)) * 4;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < K && v0 + c < V) f = *reinterpret_cast<const float4*>(start + (size_t)r * V + v0 + c);
    unsigned t01[3], t23[3];
    bf16_terms2(f.x, f.y, t01[0], t01[1], t01[2]);
    bf16_terms2(f.z, f.w, t23[0], t23[1], t23[2]);
#pragma unroll
    for (int u = 0; u < 3; ++u)
      *reinterpret_cast<uint2*>(s_s + ((size_t)u * Kp + r) * pv + c) = make_uint2(t01[u], t23[u]);
  }
  if (warp == 0) sc_gates(G, dt, in, h, at.t0, at.n);
  sc_async_wait();
  __syncthreads();
  bool bad = false;
  if (warp * 16 < at.n) {
    const int t2 = (lane & 3) * 2;
    const int ra = warp * 16 + (lane >> 2), rb = ra + 8;  // this thread's two tokens
    float p[8][4], o[SC_VT / 8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) p[j][e] = 0.f;
#pragma unroll
    for (int j = 0; j < SC_VT / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    const int arow = warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, acol = (lane >> 4) * 8;
    // scores of the warp's tokens against the chunk's tokens up to them
    const int k_steps = Kp >> 4;
    for (int k0 = 0; k0 < k_steps; k0 += 4) {
      float t[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) t[j][e] = 0.f;
      for (int kk = k0; kk < min(k0 + 4, k_steps); ++kk) {
        unsigned a[4];
        sc_ldm4(a, sc_smem(c_s + arow * pk + kk * 16 + acol));
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          if (j <= 2 * warp + 1) {
            unsigned b[4];
            sc_ldm4(b, sc_smem(b_s + (j * 8 + (lane & 7) + ((lane >> 4) & 1) * 8) * pk + kk * 16 +
                               ((lane >> 3) & 1) * 8));
            sc_mma(t[j], a, b[0], b[1]);
            sc_mma(t[j + 1], a, b[2], b[3]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) p[j][e] += t[j][e];
    }
    // the start state's part
    for (int u = 2; u >= 0; --u) {
      for (int k0 = 0; k0 < k_steps; k0 += 4) {
        float t[SC_VT / 8][4];
#pragma unroll
        for (int j = 0; j < SC_VT / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) t[j][e] = 0.f;
        for (int kk = k0; kk < min(k0 + 4, k_steps); ++kk) {
          unsigned a[4];
          sc_ldm4(a, sc_smem(c_s + arow * pk + kk * 16 + acol));
          const int brow = u * Kp + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
          for (int j = 0; j < SC_VT / 8; j += 2) {
            unsigned b[4];
            sc_ldm4t(b, sc_smem(s_s + (size_t)brow * pv + j * 8 + ((lane >> 4) & 1) * 8));
            sc_mma(t[j], a, b[0], b[1]);
            sc_mma(t[j + 1], a, b[2], b[3]);
          }
        }
#pragma unroll
        for (int j = 0; j < SC_VT / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[j][e] += t[j][e];
      }
    }
    const double Ga = G[ra], Gb = G[rb];
    const float ea = expf((float)Ga), eb = expf((float)Gb);
#pragma unroll
    for (int j = 0; j < SC_VT / 8; ++j) {
      o[j][0] *= ea; o[j][1] *= ea;
      o[j][2] *= eb; o[j][3] *= eb;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = j * 8 + t2 + e;
        const double Gc = G[c];
        const float d = dt[c];
        p[j][e] = c <= ra ? p[j][e] * (expf((float)(Ga - Gc)) * d) : 0.f;
        p[j][2 + e] = c <= rb ? p[j][2 + e] * (expf((float)(Gb - Gc)) * d) : 0.f;
      }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk > warp) break;
      unsigned a[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {          // (row half, column half) of the fragment
        unsigned t[3];
        const float* f = p[2 * kk + (e >> 1)] + (e & 1) * 2;
        bf16_terms2(f[0], f[1], t[0], t[1], t[2]);
        a[0][e] = t[0]; a[1][e] = t[1]; a[2][e] = t[2];
      }
      const int brow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int j = 0; j < SC_VT / 8; j += 2) {
        unsigned b[4];
        sc_ldm4t(b, sc_smem(x_s + brow * pv + j * 8 + ((lane >> 4) & 1) * 8));
#pragma unroll
        for (int u = 2; u >= 0; --u) {
          sc_mma(o[j], a[u], b[0], b[1]);
          sc_mma(o[j + 1], a[u], b[2], b[3]);
        }
      }
    }
    const float dsk = in.d_skip[h];
    float* ya = y + ((size_t)(at.t0 + ra) * in.H + h) * V;
    float* yb = y + ((size_t)(at.t0 + rb) * in.H + h) * V;
#pragma unroll
    for (int j = 0; j < SC_VT / 8; ++j) {
      const int c = v0 + j * 8 + t2;
      bad |= (ra < at.n && !(isfinite(o[j][0]) && isfinite(o[j][1]))) ||
             (rb < at.n && !(isfinite(o[j][2]) && isfinite(o[j][3])));
      if (c >= V) continue;
      const bf16* x_at = x_s + ra * pv + j * 8 + t2;
      const __nv_bfloat162 xa = *reinterpret_cast<const __nv_bfloat162*>(x_at);
      const __nv_bfloat162 xb = *reinterpret_cast<const __nv_bfloat162*>(x_at + 8 * pv);
      if (ra < at.n)
        *reinterpret_cast<float2*>(ya + c) = make_float2(fmaf(dsk, __low2float(xa), o[j][0]),
                                                         fmaf(dsk, __high2float(xa), o[j][1]));
      if (rb < at.n)
        *reinterpret_cast<float2*>(yb + c) = make_float2(fmaf(dsk, __low2float(xb), o[j][2]),
                                                         fmaf(dsk, __high2float(xb), o[j][3]));
    }
  }
  if (__syncthreads_or(bad)) {
    float* S = reinterpret_cast<float*>(s_s);             // [K][SC_VT], where the terms were
    for (int i = tid; i < K * SC_VT; i += SC_THREADS) {
      const int c = v0 + i % SC_VT;
      S[i] = c < V ? start[(size_t)(i / SC_VT) * V + c] : 0.f;
    }
    __syncthreads();
    if (tid < SC_VT && v0 + tid < V)
      walk_column(in.a_log[h], in.d_skip[h], dt, at.n, K, pk, b_s, c_s,
                  row + (size_t)h * V + v0 + tid, in.ld, S + tid, SC_VT,
                  y + ((size_t)at.t0 * in.H + h) * V + v0 + tid, (size_t)in.H * V);
  }
}

IX_API int ix_ssd_chunks_applies(int K, int V) {
  return K > 0 && K <= SC_MAX_K && K % 8 == 0 && V > 0 && V % 8 == 0;
}

static inline long long sc_cells(int T, int S, int H) {
  return (long long)(T / SC_L + S + 1) * H;
}

// Floats of scratch for S sequences that bring T tokens together.
IX_API long long ix_ssd_chunks_scratch_floats(int T, int S, int H, int K, int V) {
  return sc_cells(T, S, H) * ((long long)K * V + 1);
}

// Sequences s0 .. S - 1, `tokens` of them all together, the longest of max_q tokens.
IX_API int ix_ssd_chunks(const void* xbc, long long ld, const void* dt_raw, long long ld_dt,
                         const float* dt_bias, const float* a_log, const float* d_skip,
                         float* state, const int* cu_q, const int* state_slot, float* out,
                         int tokens, int S, int s0, int max_q, int H, int V, int K, int G,
                         float* scratch, cudaStream_t stream) {
  const int seqs = S - s0;
  if (seqs <= 0 || tokens <= 0) return IX_OK;
  if (s0 < 0 || H <= 0 || G <= 0 || H % G || max_q <= 0 || !scratch ||
      ld < (long long)H * V + 2LL * G * K || ld_dt < H)
    return IX_ERR_SIZE;
  if (!ix_ssd_chunks_applies(K, V)) return IX_ERR_UNSUPPORTED;
  if ((((uintptr_t)xbc | (uintptr_t)scratch | (uintptr_t)state | (uintptr_t)out) & 15) || ld % 8)
    return IX_ERR_ALIGN;
  const int chunks = (max_q + SC_L - 1) / SC_L;
  if (chunks > 65535 || (long long)H * seqs > 65535) return IX_ERR_SIZE;
  const int Kp = (K + 15) & ~15;
  float* scr_s = scratch;
  float* scr_p = scratch + sc_cells(tokens, seqs, H) * K * V;
  const ScIn in = {(const bf16*)xbc, ld, (const bf16*)dt_raw, ld_dt, dt_bias, a_log, d_skip, cu_q,
                   H, V, K, G, s0};
  const size_t own = ((size_t)SC_L * (Kp + 8) + (size_t)3 * SC_L * (SC_VT + 8)) * 2;
  const size_t tail = ((size_t)2 * SC_L * (Kp + 8) + (size_t)(SC_L + 3 * Kp) * (SC_VT + 8)) * 2;
  cudaError_t e = cudaFuncSetAttribute(ssd_chunk_own_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)own);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ssd_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)tail);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid((V + SC_VT - 1) / SC_VT, chunks, H * seqs);
  ssd_chunk_own_kernel<<<grid, SC_THREADS, own, stream>>>(in, scr_s, scr_p);
  ssd_chunk_join_kernel<<<dim3((K * V / 4 + SJ_THREADS - 1) / SJ_THREADS, H, seqs), SJ_THREADS, 0,
                          stream>>>(scr_s, scr_p, state, cu_q, state_slot, H, K * V, s0);
  ssd_chunk_out_kernel<<<grid, SC_THREADS, tail, stream>>>(in, scr_s, out);
  return ix_launch_status();
}

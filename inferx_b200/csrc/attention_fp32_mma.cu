// Paged causal attention of the 32-bit mode's prompts on the tensor cores: fp32 queries, keys and
// values in three bfloat16 terms a number (gemm_fp32_tc.cu has the arithmetic), fp32 softmax with
// the accurate expf.
//
//   a b = a2 b2 + a1 b3 + a3 b1 + a1 b2 + a2 b1  +  a1 b1
//
// The first five, small ones, and the last have accumulators of their own for a score; a tile's
// weighted values are formed from zero and then added to the fp32 running result, so that no chain
// in a tensor core is longer than 64 keys' or one head's entries.  Semantics are those of
// attention_tiled.cu (window, first keys kept beside it, squashed scores, sink, gate).
//
// A block has 64 queries of one (sequence, head); its warps are four groups of 16 queries times
// the two halves of a tile of 64 keys, each with a running maximum, sum and result of its own that meet
// at the end.  Key tiles start at multiples of 64 of the absolute position, so what a query computes
// depends neither on how its sequence was cut into portions nor on the batch.  Keys and values
// of the next tile are read into registers while the present one is in use, then split into shared
// memory in rows that ldmatrix reads without conflicts.  mma.sync and not tcgen05: a step's whole
// attention is a few hundredths of its products, and what bounds it is the chain of the longest walk.
//
// 600 queries of 16 heads of 128: 78 us against 200 on the CUDA cores, 2,048 queries 486 against
// 1,421; relative error against 64 bits 2.1e-7 against 3.5e-7.
//
// Bfloat16 has no normal third term of numbers below 2^-102: what is left out of one, 2^-126 at most,
// shows where it meets a great partner.  Computed again from the operands at the end are rows whose
// scores or result are not finite, whose result is below 2^-64 and not 0, whose query has entries
// above 2^80 (over the scale, if that is above 1), or that see a key with such entries or a value
// with entries above 2^24.  A block keeps the greatest magnitudes (summed by fours) that it split, and
// looks for the rows only where they are above that (0.5 to 2.5 % of the time; noted key by key on the
// way, 2 to 12).  All of it follows from what the row sees, so its bits do too.
#include <cfloat>

#include "attention_distance.cuh"
#include "bf16_terms.cuh"

#define FM_BQ 64
#define FM_BK 64
#define FM_THREADS 256

__device__ __forceinline__ unsigned fm_smem(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void fm_ldm(unsigned* r, unsigned at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void fm_ldm_t(unsigned* r, unsigned at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void fm_mma(float* c, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// the magnitudes of eight numbers' first terms, every second one's summed
__device__ __forceinline__ __nv_bfloat162 fm_size(const unsigned* t1) {
  auto size = [&](int i) { return __habs2(*reinterpret_cast<const __nv_bfloat162*>(t1 + i)); };
  return __hadd2(__hadd2(size(0), size(1)), __hadd2(size(2), size(3)));
}
// eight numbers of a row into the three term tiles, `part` bytes apart; `most`: the greatest fm_size
__device__ __forceinline__ void fm_split8(const float4& u, const float4& v, unsigned char* at,
                                          int part, __nv_bfloat162& most) {
  unsigned t1[4], t2[4], t3[4];
  bf16_terms2(u.x, u.y, t1[0], t2[0], t3[0]);
  bf16_terms2(u.z, u.w, t1[1], t2[1], t3[1]);
  bf16_terms2(v.x, v.y, t1[2], t2[2], t3[2]);
  bf16_terms2(v.z, v.w, t1[3], t2[3], t3[3]);
  *reinterpret_cast<uint4*>(at) = make_uint4(t1[0], t1[1], t1[2], t1[3]);
  *reinterpret_cast<uint4*>(at + part) = make_uint4(t2[0], t2[1], t2[2], t2[3]);
  *reinterpret_cast<uint4*>(at + 2 * part) = make_uint4(t3[0], t3[1], t3[2], t3[3]);
  most = __hmax2_nan(most, fm_size(t1));
}
// whether eight numbers in memory are above `limit` by fm_size, or not numbers
__device__ __forceinline__ bool fm_great8(const float* p, __nv_bfloat162 limit) {
  unsigned t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 two = __floats2bfloat162_rn(p[2 * i], p[2 * i + 1]);
    t[i] = *reinterpret_cast<const unsigned*>(&two);
  }
  return !__hble2(fm_size(t), limit);
}
// (term of the left, term of the right operand), small products first
__device__ constexpr int FM_L[6] = {1, 0, 2, 0, 1, 0}, FM_R[6] = {1, 2, 0, 1, 0, 0};

struct FmArgs {
  const float *q, *kc, *vc;
  const int *block_table, *cu_q, *q_pos0;
  float* out;
  int S, heads, kvh, page_size, max_blocks, window, keep_first;
  float scale, softcap;
  IxRows rows;
};

__device__ __forceinline__ float fm_score(const FmArgs& a, float dot) {
  float s = dot * a.scale;
  if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
  return s;
}

template <int HD, int VD>
__global__ void __launch_bounds__(FM_THREADS, 1)
attention_fp32_mma_kernel(const FmArgs a) {
  constexpr int QP = (HD + 8) * 2, VP = (VD + 8) * 2;       // row pitches in bytes
  constexpr int Q_PART = FM_BQ * QP, K_PART = FM_BK * QP, V_PART = FM_BK * VP;
  constexpr int KC = HD / 8, VC = VD / 8;                   // pieces of eight in a row
  constexpr int KN = FM_BK * KC / FM_THREADS, VN = FM_BK * VC / FM_THREADS;
  constexpr int MN = KN > VN ? KN : VN;
  extern __shared__ __align__(16) unsigned char fsm[];
  unsigned char* Qs = fsm;
  unsigned char* Ks = Qs + 3 * Q_PART;
  unsigned char* Vs = Ks + 3 * K_PART;
  __shared__ float ml[2][FM_BQ];                            // the second halves' maxima and sums
  __shared__ int again[FM_BQ];

  // which sequence and which 64 queries of it; those with the longest walks first
  int s = -1, tile = gridDim.y - 1 - blockIdx.y;
  for (int ss = 0; ss < a.S; ++ss) {
    const int tiles = (a.cu_q[ss + 1] - a.cu_q[ss] + FM_BQ - 1) / FM_BQ;
    if (tile < tiles) { s = ss; break; }
    tile -= tiles;
  }
  if (s < 0) return;
  const int h = blockIdx.x, kh = h / (a.heads / a.kvh);
  const int tok0 = a.cu_q[s] + tile * FM_BQ;
  const int rows_valid = min(FM_BQ, a.cu_q[s + 1] - tok0);
  const int pos0 = a.q_pos0[s] + tile * FM_BQ;
  const int kv_hi = pos0 + rows_valid;
  const int kv_lo = ix_first_key(pos0, a.window, 0);
  const int kv_lo_tile = kv_lo & ~(FM_BK - 1);
  const int kept = a.window > 0 ? min(a.keep_first, kv_lo) : 0;
  const int* bt = a.block_table + (size_t)s * a.max_blocks;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rw = warp & 3, half = warp >> 2;                // 16 queries, 32 keys of a tile

  // the walk over key tiles: those of kept first keys, then the window's
  auto next = [&](int kv0) {
    return kv0 + FM_BK >= kept && kv0 + FM_BK < kv_lo_tile ? kv_lo_tile : kv0 + FM_BK;
  };
  float4 buf[MN][2];
  // pieces of a tile's rows into registers; zeros where no query of the block looks
  auto fetch = [&](const float* cache, int width, int pieces, int count, int kv0) {
#pragma unroll
    for (int i = 0; i < MN; ++i) {
      if (i >= count) break;
      const int idx = tid + i * FM_THREADS, r = idx / pieces, c = idx - r * pieces;
      const int kp = kv0 + r;
      buf[i][0] = buf[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if ((kp >= kv_lo || kp < kept) && kp < kv_hi) {
        const int page = bt[kp / a.page_size];
        if (page >= 0) {
          const float* p = cache +
              (((size_t)page * a.kvh + kh) * a.page_size + kp % a.page_size) * width + 8 * c;
          buf[i][0] = *reinterpret_cast<const float4*>(p);
          buf[i][1] = *reinterpret_cast<const float4*>(p + 4);
        }
      }
    }
  };
  const __nv_bfloat162 great = __float2bfloat162_rn(1.2089258196146292e24f / fmaxf(a.scale, 1.f));
  const __nv_bfloat162 great_v = __float2bfloat162_rn(16777216.f);
  __nv_bfloat162 most = __float2bfloat162_rn(0.f), most_v = most;     // queries and keys; values
  auto store = [&](unsigned char* to, int pitch, int part, int pieces, int count,
                   __nv_bfloat162& most) {
#pragma unroll
    for (int i = 0; i < MN; ++i) {
      if (i >= count) break;
      const int idx = tid + i * FM_THREADS, r = idx / pieces, c = idx - r * pieces;
      fm_split8(buf[i][0], buf[i][1], to + r * pitch + c * 16, part, most);
    }
  };

  int kv0 = kept > 0 ? 0 : kv_lo_tile;
  fetch(a.kc, HD, KC, KN, kv0);
  for (int idx = tid; idx < FM_BQ * KC; idx += FM_THREADS) {
    const int r = idx / KC, c = idx - r * KC;
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
    if (r < rows_valid) {
      const float* p = a.q + (size_t)(tok0 + r) * a.rows.q_ld + (size_t)h * HD + 8 * c;
      u = *reinterpret_cast<const float4*>(p);
      v = *reinterpret_cast<const float4*>(p + 4);
    }
    fm_split8(u, v, Qs + r * QP + c * 16, Q_PART, most);
  }
  if (tid < FM_BQ) again[tid] = 0;

  // this thread's rows: r0 and r0 + 8; columns 2 (lane % 4) + {0, 1} of a group of eight
  const int r0 = rw * 16 + (lane >> 2);
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float o[VD / 8][4];
#pragma unroll
  for (int j = 0; j < VD / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = 0.f;
  const unsigned q_at = fm_smem(Qs) + (rw * 16 + (lane & 15)) * QP + (lane >> 4) * 16;
  const unsigned k_at = fm_smem(Ks) +
                        (half * 32 + (lane & 7) + ((lane >> 4) << 3)) * QP + ((lane >> 3) & 1) * 16;
  const unsigned v_at = fm_smem(Vs) +
                        (half * 32 + (lane & 7) + (((lane >> 3) & 1) << 3)) * VP + (lane >> 4) * 16;
  bool odd[2] = {false, false};

  for (; kv0 < kv_hi; kv0 = next(kv0)) {
    store(Ks, QP, K_PART, KC, KN, most);
    fetch(a.vc, VD, VC, VN, kv0);
    __syncthreads();
    const int k_first = kv0 + half * 32;
    // whether any of this warp's queries looks at any of its keys
    const int w_pos = pos0 + rw * 16;
    const bool used = k_first <= w_pos + 15 && rw * 16 < rows_valid &&
                      (k_first + 31 >= ix_first_key(w_pos, a.window, 0) || k_first < a.keep_first);
    unsigned pt[2][3][4];                       // weights: 16 keys, term, operand registers
    float corr[2] = {1.f, 1.f};
    if (used) {
      float hi[4][4], lo[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) hi[n][i] = lo[n][i] = 0.f;
#pragma unroll 2
      for (int k = 0; k < HD / 16; ++k) {
        unsigned qf[3][4], kf[3][2][4];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          fm_ldm(qf[t], q_at + t * Q_PART + k * 32);
          fm_ldm(kf[t][0], k_at + t * K_PART + k * 32);
          fm_ldm(kf[t][1], k_at + t * K_PART + 16 * QP + k * 32);
        }
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int n = 0; n < 4; ++n)
            fm_mma(p == 5 ? hi[n] : lo[n], qf[FM_L[p]], kf[FM_R[p]][n >> 1] + 2 * (n & 1));
      }
      float tm[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = r0 + 8 * (i >> 1), qp = pos0 + row;
          const int kp = k_first + 8 * n + 2 * (lane & 3) + (i & 1);
          const bool seen = row < rows_valid && kp <= qp &&
                            (kp >= ix_first_key(qp, a.window, 0) || kp < a.keep_first);
          const float dot = hi[n][i] + lo[n][i];
          odd[i >> 1] |= seen && !(fabsf(dot) <= FLT_MAX);
          hi[n][i] = seen ? fm_score(a, dot) : -INFINITY;
          tm[i >> 1] = fmaxf(tm[i >> 1], hi[n][i]);
        }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        tm[i] = fmaxf(tm[i], __shfl_xor_sync(0xffffffffu, tm[i], 1));
        tm[i] = fmaxf(tm[i], __shfl_xor_sync(0xffffffffu, tm[i], 2));
        const float m_new = fmaxf(m_run[i], tm[i]);
        corr[i] = m_new == -INFINITY ? 1.f : expf(m_run[i] - m_new);     // 0 at the first keys
        m_run[i] = m_new;
      }
      float psum[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float m = m_run[i >> 1];
          hi[n][i] = m == -INFINITY ? 0.f : expf(hi[n][i] - m);
          psum[i >> 1] += hi[n][i];
        }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        psum[i] += __shfl_xor_sync(0xffffffffu, psum[i], 1);
        psum[i] += __shfl_xor_sync(0xffffffffu, psum[i], 2);
        l_run[i] = l_run[i] * corr[i] + psum[i];
      }
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float* pv = hi[2 * g + u];
          bf16_terms2(pv[0], pv[1], pt[g][0][2 * u], pt[g][1][2 * u], pt[g][2][2 * u]);
          bf16_terms2(pv[2], pv[3], pt[g][0][2 * u + 1], pt[g][1][2 * u + 1], pt[g][2][2 * u + 1]);
        }
    }
    store(Vs, VP, V_PART, VC, VN, most_v);
    if (next(kv0) < kv_hi) fetch(a.kc, HD, KC, KN, next(kv0));
    __syncthreads();
    if (used) {
#pragma unroll
      for (int j = 0; j < VD / 16; ++j) {
        unsigned vf[2][3][4];
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int t = 0; t < 3; ++t)
            fm_ldm_t(vf[g][t], v_at + t * V_PART + g * 16 * VP + j * 32);
        float pv[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) pv[n][i] = 0.f;
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int n = 0; n < 2; ++n) fm_mma(pv[n], pt[g][FM_L[p]], vf[g][FM_R[p]] + 2 * n);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            o[2 * j + n][i] = fmaf(o[2 * j + n][i], corr[i >> 1], pv[n][i]);
      }
    }
  }

  // the second halves hand theirs over (in the room of the keys, which have been used)
  __syncthreads();
  float* meet = reinterpret_cast<float*>(Ks);               // [64][VD + 4]
  const int col = 2 * (lane & 3);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (odd[i]) again[r0 + 8 * i] = 1;
  if (half == 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if ((lane & 3) == 0) {
        ml[0][r0 + 8 * i] = m_run[i];
        ml[1][r0 + 8 * i] = l_run[i];
      }
#pragma unroll
      for (int j = 0; j < VD / 8; ++j)
        *reinterpret_cast<float2*>(meet + (r0 + 8 * i) * (VD + 4) + 8 * j + col) =
            make_float2(o[j][2 * i], o[j][2 * i + 1]);
    }
  }
  __syncthreads();
  if (half == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = r0 + 8 * i;
      if (r >= rows_valid) continue;
      const float m = fmaxf(m_run[i], ml[0][r]);
      const float c0 = m_run[i] == -INFINITY ? 0.f : expf(m_run[i] - m);
      const float c1 = ml[0][r] == -INFINITY ? 0.f : expf(ml[0][r] - m);
      float l = l_run[i] * c0 + ml[1][r] * c1;
      const float factor = ix_result_factor<float>(a.rows, tok0 + r, h);
      float inv_l = factor / l;
      if (a.rows.sink) {   // one more term, exp(sink - max), in the denominator
        const float sk = a.rows.sink[h], top = fmaxf(m, sk), c = expf(m - top);
        inv_l = factor * c / (l * c + expf(sk - top));
      }
      float* dst = a.out + (size_t)(tok0 + r) * a.rows.o_ld + (size_t)h * VD + col;
      bool bad = false;
#pragma unroll
      for (int j = 0; j < VD / 8; ++j) {
        const float2 u = *reinterpret_cast<const float2*>(meet + r * (VD + 4) + 8 * j + col);
        const float x = o[j][2 * i] * c0 + u.x * c1, y = o[j][2 * i + 1] * c0 + u.y * c1;
        const float least = fminf(x == 0.f ? 1.f : fabsf(x), y == 0.f ? 1.f : fabsf(y));
        bad |= !(fabsf(x) <= FLT_MAX) || !(fabsf(y) <= FLT_MAX) || least < 5.421010862427522e-20f;
        *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(x * inv_l, y * inv_l);
      }
      if (bad) again[r] = 1;
    }
  }
  const bool some_great =
      __syncthreads_or(!__hble2(most, great) || !__hble2(most_v, great_v));

  // rows that have to be, again: a warp a row, 32 keys at a time, from the operands
  for (int r = warp; r < rows_valid; r += FM_THREADS / 32) {
    if (!again[r] && !some_great) continue;
    const int qp = pos0 + r;
    const float* qr = a.q + (size_t)(tok0 + r) * a.rows.q_ld + (size_t)h * HD;
    auto page_of = [&](int kp) {                 // -1: not seen, or no page
      const bool seen = kp <= qp && (kp >= ix_first_key(qp, a.window, 0) || kp < a.keep_first);
      return seen ? bt[kp / a.page_size] : -1;
    };
    if (!again[r]) {                             // great numbers in the block: among this row's?
      bool mine = lane < KC && fm_great8(qr + 8 * lane, great);
      for (int k0 = kept > 0 ? 0 : kv_lo_tile; k0 <= qp; k0 = next(k0))
        for (int kp = k0 + lane; kp < k0 + FM_BK; kp += 32) {
          const int page = page_of(kp);
          if (page < 0) continue;
          const size_t row = ((size_t)page * a.kvh + kh) * a.page_size + kp % a.page_size;
          for (int c = 0; c < KC; ++c) mine |= fm_great8(a.kc + row * HD + 8 * c, great);
          for (int c = 0; c < VC; ++c) mine |= fm_great8(a.vc + row * VD + 8 * c, great_v);
        }
      if (!__any_sync(0xffffffffu, mine)) continue;
    }
    float m = -INFINITY, l = 0.f, acc[VD / 32];
#pragma unroll
    for (int j = 0; j < VD / 32; ++j) acc[j] = 0.f;
    for (int k0 = kept > 0 ? 0 : kv_lo_tile; k0 <= qp; k0 = next(k0))
      for (int k1 = k0; k1 < k0 + FM_BK; k1 += 32) {
        const int kp = k1 + lane;
        const bool seen = kp <= qp && (kp >= ix_first_key(qp, a.window, 0) || kp < a.keep_first);
        const int page = seen ? bt[kp / a.page_size] : -1;
        const size_t row = page < 0 ? 0 : ((size_t)page * a.kvh + kh) * a.page_size + kp % a.page_size;
        float dot = 0.f;
        if (page >= 0)
          for (int d = 0; d < HD; ++d) dot = fmaf(qr[d], a.kc[row * HD + d], dot);
        const float sc = seen ? fm_score(a, dot) : -INFINITY;
        const float m_new = fmaxf(m, warp_max(sc));
        const float p = !seen || m_new == -INFINITY ? 0.f : expf(sc - m_new);
        const float c = m_new == -INFINITY ? 1.f : expf(m - m_new);
        l = l * c + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int j = 0; j < VD / 32; ++j) acc[j] *= c;
        const unsigned there = __ballot_sync(0xffffffffu, page >= 0);
        for (int i = 0; i < 32; ++i) {
          if (!((there >> i) & 1u)) continue;
          const float pi = __shfl_sync(0xffffffffu, p, i);
          const unsigned long long ri = __shfl_sync(0xffffffffu, (unsigned long long)row, i);
#pragma unroll
          for (int j = 0; j < VD / 32; ++j)
            acc[j] = fmaf(pi, a.vc[ri * VD + lane + 32 * j], acc[j]);
        }
      }
    const float factor = ix_result_factor<float>(a.rows, tok0 + r, h);
    float inv_l = factor / l;
    if (a.rows.sink) {
      const float sk = a.rows.sink[h], top = fmaxf(m, sk), c = expf(m - top);
      inv_l = factor * c / (l * c + expf(sk - top));
    }
    float* dst = a.out + (size_t)(tok0 + r) * a.rows.o_ld + (size_t)h * VD;
#pragma unroll
    for (int j = 0; j < VD / 32; ++j) dst[lane + 32 * j] = acc[j] * inv_l;
  }
}

template <int HD, int VD>
static int launch_fm(const FmArgs& a, int T, cudaStream_t stream) {
  const int smem = 3 * ((FM_BQ + FM_BK) * (HD + 8) + FM_BK * (VD + 8)) * 2;
  auto kern = attention_fp32_mma_kernel<HD, VD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid(a.heads, (T + FM_BQ - 1) / FM_BQ + a.S);   // every sequence can add a part tile
  kern<<<grid, FM_THREADS, smem, stream>>>(a);
  return ix_launch_status();
}

bool ix_attention_fp32_mma_applies(int hd, int vd) {
  return (hd == 64 || hd == 128) && (vd == 64 || vd == 128);
}

// attention_tiled.cu's arguments, fp32, checked there.
int ix_attention_fp32_mma(const float* q, const float* k_cache, const float* v_cache,
                          const int* block_table, const int* cu_q, const int* q_pos0, float* out,
                          int T, int S, int heads, int kvh, int hd, int vd, int page_size,
                          int max_blocks, int window, float scale, float softcap, int keep_first,
                          const IxRows& rows, cudaStream_t stream) {
  const FmArgs a{q, k_cache, v_cache, block_table, cu_q, q_pos0, out, S, heads, kvh, page_size,
                 max_blocks, window, keep_first, scale, softcap, rows};
  if (hd == 128 && vd == 128) return launch_fm<128, 128>(a, T, stream);
  if (hd == 128) return launch_fm<128, 64>(a, T, stream);
  if (vd == 128) return launch_fm<64, 128>(a, T, stream);
  return launch_fm<64, 64>(a, T, stream);
}

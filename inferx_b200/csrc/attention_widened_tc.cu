// Latent attention of prompt portions over keys and values widened once per step, on the
// 5th-generation tensor cores.
//
// Folding the key matrix into the query (latent_attention_mma.cu) makes a query-key pair cost
// 2 (2 rank + dr) operations, 2,176 a head at a latent of 512 and a rotated part of 64; over
// keys of 192 and values of 128 entries it costs 640.  Widening a key's latent costs 2 rank
// (dk + dv) operations a head, once for all queries of the step, so from a few dozen queries
// on a sequence the widened form does less work.  The parts:
//
//   ix_latent_front_inplace   per token: the record [normed latent | rotated key part] into its
//                             cache slot, and the rotated parts of the queries turned in place
//   ix_latent_collect         the records that the step's queries can see, out of the pages into
//                             rows [sequence][position - base], zeros where there is none
//   (the caller's products    latents x key matrix in fp32, latents x value matrix)
//   ix_latent_key_terms       the keys of every head, [plain | rotated part of the record], and
//                             what bfloat16 leaves of the plain entries as a second term
//   ix_widened_attention      this file's attention kernel
//
// The folded form keeps a record as it is and rounds the folded query; here the widened keys would
// be rounded instead, and where attention is sharp that rounding weighs more than any other
// (queries of four times unit size: 0.00623 with rounded keys against 0.00617 folded; eight times
// 0.00817 against 0.00797).  So a key enters its product with the query as two bfloat16 terms,
// 16 bits: 0.00553 and 0.00692, and less than the folded form's error at every sharpness.  A
// softmax weight enters its product with the values as it does in the folded form, in one term or
// (WT 2) in two, the second in the columns of the score buffer that the first leaves free.
//
// The attention kernel: a block owns two tiles of 128 queries of one sequence and head (a query
// is a lane of tensor memory), or one where that leaves fewer SMs idle
// (ix_widened_attention_tiles), and walks their keys in tiles of 64.  Warps 0 and 2 bring K and V
// tiles with TMA into rings of two stages that both query tiles read (one warp for both would have
// the next K wait for the V ahead of it, whose stage is freed a softmax later); one thread of warp
// 1 issues the MMAs, S = Q K^T of tile j + 1 for both query tiles ahead of O += P V of tile j;
// warps 4-7 and 8-11 are the softmax of the two query tiles (a thread holds one query row), whose P
// goes back into the columns of tensor memory that S came from.  What bounds a step of the walk is the
// latency of that chain (read S, mask, max, 64 exponentials, write P), so two independent query
// tiles run on an SM: they hide each other's chain and halve what K and V tiles cost in L2
// traffic.  Two blocks of one tile each, as in attention_prefill_tc.cu, do not fit: the keys'
// 192 entries make Q and the ring 128 KB.  The running max is updated lazily, see there; a row
// is rescaled by its own scores alone, so what it computes does not depend on its neighbours.
//
// Every mbarrier wait is bounded; one that ran out records a code (31: copies, 32: MMA, 33:
// softmax) in the caller's status word and the block runs to its end.
//
// Requires bf16, dk in {64, 128, 192}, dv in {64, 128}.
#include "attention_distance.cuh"
#include "tma_common.cuh"
#include "tcgen05_common.cuh"

#define WA_BM 128
#define WA_BN 64
#define WA_THREADS 384
#define WA_STAGES 2
#define WA_RESCALE_STEP 8.0f   // log2 units

enum { WA_ERR_COPY = 31, WA_ERR_MMA = 32, WA_ERR_SOFTMAX = 33, WA_ERR_ALIGN = 34 };

struct WaBars {
  unsigned long long q_full, k_full[WA_STAGES], k_empty[WA_STAGES], v_full[WA_STAGES],
      v_empty[WA_STAGES], s_full[2][2], p_ready[2], o_done[2];
  unsigned tmem_holder;
  int abort_flag;
};

__device__ __forceinline__ float wa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float wa_max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
__device__ __forceinline__ void wa_fma2(float& r0, float& r1, float x0, float x1, float s,
                                        float c) {
  asm("{ .reg .b64 va, vs, vc, vd;\n\t"
      "mov.b64 va, {%2, %3};\n\t"
      "mov.b64 vs, {%4, %4};\n\t"
      "mov.b64 vc, {%5, %5};\n\t"
      "fma.rn.f32x2 vd, va, vs, vc;\n\t"
      "mov.b64 {%0, %1}, vd; }"
      : "=f"(r0), "=f"(r1)
      : "f"(x0), "f"(x1), "f"(s), "f"(c));
}
__device__ __forceinline__ void wa_add2(float& a0, float& a1, float b0, float b1) {
  asm("{ .reg .b64 va, vb, vd;\n\t"
      "mov.b64 va, {%0, %1};\n\t"
      "mov.b64 vb, {%2, %3};\n\t"
      "add.rn.f32x2 vd, va, vb;\n\t"
      "mov.b64 {%0, %1}, vd; }"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}

// The position of a sequence's first collected row: a multiple of the key tile, at or below
// the first key its first query sees.
__device__ __forceinline__ int wa_base(int first_pos, int window) {
  return ix_first_key(first_pos, window, 0) & ~(WA_BN - 1);
}

// LP: 64-column panels of a head's second key terms in a row of kv (0: one term).  WT: bfloat16
// terms of a softmax weight.
template <int DK, int DV, int LP, int WT>
__global__ void __launch_bounds__(WA_THREADS, 1)
widened_attention_kernel(const __grid_constant__ CUtensorMap map_q,
                         const __grid_constant__ CUtensorMap map_kv,
                         const int* __restrict__ cu_q, const int* __restrict__ q_pos0,
                         bf16* __restrict__ out, int S, int heads, int rows_per_seq, int window,
                         float scale_log2e, const bf16* __restrict__ gate, long long gate_ld,
                         int own, int* __restrict__ status) {
  constexpr int KP = DK / 64, VP = DV / 64;         // 64-column panels
  constexpr int Q_PANEL = WA_BM * 128, Q_BYTES = KP * Q_PANEL;
  constexpr int PANEL = WA_BN * 128, V_TILE = VP * PANEL;
  constexpr int K_LO = KP * PANEL, K_TILE = (KP + LP) * PANEL;   // second terms from K_LO on
  constexpr unsigned TMEM_COLS = 512;
  // O of the two query tiles from columns 0 and 128, S buffers of 64 columns from 256
  constexpr unsigned S_COL = 256;
  constexpr unsigned IDESC_S =
      (1u << 4) | (1u << 7) | (1u << 10) | ((WA_BN >> 3) << 17) | ((WA_BM >> 4) << 24);
  constexpr unsigned IDESC_PV =
      (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((DV >> 3) << 17) | ((WA_BM >> 4) << 24);

  extern __shared__ unsigned char smem[];
  unsigned char* Qs = smem;                          // [2 tiles][panels][128 rows][128 B]
  unsigned char* Ks = Qs + 2 * Q_BYTES;
  unsigned char* Vs = Ks + WA_STAGES * K_TILE;
  WaBars* bars = reinterpret_cast<WaBars*>(Vs + WA_STAGES * V_TILE);

  // which sequence and which `own` tiles of its queries; those with the longest walks first
  int s = 0, tile = gridDim.y - 1 - blockIdx.y;
  {
    bool found = false;
    for (int ss = 0; ss < S; ++ss) {
      const int n = cu_q[ss + 1] - cu_q[ss];
      const int tiles = (n + own * WA_BM - 1) / (own * WA_BM);
      if (tile < tiles) { s = ss; found = true; break; }
      tile -= tiles;
    }
    if (!found) return;
  }
  const int h = blockIdx.x;
  const int tok0 = cu_q[s];
  const int nq = cu_q[s + 1] - tok0;
  const int q0 = tile * own * WA_BM;
  const int rows_valid = min(own * WA_BM, nq - q0);
  const int halves = rows_valid > WA_BM ? 2 : 1;
  const int base = wa_base(q_pos0[s], window);
  const int pos0 = q_pos0[s] + q0;
  const int pmax = pos0 + rows_valid - 1;
  const int kv_lo = ix_first_key(pos0, window, 0);
  const int kt0 = kv_lo & ~(WA_BN - 1);              // base is on a tile's edge too
  const int n_tiles = (pmax + 1 - kt0 + WA_BN - 1) / WA_BN;
  // the first query tile of two ends its walk with its own last position
  const int n_first = (min(pmax, pos0 + WA_BM - 1) + 1 - kt0 + WA_BN - 1) / WA_BN;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  if ((smem_u32(smem) & 1023u) != 0) {
    if (tid == 0) atomicExch(status, WA_ERR_ALIGN);
    return;
  }
  if (tid == 0) {
    mbar_init(&bars->q_full, 1);
    for (int i = 0; i < WA_STAGES; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bars->s_full[t][0], 1);
      mbar_init(&bars->s_full[t][1], 1);
      mbar_init(&bars->p_ready[t], 4);
      mbar_init(&bars->o_done[t], 1);
    }
    bars->abort_flag = 0;
    mbar_init_fence();
    fence_proxy_async();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&bars->tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = __shfl_sync(0xffffffffu, bars->tmem_holder, 0);
  volatile int* abortp = &bars->abort_flag;
  int copied = 0;                        // tiles whose copies this thread started (warps 0 and 2)

  // The copying warps walk the tiles whole too, one lane issuing, so that coordinates stay in
  // uniform registers; with that and with one load of a row's 64 scores, 3,000 queries of 16 heads
  // take 104 us instead of 130, 1,500 of 32 heads 56 instead of 69.
  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(&bars->q_full, halves * Q_BYTES);
      for (int t = 0; t < halves; ++t)
#pragma unroll
        for (int p = 0; p < KP; ++p)
          tma_load_2d(Qs + t * Q_BYTES + p * Q_PANEL, &map_q, h * DK + p * 64,
                      tok0 + q0 + t * WA_BM, &bars->q_full);
    }
    __syncwarp();
    const int row0 = __shfl_sync(0xffffffffu, s * rows_per_seq + (kt0 - base), 0);
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j % WA_STAGES, row = row0 + j * WA_BN;
      ok = __all_sync(0xffffffffu,
                      mbar_wait(&bars->k_empty[st], ((j / WA_STAGES) & 1) ^ 1, abortp));
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(&bars->k_full[st], K_TILE);
#pragma unroll
        for (int p = 0; p < KP; ++p)
          tma_load_2d(Ks + st * K_TILE + p * PANEL, &map_kv, h * DK + p * 64, row,
                      &bars->k_full[st]);
#pragma unroll
        for (int p = 0; p < LP; ++p)
          tma_load_2d(Ks + st * K_TILE + K_LO + p * PANEL, &map_kv,
                      heads * DK + (h * LP + p) * 64, row, &bars->k_full[st]);
      }
      __syncwarp();
      copied = j + 1;
    }
    if (!ok && lane == 0 && !*abortp) { atomicExch(status, WA_ERR_COPY); *abortp = 1; }
  } else if (warp == 2) {
    const int row0 = __shfl_sync(0xffffffffu, s * rows_per_seq + (kt0 - base), 0);
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j % WA_STAGES, row = row0 + j * WA_BN;
      ok = __all_sync(0xffffffffu,
                      mbar_wait(&bars->v_empty[st], ((j / WA_STAGES) & 1) ^ 1, abortp));
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(&bars->v_full[st], V_TILE);
#pragma unroll
        for (int p = 0; p < VP; ++p)
          tma_load_2d(Vs + st * V_TILE + p * PANEL, &map_kv,
                      heads * (DK + LP * 64) + h * DV + p * 64, row, &bars->v_full[st]);
      }
      __syncwarp();
      copied = j + 1;
    }
    if (!ok && lane == 0 && !*abortp) { atomicExch(status, WA_ERR_COPY); *abortp = 1; }
  } else if (warp == 1) {
    // The whole warp walks the tiles and one lane issues: where descriptors are the warp's and not a
    // thread's they stay in uniform registers.  (One lane alone took some 130 cycles an MMA.)
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bars->q_full, 0, abortp));
    // (a descriptor's low bits are the address in 16-byte units)
    const unsigned long long q_desc = umma_desc(Qs), k_desc = umma_desc(Ks);
    const unsigned long long v_desc = umma_desc_mn(Vs, PANEL, 1024);
    auto issue_s = [&](int j) {
      const int st = j % WA_STAGES;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->k_full[st], (j / WA_STAGES) & 1, abortp)))
        return false;
      tc_fence_after();
      const unsigned long long kd = k_desc + (unsigned)((st * K_TILE) >> 4);
      for (int t = j < n_first ? 0 : 1; t < halves; ++t) {
        // the buffer's last reader, P V of tile j - 2, was issued before: the tensor pipe
        // keeps the order
        const unsigned s_col = tmem_base + S_COL + (2 * t + (j & 1)) * WA_BN;
        const unsigned long long qd = q_desc + (unsigned)((t * Q_BYTES) >> 4);
        if (lane == 0) {
#pragma unroll
          for (int kk = 0; kk < 4 * LP; ++kk)          // second terms first: the small ones
            tc_mma(s_col, qd + (((kk >> 2) * Q_PANEL) >> 4) + 2 * (kk & 3),
                   kd + ((K_LO + (kk >> 2) * PANEL) >> 4) + 2 * (kk & 3), IDESC_S,
                   kk > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < 4 * KP; ++kk)
            tc_mma(s_col, qd + (((kk >> 2) * Q_PANEL) >> 4) + 2 * (kk & 3),
                   kd + (((kk >> 2) * PANEL) >> 4) + 2 * (kk & 3), IDESC_S,
                   kk + LP > 0 ? 1u : 0u);
          tc_commit(&bars->s_full[t][j & 1]);
        }
        __syncwarp();
      }
      if (lane == 0) tc_commit(&bars->k_empty[st]);
      __syncwarp();
      return true;
    };
    if (ok) ok = issue_s(0);
    for (int j = 0; j < n_tiles && ok; ++j) {
      if (j + 1 < n_tiles) {
        ok = issue_s(j + 1);
        if (!ok) break;
      }
      const int st = j % WA_STAGES;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->v_full[st], (j / WA_STAGES) & 1, abortp));
      const unsigned long long vd = v_desc + (unsigned)((st * V_TILE) >> 4);
      for (int t = j < n_first ? 0 : 1; t < halves && ok; ++t) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->p_ready[t], j & 1, abortp));
        if (!ok) break;
        tc_fence_after();
        const unsigned p_col = tmem_base + S_COL + (2 * t + (j & 1)) * WA_BN;
        if (lane == 0) {
#pragma unroll
          for (int k4 = 0; k4 < WT * WA_BN / 16; ++k4)
            // 16 keys: 8 columns of packed P (the second terms 32 columns on), two 8-key
            // groups of V's tile
            tc_mma_ts(tmem_base + t * 128, p_col + 8 * k4, vd + 128 * (k4 & 3), IDESC_PV,
                      (j > 0 || k4 > 0) ? 1u : 0u);
          tc_commit(&bars->o_done[t]);
        }
        __syncwarp();
      }
      if (ok && lane == 0) tc_commit(&bars->v_empty[st]);
      __syncwarp();
    }
    if (!ok && lane == 0 && !*abortp) { atomicExch(status, WA_ERR_MMA); *abortp = 1; }
  } else if (warp >= 4 && ((warp - 4) >> 2) < halves) {
    // ---- softmax of query tile t ----
    const int t = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int row = t * WA_BM + quarter * 32 + lane;
    const int pos = pos0 + row;
    const int tile_pos0 = pos0 + t * WA_BM;
    const int lo_last = ix_first_key(min(pmax, tile_pos0 + WA_BM - 1), window, 0);
    const int lo_r = ix_first_key(pos, window, 0);
    const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
    const unsigned o_addr = lane_addr + t * 128;
    const int my_tiles = t == 0 ? n_first : n_tiles;
    float m_ref = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < my_tiles; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[t][j & 1], (j >> 1) & 1, abortp));
      if (!ok) break;
      tc_fence_after();
      const unsigned s_addr = lane_addr + S_COL + (2 * t + (j & 1)) * WA_BN;
      float sc[WA_BN];
      tc_ld64(s_addr, sc);
      const int kbase = kt0 + j * WA_BN;
      if (kbase + WA_BN - 1 > tile_pos0 || kbase < lo_last) {
#pragma unroll
        for (int i = 0; i < WA_BN; ++i) {
          const int kp = kbase + i;
          if (kp > pos || kp < lo_r) sc[i] = -INFINITY;
        }
      }
      float mxa = -INFINITY, mxb = -INFINITY;
#pragma unroll
      for (int i = 0; i < WA_BN; i += 4) {
        mxa = wa_max3(mxa, sc[i], sc[i + 1]);
        mxb = wa_max3(mxb, sc[i + 2], sc[i + 3]);
      }
      const float m_new = fmaxf(m_ref, fmaxf(mxa, mxb) * scale_log2e);
      const bool grow = m_new > m_ref + WA_RESCALE_STEP || (m_ref == -INFINITY && m_new > m_ref);
      const bool rescale = __any_sync(0xffffffffu, grow);
      float corr = 1.f;
      if (grow) {
        corr = wa_exp2(m_ref - m_new);
        m_ref = m_new;
        l_run *= corr;
      }
      const float nbase = m_ref == -INFINITY ? 0.f : -m_ref;
      float pk[WA_BN / 2];
      float pl[WT == 2 ? WA_BN / 2 : 1];   // what the rounding of each pair left over
      float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
#pragma unroll
      for (int i = 0; i < WA_BN; i += 4) {
        float a0, a1, a2, a3;
        wa_fma2(a0, a1, sc[i], sc[i + 1], scale_log2e, nbase);
        wa_fma2(a2, a3, sc[i + 2], sc[i + 3], scale_log2e, nbase);
        const float p0 = wa_exp2(a0), p1 = wa_exp2(a1), p2 = wa_exp2(a2), p3 = wa_exp2(a3);
        wa_add2(sum0, sum1, p0, p1);
        wa_add2(sum2, sum3, p2, p3);
        __nv_bfloat162 v = __floats2bfloat162_rn(p0, p1), v2 = __floats2bfloat162_rn(p2, p3);
        pk[i >> 1] = __uint_as_float(*reinterpret_cast<unsigned*>(&v));
        pk[(i >> 1) + 1] = __uint_as_float(*reinterpret_cast<unsigned*>(&v2));
        if (WT == 2) {
          const float2 f = __bfloat1622float2(v), f2 = __bfloat1622float2(v2);
          __nv_bfloat162 r = __floats2bfloat162_rn(p0 - f.x, p1 - f.y);
          __nv_bfloat162 r2 = __floats2bfloat162_rn(p2 - f2.x, p3 - f2.y);
          pl[(i >> 1) * (WT - 1)] = __uint_as_float(*reinterpret_cast<unsigned*>(&r));
          pl[((i >> 1) + 1) * (WT - 1)] = __uint_as_float(*reinterpret_cast<unsigned*>(&r2));
        }
      }
      l_run += (sum0 + sum1) + (sum2 + sum3);
      if (j > 0) {
        // O may be touched once the previous P V has completed; every phase of this barrier
        // is waited for, in order, also when nothing is rescaled
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_done[t], (j - 1) & 1, abortp));
        if (!ok) break;
        if (rescale) {
          tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < DV; c0 += 32) {
            float o[32];
            tc_ld32(o_addr + c0, o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= corr;
            tc_st32(o_addr + c0, o);
          }
        }
      }
      tc_st32(s_addr, pk);
      if (WT == 2) tc_st32(s_addr + 32, pl);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_ready[t]);
    }
    if (ok)
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_done[t], (my_tiles - 1) & 1, abortp));
    if (!ok) {
      if (lane == 0 && !*abortp) { atomicExch(status, WA_ERR_SOFTMAX); *abortp = 1; }
    } else {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const size_t token = (size_t)(tok0 + q0 + row);
      bf16* dst = out + token * ((size_t)heads * DV) + (size_t)h * DV;
      const bf16* g = gate ? gate + token * gate_ld + (size_t)h * DV : nullptr;
#pragma unroll
      for (int c0 = 0; c0 < DV; c0 += 32) {
        float o[32];
        tc_ld32(o_addr + c0, o);               // every lane takes part in the load
        if (row < rows_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = o[i + u] * inv;
            if (g) {
              const uint4 z4 = *reinterpret_cast<const uint4*>(g + c0 + i);
              const unsigned zw[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float2 z = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zw[u]));
                f[2 * u] *= __fdividef(1.f, 1.f + __expf(-z.x));
                f[2 * u + 1] *= __fdividef(1.f, 1.f + __expf(-z.y));
              }
            }
            unsigned w4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              __nv_bfloat162 v = __floats2bfloat162_rn(f[2 * u], f[2 * u + 1]);
              w4[u] = *reinterpret_cast<unsigned*>(&v);
            }
            *reinterpret_cast<uint4*>(dst + c0 + i) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abortp && lane == 0 && (warp == 0 || warp == 2)) {
    // let copies in flight land before shared memory is given up
    if (warp == 0) mbar_drain(&bars->q_full, 0);
    unsigned long long* full = warp == 0 ? bars->k_full : bars->v_full;
    for (int j = max(0, copied - WA_STAGES); j < copied; ++j)
      mbar_drain(&full[j % WA_STAGES], (j / WA_STAGES) & 1);
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  }
}

// Query tiles a block owns: two, whose chains hide each other (2.1 us a key tile for both), or where
// the device has room for twice the blocks one (1.3 us a key tile, 5 us a block beside its walk).
// By the longest block, or an SM's share of all and half of a shortest one that ends alone
// (sequences taken as equally long).  Two / one tile a block, us: 2,048 queries of 16 heads 72.2 /
// 46.5, 300 behind 2,000 78.6 / 48.1, 1,000 of 32 heads 38.2 / 30.8, but 1,500 of 32 54.8 / 59.0, four
// times 300 behind 200 of 16 22.3 / 28.3.  A row's arithmetic is its own either way.
IX_API int ix_widened_attention_tiles(int T, int S, int heads, int rows_per_seq, int window) {
  const long long each = (T + S - 1LL) / S, most = 8 * 148;
  if ((each + WA_BM - 1) / WA_BM * heads * S > most) return 2;
  double us[2];
  for (int own = 1; own <= 2; ++own) {
    const double step = own == 2 ? 2.1 : 1.3, rest = 5.0;
    const long long blocks = (each + own * WA_BM - 1) / (own * WA_BM);
    long long longest = rows_per_seq / WA_BN, least = 0, all = 0;
    if (window > 0 && longest > (window + own * WA_BM) / WA_BN + 1)
      longest = (window + own * WA_BM) / WA_BN + 1;
    for (long long i = 0; i < blocks; ++i) {
      const long long n = rows_per_seq / WA_BN - i * (own * WA_BM / WA_BN);
      least = n < 1 ? 1 : n < longest ? n : longest;
      all += least;
    }
    const double share = (all * step + blocks * rest) * heads * S / 148.0;
    const double alone = longest * step + rest, tail = 0.5 * (least * step + rest);
    us[own - 1] = blocks * heads * S <= 148 || alone > share + tail ? alone : share + tail;
  }
  return us[0] < 0.97 * us[1] ? 1 : 2;
}

template <int DK, int DV, int LP, int WT>
static int launch_widened(const void* q, long long q_ld, const void* kv, const int* cu_q,
                          const int* q_pos0, void* out, int T, int S, int heads, int rows_per_seq,
                          int window, float scale, const void* gate, long long gate_ld,
                          int* status, cudaStream_t stream) {
  CUtensorMap map_q, map_kv;
  int rc = ix_tensor_map_bf16_2d(&map_q, q, T, (long long)heads * DK, 64, WA_BM, q_ld);
  if (rc != IX_OK) return rc;
  rc = ix_tensor_map_bf16_2d(&map_kv, kv, (long long)S * rows_per_seq,
                             (long long)heads * (DK + LP * 64 + DV), 64, WA_BN);
  if (rc != IX_OK) return rc;
  int smem = 2 * WA_BM * DK * 2 + WA_STAGES * WA_BN * (DK + LP * 64 + DV) * 2 +
             (int)sizeof(WaBars);
  // more than half of an SM's: a second block could not have tensor memory anyway
  if (smem < 120 * 1024) smem = 120 * 1024;
  auto kern = widened_attention_kernel<DK, DV, LP, WT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const int own = ix_widened_attention_tiles(T, S, heads, rows_per_seq, window);
  const int tiles = (T + own * WA_BM - 1) / (own * WA_BM) + S;   // every sequence can add a part tile
  if (tiles > 65535) return IX_ERR_SIZE;
  kern<<<dim3(heads, tiles), WA_THREADS, smem, stream>>>(
      map_q, map_kv, cu_q, q_pos0, (bf16*)out, S, heads, rows_per_seq, window,
      scale * 1.4426950408889634f, (const bf16*)gate, gate_ld, own, status);
  return ix_launch_status();
}

IX_API int ix_widened_attention_applies(int dk, int dv) {
  return (dk == 64 || dk == 128 || dk == 192) && (dv == 64 || dv == 128);
}

// Entries a head's second key terms take in a row of kv, when its first `dn` of dk have some: dn
// rounded up to what the kernel has a form for.
IX_API int ix_widened_second(int dk, int dn) {
  return dn <= 0 ? 0 : dk == 192 && dn <= 128 ? 128 : dk;
}

// q: rows of pitch q_ld (elements), head h's dk entries at h * dk, rotated parts turned.
// kv: [S, rows_per_seq, heads * dk + heads * lo + heads * dv], row r of sequence s the key, the
// second terms of its first lo entries (ix_widened_second; 0: none) and the value of position
// base(s) + r (rows_per_seq a multiple of 64).  weight_terms: 1 or 2.
// out: [T, heads * dv].  gate (null: none): rows of pitch gate_ld, head h's entries at h * dv.
IX_API int ix_widened_attention(const void* q, long long q_ld, const void* kv, const int* cu_q,
                                const int* q_pos0, void* out, int T, int S, int heads, int dk,
                                int dv, int lo, int weight_terms, int rows_per_seq, int window,
                                float scale, const void* gate, long long gate_ld, int* status,
                                cudaStream_t stream) {
  if (T <= 0 || S <= 0) return IX_OK;
  if (heads <= 0 || heads > 65535 || rows_per_seq <= 0 || rows_per_seq % WA_BN || window < 0 ||
      status == nullptr || !(scale > 0.f) || q_ld < (long long)heads * dk ||
      (gate && gate_ld < (long long)heads * dv) || weight_terms < 1 || weight_terms > 2)
    return IX_ERR_SIZE;
  if ((long long)S * rows_per_seq > 0x7fffffffLL) return IX_ERR_SIZE;
  if (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)out | (uintptr_t)gate) & 15) return IX_ERR_ALIGN;
  if (q_ld % 8 || (gate && gate_ld % 8)) return IX_ERR_ALIGN;
#define IX_WA(K, V, L)                                                                          \
  if (dk == K && dv == V && lo == L * 64) {                                                     \
    auto go = weight_terms == 2 ? launch_widened<K, V, L, 2> : launch_widened<K, V, L, 1>;      \
    return go(q, q_ld, kv, cu_q, q_pos0, out, T, S, heads, rows_per_seq, window, scale, gate,   \
              gate_ld, status, stream);                                                         \
  }
#define IX_WA2(K, L)                                                                            \
  IX_WA(K, 64, L)                                                                               \
  IX_WA(K, 128, L)
  IX_WA2(64, 0)
  IX_WA2(64, 1)
  IX_WA2(128, 0)
  IX_WA2(128, 2)
  IX_WA2(192, 0)
  IX_WA2(192, 2)
  IX_WA2(192, 3)
#undef IX_WA2
#undef IX_WA
  return IX_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------------------
// Keys out of their fp32 product, in two bfloat16 terms: a block per row, a thread per 8 entries.
// Bound by its bytes (fp32 in, 4 bytes out an entry).  Entries of a head in kv: dn plain and dr of
// the record's rotated part, then at heads * (dn + dr) the second terms, `lo` a head (dn rounded up
// to ix_widened_second, zeros from dn on).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512)
latent_key_terms_kernel(const float* __restrict__ keys, const bf16* __restrict__ records,
                        int rank, bf16* __restrict__ kv, long long kv_ld, int heads, int dn,
                        int dr, int lo) {
  IX_PDL_WAIT();
  const size_t row = blockIdx.x;
  const int per = (dn + dr) / 8, per_lo = lo / 8;
  const float* k = keys + row * heads * dn;
  const uint4* rot = reinterpret_cast<const uint4*>(records + row * (rank + dr) + rank);
  uint4* hi_row = reinterpret_cast<uint4*>(kv + row * kv_ld);
  uint4* lo_row = hi_row + (size_t)heads * per;
  for (int i = threadIdx.x; i < heads * per; i += blockDim.x) {
    const int h = i / per, c = i - h * per;
    if (c * 8 >= dn) {
      hi_row[i] = rot[c - dn / 8];
      continue;
    }
    const float4* src = reinterpret_cast<const float4*>(k + (size_t)h * dn + c * 8);
    const float4 a = src[0], b = src[1];
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    unsigned t[4], u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
      t[e] = *reinterpret_cast<const unsigned*>(&p);
      // an infinite first term is the whole of it (infinity minus infinity is not a number)
      const float x = __low2float(p), y = __high2float(p);
      const __nv_bfloat162 r = __floats2bfloat162_rn(isinf(x) ? 0.f : f[2 * e] - x,
                                                     isinf(y) ? 0.f : f[2 * e + 1] - y);
      u[e] = *reinterpret_cast<const unsigned*>(&r);
    }
    hi_row[i] = make_uint4(t[0], t[1], t[2], t[3]);
    lo_row[h * per_lo + c] = make_uint4(u[0], u[1], u[2], u[3]);
  }
  const int pad = per_lo - dn / 8;
  for (int i = threadIdx.x; i < heads * pad; i += blockDim.x)
    lo_row[(i / pad) * per_lo + dn / 8 + i % pad] = make_uint4(0u, 0u, 0u, 0u);
}

// keys: [rows, heads * dn] fp32; records: [rows, rank + dr]; kv: rows of pitch kv_ld.
IX_API int ix_latent_key_terms(const float* keys, const void* records, int rank, void* kv,
                               long long kv_ld, long long rows, int heads, int dn, int dr, int lo,
                               cudaStream_t stream) {
  if (rows <= 0) return IX_OK;
  if (rows > 0x7fffffffLL || heads <= 0 || dn <= 0 || dr < 0 || rank <= 0 ||
      lo != ix_widened_second(dn + dr, dn) || kv_ld < (long long)heads * (dn + dr + lo))
    return IX_ERR_SIZE;
  if (dn % 8 || dr % 8 || rank % 8 || kv_ld % 8 ||
      (((uintptr_t)keys | (uintptr_t)records | (uintptr_t)kv) & 15))
    return IX_ERR_ALIGN;
  const int chunks = heads * (dn + dr) / 8;
  const int threads = chunks >= 512 ? 512 : (chunks + 31) / 32 * 32;
  ix_launch(latent_key_terms_kernel, dim3((unsigned)rows), dim3(threads), 0, stream, keys,
            (const bf16*)records, rank, (bf16*)kv, kv_ld, heads, dn, dr, lo);
  return ix_launch_status();
}

// ---------------------------------------------------------------------------
// Records out of the pages: a warp per row, 16-byte copies.
// ---------------------------------------------------------------------------
__global__ void latent_collect_kernel(const uint4* __restrict__ cache,
                                      const int* __restrict__ block_table, int maxb,
                                      const int* __restrict__ q_pos0,
                                      const int* __restrict__ kv_len, uint4* __restrict__ dst,
                                      int rows_per_seq, int page, int window, int chunks) {
  IX_PDL_WAIT();
  const int s = blockIdx.y, r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= rows_per_seq) return;
  const int pos = wa_base(q_pos0[s], window) + r;
  int id = -1;
  if (pos < kv_len[s] && pos / page < maxb) id = block_table[(size_t)s * maxb + pos / page];
  uint4* d = dst + ((size_t)s * rows_per_seq + r) * chunks;
  const uint4* src = cache + ((size_t)max(id, 0) * page + pos % page) * chunks;
  for (int c = threadIdx.x & 31; c < chunks; c += 32)
    d[c] = id >= 0 ? src[c] : make_uint4(0u, 0u, 0u, 0u);
}

IX_API int ix_latent_collect(const void* cache, const int* block_table, int maxb,
                             const int* q_pos0, const int* kv_len, void* dst, int S,
                             int rows_per_seq, int page, int window, int record_bytes,
                             cudaStream_t stream) {
  if (S <= 0) return IX_OK;
  if (S > 65535 || rows_per_seq <= 0 || page <= 0 || maxb <= 0 || window < 0) return IX_ERR_SIZE;
  if (record_bytes <= 0 || record_bytes % 16) return IX_ERR_UNSUPPORTED;
  if (((uintptr_t)cache | (uintptr_t)dst) & 15) return IX_ERR_ALIGN;
  ix_launch(latent_collect_kernel, dim3((rows_per_seq + 7) / 8, S), dim3(256), 0, stream,
            (const uint4*)cache, block_table, maxb, q_pos0, kv_len, (uint4*)dst, rows_per_seq,
            page, window, record_bytes / 16);
  return ix_launch_status();
}

// ---------------------------------------------------------------------------
// front, in place.  q (null: none): row t at t * q_ld, head h's dn plain and dr rotated entries
// at h * (dn + dr); the rotated ones are turned where they lie.  kv: row t at t * kv_ld, the
// down-projection (rank, then dr); its record goes into `cache` at slots[t] (null: none).
// Pairs, angles and the norm as in ix_latent_prepare.  cos and sin of a token's pairs are made
// once, in shared memory, for all heads and the key.
// ---------------------------------------------------------------------------
#define LF_MAX_PAIRS 256

__global__ void latent_front_inplace_kernel(bf16* __restrict__ q, long long q_ld,
                                            const bf16* __restrict__ kv_rows, long long kv_ld,
                                            const int* __restrict__ positions,
                                            const float* __restrict__ freq, float mag,
                                            const float* __restrict__ gain, float eps,
                                            const int* __restrict__ slots,
                                            bf16* __restrict__ cache, int H, int dn, int dr,
                                            int half, int rank) {
  __shared__ float scratch[32];
  __shared__ float2 cs[LF_MAX_PAIRS];
  IX_PDL_WAIT();
  const int t = blockIdx.x;
  const float pos = (float)positions[t];
  for (int p = threadIdx.x; p < half; p += blockDim.x) {
    const float ang = pos * freq[p];
    cs[p] = make_float2(cosf(ang) * mag, sinf(ang) * mag);
  }
  __syncthreads();
  if (cache) {
    const __nv_bfloat162* kv = reinterpret_cast<const __nv_bfloat162*>(kv_rows + (size_t)t * kv_ld);
    __nv_bfloat162* rec =
        reinterpret_cast<__nv_bfloat162*>(cache + (size_t)slots[t] * (rank + dr));
    float ss = 0.f;
    for (int i = threadIdx.x; i < rank / 2; i += blockDim.x) {
      const float2 v = __bfloat1622float2(kv[i]);
      ss += v.x * v.x + v.y * v.y;
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)rank + eps);
    for (int i = threadIdx.x; i < rank / 2; i += blockDim.x) {
      const float2 v = __bfloat1622float2(kv[i]);
      rec[i] = __floats2bfloat162_rn(v.x * inv * gain[2 * i], v.y * inv * gain[2 * i + 1]);
    }
    for (int p = threadIdx.x; p < dr / 2; p += blockDim.x) {
      __nv_bfloat162 v2 = kv[rank / 2 + p];
      if (p < half) {
        const float2 v = __bfloat1622float2(v2);
        v2 = __floats2bfloat162_rn(v.x * cs[p].x - v.y * cs[p].y, v.y * cs[p].x + v.x * cs[p].y);
      }
      rec[rank / 2 + p] = v2;
    }
  }
  if (q) {
    __nv_bfloat162* row = reinterpret_cast<__nv_bfloat162*>(q + (size_t)t * q_ld);
    for (int i = threadIdx.x; i < H * half; i += blockDim.x) {
      const int h = i / half, p = i - h * half;
      __nv_bfloat162* at = row + (h * (dn + dr) + dn) / 2 + p;
      const float2 v = __bfloat1622float2(*at);
      *at = __floats2bfloat162_rn(v.x * cs[p].x - v.y * cs[p].y, v.y * cs[p].x + v.x * cs[p].y);
    }
  }
}

IX_API int ix_latent_front_inplace(void* q, long long q_ld, const void* kv, long long kv_ld,
                                   const int* positions, const float* freq, float mag,
                                   const float* gain, float eps, const int* slots, void* cache,
                                   int T, int H, int dn, int dr, int rot_dims, int rank,
                                   cudaStream_t stream) {
  if (T <= 0) return IX_OK;
  if (H <= 0 || dn < 0 || dr < 0 || rank <= 0 || rot_dims < 0 || rot_dims > dr || rot_dims % 2 ||
      rot_dims / 2 > LF_MAX_PAIRS)
    return IX_ERR_SIZE;
  if (cache && (!kv || !slots || !gain)) return IX_ERR_SIZE;
  if (dn % 2 || dr % 2 || rank % 2 || q_ld % 2 || kv_ld % 2 ||
      (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)cache) & 3))
    return IX_ERR_ALIGN;
  ix_launch(latent_front_inplace_kernel, dim3(T), dim3(128), 0, stream, (bf16*)q, q_ld,
            (const bf16*)kv, kv_ld, positions, freq, mag, gain, eps, slots, (bf16*)cache, H, dn,
            dr, rot_dims / 2, rank);
  return ix_launch_status();
}

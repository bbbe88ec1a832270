// The linear recurrence of recurrent_parts.cu over prompts long enough to be cut into segments that
// are walked side by side.  Per head, with a decay w per key entry:
//
//   S_t = diag(w_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t
//   with a bonus u:                        o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t
//
// Four passes:
//   prepare  q (times q_scale) and k of every token in fp32, rows padded for 16-byte copies
//   local    every segment but a sequence's last, from a zero state without outputs: its own state
//            and the product of its decays
//   join     the segments' start states, S <- P_e S + S_e in ascending e, from the slot's state on
//   walk     every segment from its start state, with outputs; the last one leaves the slot's state
// All of it is fp32, as in the walk from end to end, and differs from it by rounding only.
//
// Lanes and columns, packed arithmetic and the chunks' copies are laid out as in delta_segments.cu
// (segments.cuh); what bounds the walks is a token's chain with four to five warps a scheduler (2
// instructions a cycle of 4; FMA pipe 31 %, shared memory 40 to 47 %).  Walks whose eight warps were
// slices of the key over 32 shared columns took 243 us for the two passes over 2,048 tokens of 16
// heads of 64 x 128, 261 with the bonus, these four 111 and 125 (32 heads 472 and 217, 8 heads 161
// and 67, 256 tokens 49 and 32).
#include "segments.cuh"

// ---------------------------------------------------------------------------
// prepare: a warp per (token, head)
// ---------------------------------------------------------------------------
template <typename TA>
__global__ void __launch_bounds__(128)
linear_prepare_kernel(const TA* __restrict__ q, long long ldq, const TA* __restrict__ k,
                      long long ldk, float* __restrict__ qn, float* __restrict__ kn, int H, int K,
                      int KP, float q_scale) {
  IX_PDL_WAIT();
  const int t = blockIdx.x, lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (h >= H) return;
  const TA* qr = q + (size_t)t * ldq + (size_t)h * K;
  const TA* kr = k + (size_t)t * ldk + (size_t)h * K;
  const size_t at = ((size_t)t * H + h) * KP;
  for (int c = lane; c < KP; c += 32) {
    qn[at + c] = c < K ? __fmul_rn(to_f32(qr[c]), q_scale) : 0.f;
    kn[at + c] = c < K ? to_f32(kr[c]) : 0.f;
  }
}

// ---------------------------------------------------------------------------
// local and walk: grid (column tiles * segments, heads, sequences)
// ---------------------------------------------------------------------------
struct LsIn {
  const float *qn, *kn, *decay, *bonus;
  const int *cu_q, *state_slot;
  int H, K, V, seg_len, vec_w;
};
enum { LS_LOCAL = 0, LS_WALK = 1, LS_BONUS = 2 };

template <typename TA, int KQ, int C, int FORM>
__global__ void __launch_bounds__(DS_THREADS, ds_min_blocks<KQ>())
linear_segment_kernel(LsIn in, const TA* __restrict__ v, long long ldv, float* __restrict__ state,
                      float* __restrict__ out, float* __restrict__ scr_s,
                      float* __restrict__ scr_p) {
  constexpr bool LOCAL = FORM == LS_LOCAL, BONUS = FORM == LS_BONUS;
  constexpr int COLS = DS_GROUPS * C;                     // columns of a block
  constexpr int KP = DS_LANES * KQ * 4;
  constexpr int ROWS = DS_CHUNK * KP;                     // floats of one operand's chunk
  constexpr int PV = DS_CHUNK * COLS / DS_THREADS;        // values a thread stages
  extern __shared__ __align__(16) float sm[];
  float* q_s = sm;                          // [2][DS_CHUNK][KP]
  float* k_s = q_s + 2 * ROWS;
  float* w_s = k_s + 2 * ROWS;
  float* v_s = w_s + 2 * ROWS;              // [2][DS_CHUNK][COLS]
  IX_PDL_WAIT();
  const int K = in.K, V = in.V, H = in.H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l = lane % DS_LANES;
  const int my_col = (tid / DS_LANES) * C;  // the first of this thread's columns
  const int tiles = (V + COLS - 1) / COLS;
  const int seg = blockIdx.x / tiles, v0 = (blockIdx.x % tiles) * COLS;
  const int h = blockIdx.y, s = blockIdx.z, col = v0 + my_col;
  const int seq_begin = in.cu_q[s], seq_end = in.cu_q[s + 1];
  const int nseg_s = (seq_end - seq_begin + in.seg_len - 1) / in.seg_len;
  if (seg >= nseg_s || (LOCAL && seg == nseg_s - 1)) return;
  const int t_begin = seq_begin + seg * in.seg_len, t_end = min(seq_end, t_begin + in.seg_len);
  const size_t cell = ds_cell(in.cu_q, s, in.seg_len, seg, H, h);
  float* my_s = scr_s + cell * K * V;       // local: the segment's own state; walk: its start
  float* my_p = scr_p + cell * K;
  const bool keeps_p = LOCAL && v0 == 0 && warp == 0;     // the decays' products
  auto entry = [&](int i) { return 4 * (l + DS_LANES * (i >> 2)) + (i & 3); };

  ds_pair S[C][KQ * 2], u[KQ * 2], P[KQ * 2];
#pragma unroll
  for (int i = 0; i < KQ * 2; ++i) {
    float uf[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int kk = entry(2 * i + e);
      uf[e] = BONUS && kk < K ? in.bonus[(size_t)h * K + kk] : 0.f;
    }
    u[i] = ds_pack(uf[0], uf[1]);
    P[i] = ds_pack(1.f, 1.f);
#pragma unroll
    for (int y = 0; y < C; ++y) {
      float f[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int kk = entry(2 * i + e);
        f[e] = !LOCAL && kk < K && col + y < V ? my_s[(size_t)kk * V + col + y] : 0.f;
      }
      S[y][i] = ds_pack(f[0], f[1]);
    }
  }

  float pv[PV];
  auto fetch_v = [&](int t0) {
#pragma unroll
    for (int e = 0; e < PV; ++e) {
      const int i = tid + e * DS_THREADS, c = i / COLS, x = v0 + i % COLS;
      pv[e] = (t0 + c < t_end && x < V)
                  ? to_f32(v[(size_t)(t0 + c) * ldv + (size_t)h * V + x]) : 0.f;
    }
  };
  auto fetch = [&](int t0, int buf) {
    const int n = min(DS_CHUNK, t_end - t0);
    for (int i = tid; i < n * (KP / 4); i += DS_THREADS) {
      const int c = i / (KP / 4), x = (i % (KP / 4)) * 4;
      const size_t row = ((size_t)(t0 + c) * H + h) * KP + x;
      const int at = buf * ROWS + c * KP + x;
      if (!LOCAL) ds_async(q_s + at, in.qn + row, 16);
      ds_async(k_s + at, in.kn + row, 16);
      const float* w = in.decay + ((size_t)(t0 + c) * H + h) * K + x;
      if (in.vec_w) {
        if (x < K) ds_async(w_s + at, w, 16);
        else *reinterpret_cast<float4*>(w_s + at) = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) w_s[at + e] = x + e < K ? w[e] : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(t_begin, 0);
  fetch_v(t_begin);
  int buf = 0;
  for (int t0 = t_begin; t0 < t_end; t0 += DS_CHUNK, buf ^= 1) {
    const int n = min(DS_CHUNK, t_end - t0);
#pragma unroll
    for (int e = 0; e < PV; ++e) v_s[buf * DS_CHUNK * COLS + tid + e * DS_THREADS] = pv[e];
    if (t0 + DS_CHUNK < t_end) {
      fetch(t0 + DS_CHUNK, buf ^ 1);
      fetch_v(t0 + DS_CHUNK);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const ulonglong2* w4 = reinterpret_cast<const ulonglong2*>(w_s + buf * ROWS) + l;
    const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(k_s + buf * ROWS) + l;
    const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(q_s + buf * ROWS) + l;
    const int own = my_col + ds_own<C>(l);        // the column whose sum this lane gets
    const float* vc = v_s + buf * DS_CHUNK * COLS + my_col;
    float* dst = LOCAL ? nullptr : out + ((size_t)t0 * H + h) * V + v0 + own;
    // (the lanes that share a column write it once)
    const bool writes = (l & (DS_LANES / C - 1)) == 0 && v0 + own < V;
    for (int c = 0; c < n; ++c) {
      ds_pair vj[C], acc[C];
#pragma unroll
      for (int y = 0; y < C; ++y) {
        vj[y] = ds_pack(vc[c * COLS + y], vc[c * COLS + y]);
        acc[y] = 0;
      }
#pragma unroll
      for (int i = 0; i < KQ; ++i) {
        const ulonglong2 kv = k4[i * DS_LANES], wv = w4[i * DS_LANES];
        const ds_pair k2[2] = {kv.x, kv.y}, w2[2] = {wv.x, wv.y};
        ds_pair q2[2];
        if (!LOCAL) {
          const ulonglong2 qv = q4[i * DS_LANES];
          q2[0] = qv.x;
          q2[1] = qv.y;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (keeps_p) P[2 * i + e] = ds_mul2(P[2 * i + e], w2[e]);
#pragma unroll
          for (int y = 0; y < C; ++y) {
            ds_pair& x = S[y][2 * i + e];
            const ds_pair p = ds_mul2(k2[e], vj[y]);
            if (BONUS) acc[y] = ds_fma2(ds_fma2(u[2 * i + e], p, x), q2[e], acc[y]);
            x = ds_fma2(w2[e], x, p);
            if (!LOCAL && !BONUS) acc[y] = ds_fma2(x, q2[e], acc[y]);
          }
        }
      }
      if (!LOCAL) {
        float part[C];
#pragma unroll
        for (int y = 0; y < C; ++y) {
          const float2 f = ds_unpack(acc[y]);
          part[y] = f.x + f.y;
        }
        const float total = ds_sum<C>(part, l);
        if (writes) *dst = total;
        dst += (size_t)H * V;
      }
      w4 += KP / 4;
      k4 += KP / 4;
      q4 += KP / 4;
    }
    __syncthreads();
  }
  if (!LOCAL && seg != nseg_s - 1) return;
  float* st = LOCAL ? my_s : state + ((size_t)in.state_slot[s] * H + h) * K * V;
#pragma unroll
  for (int i = 0; i < KQ * 2; ++i) {
    const float2 p = ds_unpack(P[i]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int kk = entry(2 * i + e);
      if (kk >= K) continue;
      if (keeps_p && lane < DS_LANES) my_p[kk] = e ? p.y : p.x;
#pragma unroll
      for (int y = 0; y < C; ++y) {
        const float2 f = ds_unpack(S[y][i]);
        if (col + y < V) st[(size_t)kk * V + col + y] = e ? f.y : f.x;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// join: grid (groups of entries, heads, sequences); a thread owns an entry of the state along the
// sequence's segments, eight of which it fetches at a time.  A segment's own state in scratch
// gives way to its start state.
// ---------------------------------------------------------------------------
#define LJ_THREADS 256
#define LJ_AHEAD 8

__global__ void __launch_bounds__(LJ_THREADS)
linear_join_kernel(float* __restrict__ scr_s, const float* __restrict__ scr_p,
                   const float* __restrict__ state, const int* __restrict__ cu_q,
                   const int* __restrict__ state_slot, int H, int K, int V, int seg_len) {
  IX_PDL_WAIT();
  const int h = blockIdx.y, s = blockIdx.z, i = blockIdx.x * LJ_THREADS + threadIdx.x;
  const int nseg_s = (cu_q[s + 1] - cu_q[s] + seg_len - 1) / seg_len;
  if (nseg_s <= 0 || i >= K * V) return;
  const size_t cell = ds_cell(cu_q, s, seg_len, 0, H, h);
  float* own = scr_s + cell * K * V + i;
  const float* p = scr_p + cell * K + i / V;
  float x = state[((size_t)state_slot[s] * H + h) * K * V + i];
  for (int e0 = 0; e0 < nseg_s; e0 += LJ_AHEAD) {
    float o[LJ_AHEAD], w[LJ_AHEAD];
#pragma unroll
    for (int e = 0; e < LJ_AHEAD; ++e)
      if (e0 + e + 1 < nseg_s) {
        o[e] = own[(size_t)(e0 + e) * H * K * V];
        w[e] = p[(size_t)(e0 + e) * H * K];
      }
#pragma unroll
    for (int e = 0; e < LJ_AHEAD; ++e)
      if (e0 + e < nseg_s) {
        own[(size_t)(e0 + e) * H * K * V] = x;
        if (e0 + e + 1 < nseg_s) x = w[e] * x + o[e];
      }
  }
}

static inline size_t ls_smem(int K) {
  return 2 * ((size_t)3 * DS_CHUNK * ds_pitch(K) + DS_CHUNK * ds_cols(K)) * sizeof(float);
}

// Segments for a step whose longest sequence brings max_q_len tokens: as many as keep a pass within
// the blocks the device holds at once, none shorter than 64 tokens.  Returns the number of segments
// and sets *seg_len; 1 and 0 when the sequences are walked from end to end.
IX_API int ix_linear_recurrence_segments(int S, int H, int K, int V, int max_q_len, int min_tokens,
                                         int max_segments, int* seg_len) {
  *seg_len = 0;
  if (S <= 0 || H <= 0 || K <= 0 || V <= 0 || K > 8 * 64 || max_q_len < min_tokens) return 1;
  const long long per = (long long)S * H * ((V + ds_cols(K) - 1) / ds_cols(K));
  long long want = ds_blocks_at_once(K, ls_smem(K)) / per;
  // beyond 256 entries the walk from end to end is the slower one however many heads there are (16
  // heads of 384 x 128, 3,000 tokens: 5,808 us, two segments 2,301)
  if (K > 256 && want < 2) want = 2;
  if (want > max_segments) want = max_segments;
  if (want < 2) return 1;
  int len = (int)((max_q_len + want - 1) / want);
  len = (len + DS_CHUNK - 1) / DS_CHUNK * DS_CHUNK;
  if (len < 64) len = 64;
  const int nseg = (max_q_len + len - 1) / len;
  if (nseg <= 1) return 1;
  *seg_len = len;
  return nseg;
}

// Floats of scratch: the segments' states and decays, q and k in fp32.
IX_API long long ix_linear_segments_scratch_floats(int T, int S, int H, int K, int V,
                                                   int seg_len) {
  const long long cells = ds_cells(T, S, seg_len, H);
  return ((cells * K * V + 3) & ~3LL) + ((cells * K + 3) & ~3LL) + 2LL * T * H * ds_pitch(K);
}

// Sequences are cut into segments of seg_len tokens (nseg covers the longest).
IX_API int ix_linear_segments(const void* q, long long ldq, const void* k, long long ldk,
                              const void* v, long long ldv, int dtype, const float* decay,
                              const float* bonus, float* state, const int* cu_q,
                              const int* state_slot, float* out, int T, int S, int H, int K, int V,
                              float q_scale, int bonus_form, int seg_len, int nseg, float* scratch,
                              cudaStream_t stream) {
  if (S <= 0 || T <= 0) return IX_OK;
  if (H <= 0 || K <= 0 || V <= 0 || K > 8 * 64 || H > 65535 || S > 65535) return IX_ERR_SIZE;
  if (bonus_form && !bonus) return IX_ERR_SIZE;
  if (nseg < 2 || seg_len <= 0 || seg_len % DS_CHUNK || !scratch) return IX_ERR_SIZE;
  if ((uintptr_t)scratch & 15) return IX_ERR_ALIGN;
  const int KP = ds_pitch(K), tiles = (V + ds_cols(K) - 1) / ds_cols(K);
  const long long cells = ds_cells(T, S, seg_len, H);
  float* scr_s = scratch;
  float* scr_p = scr_s + ((cells * K * V + 3) & ~3LL);
  float* qn = scr_p + ((cells * K + 3) & ~3LL);
  float* kn = qn + (size_t)T * H * KP;
  const LsIn in = {qn, kn, decay, bonus, cu_q, state_slot, H, K, V, seg_len,
                   K % 4 == 0 && ((uintptr_t)decay & 15) == 0 ? 1 : 0};
  const size_t smem = ls_smem(K);
#define LS_ONE(L, Q, FORM)                                                                      \
  do {                                                                                          \
    auto kern = linear_segment_kernel<TA, L, Q, FORM>;                                          \
    if (smem > 48 * 1024)                                                                       \
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
    ix_launch(kern, dim3(tiles * nseg, H, S), dim3(DS_THREADS), smem, stream, in, (const TA*)v, \
              ldv, state, out, scr_s, scr_p);                                                   \
  } while (0)
#define LS_GO_LOCAL(L, Q) LS_ONE(L, Q, LS_LOCAL)
#define LS_GO_WALK(L, Q) LS_ONE(L, Q, LS_WALK)
#define LS_GO_BONUS(L, Q) LS_ONE(L, Q, LS_BONUS)
  IX_DISPATCH_DTYPE(dtype, TA, {
    ix_launch(linear_prepare_kernel<TA>, dim3(T, (H + 3) / 4), dim3(128), 0, stream, (const TA*)q,
              ldq, (const TA*)k, ldk, qn, kn, H, K, KP, q_scale);
    DS_BY_K(K, LS_GO_LOCAL);
    ix_launch(linear_join_kernel, dim3((K * V + LJ_THREADS - 1) / LJ_THREADS, H, S),
              dim3(LJ_THREADS), 0, stream, scr_s, (const float*)scr_p, (const float*)state, cu_q,
              state_slot, H, K, V, seg_len);
    if (bonus_form) DS_BY_K(K, LS_GO_BONUS);
    else DS_BY_K(K, LS_GO_WALK);
  });
#undef LS_GO_BONUS
#undef LS_GO_WALK
#undef LS_GO_LOCAL
#undef LS_ONE
  return ix_launch_status();
}

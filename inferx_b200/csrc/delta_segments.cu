// The gated delta rule of delta_parts.cu over prompts long enough to be cut into segments that
// are walked side by side.  Per head, with D_t = diag(g_t) S_(t-1):
//
//   u_t = beta_t (v_t - D_t^T k_t),   S_t = D_t + k_t u_t^T,   o_t = D_t^T q_t + (k_t . q_t) u_t
//
// which is linear in the state, S_t = A_t S_(t-1) + beta_t k_t v_t^T with
// A_t = (I - beta_t k_t k_t^T) diag(g_t).  Four passes:
//   prepare  unit vectors q (times q_scale) and k in fp32, k . q and beta of every token
//   local    every segment but a sequence's last, from a zero state without outputs: its own state,
//            and, as the same walk over the identity's columns with values of zero, the product
//            of its A_t
//   join     the segments' start states, S <- A_e S + S_e in ascending e, from the slot's state on
//   walk     every segment from its start state, with outputs; the last one leaves the slot's state
// All of it is fp32, as in the walk from end to end, and differs from it by rounding only.
//
// In local and walk lanes share columns of the state, in registers (segments.cuh): a token's two
// sums over the key's entries are met by shuffles inside the warp, and warps meet once per 16
// tokens.  Multiplies and adds are packed, two to an instruction; the chunks arrive by cp.async,
// two buffers.  What bounds them is a token's chain of sums, shuffles and updates with four to five
// warps a scheduler (2.1 instructions a cycle of 4; FMA pipe 34 %, shared memory 40 %).  Measured
// (B200, 16 heads of 64 x 128, 2,048 tokens): walks whose eight warps were slices of the key that
// met at a barrier for every token, and that made the unit vectors once per column tile, took 595
// us for both passes, these four 210 us (8 heads 477 and 148, 256 tokens 144 and 56).
#include "segments.cuh"

// ---------------------------------------------------------------------------
// prepare: a warp per (token, key head); rows of KP entries, zero from K on
// ---------------------------------------------------------------------------
template <typename TA>
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const TA* __restrict__ q, long long ldq, const TA* __restrict__ k,
                     long long ldk, const TA* __restrict__ beta_raw, long long ldb,
                     float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ kq,
                     float* __restrict__ beta, int T, int H, int HK, int K, int KP,
                     float unit_eps, float q_scale) {
  IX_PDL_WAIT();
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  for (int h = threadIdx.x; h < H && blockIdx.y == 0; h += 128)
    beta[(size_t)t * H + h] = 1.0f / (1.0f + expf(-to_f32(beta_raw[(size_t)t * ldb + h])));
  const int j = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (j >= HK) return;
  const TA* qr = q + (size_t)t * ldq + (size_t)j * K;
  const TA* kr = k + (size_t)t * ldk + (size_t)j * K;
  float sq = 0.f, sk = 0.f;
  for (int c = lane; c < K; c += 32) {
    const float a = to_f32(qr[c]), b = to_f32(kr[c]);
    sq = fmaf(a, a, sq);
    sk = fmaf(b, b, sk);
  }
  const float iq = q_scale / sqrtf(warp_sum(sq) + unit_eps);
  const float ik = 1.0f / sqrtf(warp_sum(sk) + unit_eps);
  const size_t at = ((size_t)t * HK + j) * KP;
  float dot = 0.f;
  for (int c = lane; c < KP; c += 32) {
    const float a = c < K ? to_f32(qr[c]) * iq : 0.f, b = c < K ? to_f32(kr[c]) * ik : 0.f;
    qn[at + c] = a;
    kn[at + c] = b;
    dot = fmaf(a, b, dot);
  }
  dot = warp_sum(dot);
  if (lane == 0) kq[(size_t)t * HK + j] = dot;
}

// ---------------------------------------------------------------------------
// local and walk: grid (column tiles * segments, heads, sequences)
// ---------------------------------------------------------------------------
struct DsIn {
  const float *qn, *kn, *kq, *beta, *decay;
  const int *cu_q, *state_slot;
  int H, HK, K, V, seg_len, vec_g;
};

template <typename TA, int KQ, int C, bool LOCAL>
__global__ void __launch_bounds__(DS_THREADS, ds_min_blocks<KQ>())
delta_segment_kernel(DsIn in, const TA* __restrict__ v, long long ldv, float* __restrict__ state,
                     float* __restrict__ out, float* __restrict__ scr_s,
                     float* __restrict__ scr_a) {
  constexpr int COLS = DS_GROUPS * C;                     // columns of a block
  constexpr int KP = DS_LANES * KQ * 4;
  constexpr int ROWS = DS_CHUNK * KP;                     // floats of one operand's chunk
  constexpr int PV = DS_CHUNK * COLS / DS_THREADS;        // values a thread stages
  extern __shared__ __align__(16) float sm[];
  float* q_s = sm;                          // [2][DS_CHUNK][KP]
  float* k_s = q_s + 2 * ROWS;
  float* g_s = k_s + 2 * ROWS;
  float* v_s = g_s + 2 * ROWS;              // [2][DS_CHUNK][COLS]
  float* b_s = v_s + 2 * DS_CHUNK * COLS;   // [2][DS_CHUNK] beta
  float* kq_s = b_s + 2 * DS_CHUNK;         // [2][DS_CHUNK]
  IX_PDL_WAIT();
  const int K = in.K, V = in.V, H = in.H;
  const int tid = threadIdx.x, lane = tid & 31;
  const int l = lane % DS_LANES;
  const int my_col = (tid / DS_LANES) * C;  // the first of this thread's columns
  const int vtiles = (V + COLS - 1) / COLS;
  const int tiles = vtiles + (LOCAL ? (K + COLS - 1) / COLS : 0);
  const int seg = blockIdx.x / tiles, tile = blockIdx.x % tiles;
  const bool a_tile = tile >= vtiles;       // columns of the segment's transition matrix
  const int v0 = (a_tile ? tile - vtiles : tile) * COLS, h = blockIdx.y, s = blockIdx.z;
  const int col = v0 + my_col, width = a_tile ? K : V;    // columns col .. col + C - 1
  const int j = h / (H / in.HK);
  const int seq_begin = in.cu_q[s], seq_end = in.cu_q[s + 1];
  const int nseg_s = (seq_end - seq_begin + in.seg_len - 1) / in.seg_len;
  if (seg >= nseg_s || (LOCAL && seg == nseg_s - 1)) return;
  const int t_begin = seq_begin + seg * in.seg_len, t_end = min(seq_end, t_begin + in.seg_len);
  const size_t cell = ds_cell(in.cu_q, s, in.seg_len, seg, H, h);
  float* my_s = scr_s + cell * K * V;       // local: the segment's own state; walk: its start
  float* my_a = scr_a + cell * K * K;
  auto entry = [&](int i) { return 4 * (l + DS_LANES * (i >> 2)) + (i & 3); };

  ds_pair S[C][KQ * 2];
#pragma unroll
  for (int y = 0; y < C; ++y)
#pragma unroll
    for (int i = 0; i < KQ * 2; ++i) {
      float f[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int kk = entry(2 * i + e);
        const bool ok = kk < K && col + y < width;
        f[e] = LOCAL ? (a_tile && ok && kk == col + y ? 1.f : 0.f)
                     : (ok ? my_s[(size_t)kk * V + col + y] : 0.f);
      }
      S[y][i] = ds_pack(f[0], f[1]);
    }

  float pv[PV];
  auto fetch_v = [&](int t0) {
#pragma unroll
    for (int e = 0; e < PV; ++e) {
      const int i = tid + e * DS_THREADS, c = i / COLS, x = v0 + i % COLS;
      pv[e] = (!a_tile && t0 + c < t_end && x < V)
                  ? to_f32(v[(size_t)(t0 + c) * ldv + (size_t)h * V + x]) : 0.f;
    }
  };
  auto fetch = [&](int t0, int buf) {
    const int n = min(DS_CHUNK, t_end - t0);
    for (int i = tid; i < n * (KP / 4); i += DS_THREADS) {
      const int c = i / (KP / 4), x = (i % (KP / 4)) * 4;
      const size_t row = ((size_t)(t0 + c) * in.HK + j) * KP + x;
      const int at = buf * ROWS + c * KP + x;
      if (!LOCAL) ds_async(q_s + at, in.qn + row, 16);
      ds_async(k_s + at, in.kn + row, 16);
      const float* g = in.decay + ((size_t)(t0 + c) * H + h) * K + x;
      if (in.vec_g) {
        if (x < K) ds_async(g_s + at, g, 16);
        else *reinterpret_cast<float4*>(g_s + at) = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) g_s[at + e] = x + e < K ? g[e] : 0.f;
      }
    }
    if (tid < n) ds_async(b_s + buf * DS_CHUNK + tid, in.beta + (size_t)(t0 + tid) * H + h, 4);
    else if (!LOCAL && tid >= 32 && tid - 32 < n)
      ds_async(kq_s + buf * DS_CHUNK + tid - 32, in.kq + (size_t)(t0 + tid - 32) * in.HK + j, 4);
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
    const ulonglong2* g4 = reinterpret_cast<const ulonglong2*>(g_s + buf * ROWS) + l;
    const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(k_s + buf * ROWS) + l;
    const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(q_s + buf * ROWS) + l;
    const int own = my_col + ds_own<C>(l);        // the column whose sums this lane gets
    const float* vc = v_s + buf * DS_CHUNK * COLS + own;
    const float* bc = b_s + buf * DS_CHUNK;
    const float* dc = kq_s + buf * DS_CHUNK;
    float* dst = LOCAL ? nullptr : out + ((size_t)t0 * H + h) * V + v0 + own;
    // (the lanes that share a column write it once)
    const bool writes = (l & (DS_LANES / C - 1)) == 0 && v0 + own < V;
    for (int c = 0; c < n; ++c) {
      ds_pair ka[C], qa[C];
      ulonglong2 kv[KQ];
#pragma unroll
      for (int i = 0; i < KQ; ++i) {
        const ulonglong2 gv = g4[i * DS_LANES];
        kv[i] = k4[i * DS_LANES];
        ulonglong2 qv;
        if (!LOCAL) qv = q4[i * DS_LANES];
#pragma unroll
        for (int y = 0; y < C; ++y) {
          S[y][2 * i] = ds_mul2(gv.x, S[y][2 * i]);
          S[y][2 * i + 1] = ds_mul2(gv.y, S[y][2 * i + 1]);
          ka[y] = i ? ds_fma2(S[y][2 * i], kv[i].x, ka[y]) : ds_mul2(S[y][0], kv[0].x);
          ka[y] = ds_fma2(S[y][2 * i + 1], kv[i].y, ka[y]);
          if (!LOCAL) {
            qa[y] = i ? ds_fma2(S[y][2 * i], qv.x, qa[y]) : ds_mul2(S[y][0], qv.x);
            qa[y] = ds_fma2(S[y][2 * i + 1], qv.y, qa[y]);
          }
        }
      }
      float part[C], u[C];
#pragma unroll
      for (int y = 0; y < C; ++y) {
        const float2 f = ds_unpack(ka[y]);
        part[y] = f.x + f.y;
      }
      const float mine = __fmul_rn(bc[c], vc[c * COLS] - ds_sum<C>(part, l));
      ds_share<C>(mine, u, l);
#pragma unroll
      for (int y = 0; y < C; ++y) {
        const ds_pair uu = ds_pack(u[y], u[y]);
#pragma unroll
        for (int i = 0; i < KQ; ++i) {
          S[y][2 * i] = ds_fma2(kv[i].x, uu, S[y][2 * i]);
          S[y][2 * i + 1] = ds_fma2(kv[i].y, uu, S[y][2 * i + 1]);
        }
      }
      if (!LOCAL) {
#pragma unroll
        for (int y = 0; y < C; ++y) {
          const float2 f = ds_unpack(qa[y]);
          part[y] = f.x + f.y;
        }
        const float qd = ds_sum<C>(part, l);
        if (writes) *dst = __fmaf_rn(dc[c], mine, qd);
        dst += (size_t)H * V;
      }
      g4 += KP / 4;
      k4 += KP / 4;
      q4 += KP / 4;
    }
    __syncthreads();
  }
  if (!LOCAL && seg != nseg_s - 1) return;
  float* st = state + ((size_t)in.state_slot[s] * H + h) * K * V;
#pragma unroll
  for (int y = 0; y < C; ++y)
#pragma unroll
    for (int i = 0; i < KQ * 2; ++i) {
      const float2 f = ds_unpack(S[y][i]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int kk = entry(2 * i + e);
        const float x = e ? f.y : f.x;
        if (kk >= K || col + y >= width) continue;
        if (!LOCAL) st[(size_t)kk * V + col + y] = x;
        else if (a_tile) my_a[(size_t)kk * K + col + y] = x;
        else my_s[(size_t)kk * V + col + y] = x;
      }
    }
}

// ---------------------------------------------------------------------------
// join: grid (tiles of 16 value columns, heads, sequences).  A segment's own state in scratch gives
// way to its start state.  An entry is one chain of multiply-adds from the segment's own state on,
// over the key in ascending order, in every form.
//
// STAGES > 0 (K a multiple of 4 up to 128): a warp for every 32 rows makes the sums, the others bring
// transitions into shared memory STAGES - 1 segments ahead and write the start states out; a
// segment's own state comes into registers one ahead, so that a step waits for none of them.  What is
// left is the reading of shared memory, 512 bytes of registers for a warp's 16-byte read however few
// addresses it has, and the chains: a thread takes four rows by four columns (a read for eight
// multiplies and adds a lane, where one column a thread has a read for three).  Rows are an odd number
// of 16-byte parts apart, so that the eight rows of a quarter-warp's read meet no bank twice.  All four
// passes, one column a thread with transitions one segment ahead against this, us: 16 heads of
// 64 x 128, 2,048 tokens 216 and 210; 12 heads of 96 x 64, 1,000 tokens 170 and 142; 16 heads of
// 128 x 128, 3,000 tokens 597 and 582; the join itself in a step of the first 38.5 and 31.1.  (Quarters
// of the key summed side by side by all eight warps take 26.8, but theirs is another sum, and last bits
// of every prompt's states follow.  Reads a step ahead of the sums, by hand or unrolled, are no faster.)
//
// STAGES 0: a thread owns a column and every sixteenth row, four at a time; transitions from L2.
// ---------------------------------------------------------------------------
#define DJ_COLS 16
#define DJ_THREADS 256
#define DJ_GROUPS (DJ_THREADS / DJ_COLS)
#define DJ_MAX_STAGED 128                        // rows of four warps

// floats between rows (of the transitions) and between columns (of the state)
__host__ __device__ __forceinline__ int dj_pitch(int K) { return ((K >> 2) | 1) * 4; }

template <int STAGES>
__global__ void __launch_bounds__(DJ_THREADS)
delta_join_staged_kernel(float* __restrict__ scr_s, const float* __restrict__ scr_a,
                         const float* __restrict__ state, const int* __restrict__ cu_q,
                         const int* __restrict__ state_slot, int H, int K, int V, int seg_len) {
  extern __shared__ __align__(16) float sm[];    // the state [2][DJ_COLS][pitch], [STAGES][K][pitch]
  IX_PDL_WAIT();
  const int tid = threadIdx.x, pitch = dj_pitch(K);
  const int h = blockIdx.y, s = blockIdx.z, col0 = blockIdx.x * DJ_COLS;
  const int nseg_s = (cu_q[s + 1] - cu_q[s] + seg_len - 1) / seg_len;
  if (nseg_s <= 0) return;
  const float* st = state + ((size_t)state_slot[s] * H + h) * K * V;
  const size_t cell = ds_cell(cu_q, s, seg_len, 0, H, h);
  float *x = sm, *y = x + DJ_COLS * pitch;
  float* a_s = sm + 2 * DJ_COLS * pitch;
  const int summing = (K + 31) & ~31;            // threads; the others copy
  const int copier = tid - summing, copiers = DJ_THREADS - summing;
  auto fetch = [&](int e) {
    if (copier >= 0 && e + 1 < nseg_s) {         // (the last segment has no transitions)
      const float* A = scr_a + (cell + (size_t)e * H) * K * K;
      float* to = a_s + (size_t)(e % STAGES) * K * pitch;
      for (int i = copier * 4; i < K * K; i += copiers * 4) {
        const int row = i / K;
        ds_async(to + row * pitch + (i - row * K), A + i, 16);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // sums: rows m + 8 r, columns n .. n + 3
  const int m = (tid & 7) + (tid & ~31), n = ((tid >> 3) & 3) * 4;
  float next[4][4];                              // these entries of a segment's own state
  auto bring = [&](int e) {
    const float* own = scr_s + (cell + (size_t)e * H) * K * V + col0 + n;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int kk = m + 8 * r;
      const bool there = kk < K && e + 1 < nseg_s;
      if ((V & 3) == 0) {
        const float4 f = there && col0 + n < V ? *reinterpret_cast<const float4*>(own + (size_t)kk * V)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        next[r][0] = f.x, next[r][1] = f.y, next[r][2] = f.z, next[r][3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          next[r][j] = there && col0 + n + j < V ? own[(size_t)kk * V + j] : 0.f;
      }
    }
  };
#pragma unroll
  for (int e = 0; e < STAGES - 1; ++e) fetch(e);
  if (tid < summing) bring(0);
  {
    const int c = tid % DJ_COLS;
    for (int kk = tid / DJ_COLS; kk < K; kk += DJ_GROUPS)
      x[c * pitch + kk] = col0 + c < V ? st[(size_t)kk * V + col0 + c] : 0.f;
  }
  for (int e = 0; e < nseg_s; ++e) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                             // x and A_e are there; y and A_(e-1) have been read
    fetch(e + STAGES - 1);
    if (tid >= summing) {                        // the start state, where the own one has been read
      float* own = scr_s + (cell + (size_t)e * H) * K * V;
      const int c = copier % DJ_COLS, col = col0 + c;
      if (col < V)
        for (int k0 = copier / DJ_COLS * 4; k0 < K; k0 += copiers / DJ_COLS * 4) {
          const float4 v = *reinterpret_cast<const float4*>(x + c * pitch + k0);
          own[(size_t)k0 * V + col] = v.x;
          own[(size_t)(k0 + 1) * V + col] = v.y;
          own[(size_t)(k0 + 2) * V + col] = v.z;
          own[(size_t)(k0 + 3) * V + col] = v.w;
        }
    } else if (e + 1 < nseg_s) {
      float acc[4][4];                           // [row][column]
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][j] = next[r][j];
      bring(e + 1);
      const float* A = a_s + (size_t)(e % STAGES) * K * pitch;
      const float* row[4];
#pragma unroll
      for (int r = 0; r < 4; ++r)                // (a row past the key's is read as its last)
        row[r] = A + min(m + 8 * r, K - 1) * pitch;
#pragma unroll 2
      for (int i = 0; i < K; i += 4) {
        float4 a[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(row[r] + i);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(x + (n + j) * pitch + i);
#pragma unroll
          for (int r = 0; r < 4; ++r)
            acc[r][j] = fmaf(a[r].w, v.w, fmaf(a[r].z, v.z, fmaf(a[r].y, v.y,
                                                                 fmaf(a[r].x, v.x, acc[r][j]))));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (m + 8 * r < K) y[(n + j) * pitch + m + 8 * r] = acc[r][j];
    }
    float* z = x;
    x = y;
    y = z;
  }
}

__global__ void __launch_bounds__(DJ_THREADS)
delta_join_kernel(float* __restrict__ scr_s, const float* __restrict__ scr_a,
                  const float* __restrict__ state, const int* __restrict__ cu_q,
                  const int* __restrict__ state_slot, int H, int K, int V, int seg_len) {
  extern __shared__ __align__(16) float sm[];   // [2][K][DJ_COLS] the state's columns
  IX_PDL_WAIT();
  const int tid = threadIdx.x, c = tid % DJ_COLS, group = tid / DJ_COLS;
  const int h = blockIdx.y, s = blockIdx.z, col = blockIdx.x * DJ_COLS + c;
  const int nseg_s = (cu_q[s + 1] - cu_q[s] + seg_len - 1) / seg_len;
  if (nseg_s <= 0) return;
  const bool ok = col < V;
  const float* st = state + ((size_t)state_slot[s] * H + h) * K * V;
  const size_t cell = ds_cell(cu_q, s, seg_len, 0, H, h);
  float *x = sm, *y = sm + K * DJ_COLS;
  for (int kk = group; kk < K; kk += DJ_GROUPS)
    x[kk * DJ_COLS + c] = ok ? st[(size_t)kk * V + col] : 0.f;
  for (int e = 0; e < nseg_s; ++e) {
    float* own = scr_s + (cell + (size_t)e * H) * K * V;
    const float* A = scr_a + (cell + (size_t)e * H) * K * K;
    const bool more = e + 1 < nseg_s;
    __syncthreads();
    for (int k0 = group; k0 < K; k0 += 4 * DJ_GROUPS) {
      float acc[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int kk = k0 + r * DJ_GROUPS;
        acc[r] = 0.f;
        if (kk < K && ok) {
          if (more) acc[r] = own[(size_t)kk * V + col];
          own[(size_t)kk * V + col] = x[kk * DJ_COLS + c];
        }
      }
      if (!more) continue;
      if ((K & 3) == 0) {
#pragma unroll 4
        for (int i = 0; i < K; i += 4) {
          const float x0 = x[i * DJ_COLS + c], x1 = x[(i + 1) * DJ_COLS + c];
          const float x2 = x[(i + 2) * DJ_COLS + c], x3 = x[(i + 3) * DJ_COLS + c];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int kk = k0 + r * DJ_GROUPS;
            if (kk < K) {
              const float4 a = *reinterpret_cast<const float4*>(A + (size_t)kk * K + i);
              acc[r] = fmaf(a.w, x3, fmaf(a.z, x2, fmaf(a.y, x1, fmaf(a.x, x0, acc[r]))));
            }
          }
        }
      } else {
        for (int i = 0; i < K; ++i) {
          const float x0 = x[i * DJ_COLS + c];
#pragma unroll
          for (int r = 0; r < 4; ++r)
            if (k0 + r * DJ_GROUPS < K)
              acc[r] = fmaf(A[(size_t)(k0 + r * DJ_GROUPS) * K + i], x0, acc[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (k0 + r * DJ_GROUPS < K) y[(k0 + r * DJ_GROUPS) * DJ_COLS + c] = acc[r];
    }
    float* z = x;
    x = y;
    y = z;
  }
}

static inline size_t dj_smem(int K, int stages) {
  if (stages == 0) return (size_t)2 * K * DJ_COLS * sizeof(float);
  return (size_t)(2 * DJ_COLS + stages * K) * dj_pitch(K) * sizeof(float);
}

// Buffers of transitions: four where all blocks are resident with them, else two (blocks that come
// in two rounds lose more than a wait for L2 a segment); none where rows are not whole 16-byte parts
// or are above 128, where two do not fit.
static inline int dj_stages(int K, long long blocks) {
  if (K % 4 || K > DJ_MAX_STAGED) return 0;
  const long long an_sm = 227 * 1024 / (long long)(dj_smem(K, 4) + 1024);
  return an_sm * 148 >= blocks ? 4 : 2;
}

static inline size_t ds_smem(int K) {
  return 2 * ((size_t)3 * DS_CHUNK * ds_pitch(K) + DS_CHUNK * ds_cols(K) + 2 * DS_CHUNK) *
         sizeof(float);
}

// Segments for a step whose longest sequence brings max_q_len tokens: as many as keep the local
// pass within the blocks the device holds at once (a second, nearly empty round would double it),
// none shorter than 64 tokens.  Returns the number of segments and sets *seg_len; 1 and 0 when the
// sequences are walked from end to end.
IX_API int ix_delta_recurrence_segments(int S, int H, int K, int V, int max_q_len, int min_tokens,
                                        int max_segments, int* seg_len) {
  *seg_len = 0;
  if (S <= 0 || H <= 0 || K <= 0 || V <= 0 || K > 8 * 64 || max_q_len < min_tokens) return 1;
  const int cols = ds_cols(K);
  const long long per = (long long)S * H * ((V + cols - 1) / cols + (K + cols - 1) / cols);
  // (the last segment has no local pass)
  long long want = ds_blocks_at_once(K, ds_smem(K)) / per + 1;
  if (want > max_segments) want = max_segments;
  if (want < 2) return 1;
  // two segments on a device that the sequences nearly fill: four passes over a few dozen tokens
  // each take longer than one (64 heads of 128 x 128: 128 tokens 131 us against 109, 200 183
  // against 168, 256 207 against 213)
  if (want == 2 && K > 64 && max_q_len < 256) return 1;
  int len = (int)((max_q_len + want - 1) / want);
  len = (len + DS_CHUNK - 1) / DS_CHUNK * DS_CHUNK;
  if (len < 64) len = 64;
  const int nseg = (max_q_len + len - 1) / len;
  if (nseg <= 1) return 1;
  *seg_len = len;
  return nseg;
}

// Floats of scratch: the segments' states and transitions, unit vectors, k . q and beta.
IX_API long long ix_delta_segments_scratch_floats(int T, int S, int H, int HK, int K, int V,
                                                  int seg_len) {
  const long long cells = ds_cells(T, S, seg_len, H);
  return ((cells * K * V + 3) & ~3LL) + ((cells * K * K + 3) & ~3LL) +
         2LL * T * HK * ds_pitch(K) + (long long)T * (HK + H) + 8;
}

// Sequences are cut into segments of seg_len tokens (nseg covers the longest).
IX_API int ix_delta_segments(const void* q, long long ldq, const void* k, long long ldk,
                             const void* v, long long ldv, const void* beta_raw, long long ldb,
                             int dtype, const float* decay, float* state, const int* cu_q,
                             const int* state_slot, float* out, int T, int S, int H, int HK, int K,
                             int V, float unit_eps, float q_scale, int seg_len, int nseg,
                             float* scratch, cudaStream_t stream) {
  if (S <= 0 || T <= 0) return IX_OK;
  if (H <= 0 || HK <= 0 || H % HK || K <= 0 || V <= 0 || K > 8 * 64 || H > 65535 || S > 65535)
    return IX_ERR_SIZE;
  if (ldq < (long long)HK * K || ldk < (long long)HK * K || ldv < (long long)H * V || ldb < H)
    return IX_ERR_SIZE;
  if (nseg < 2 || seg_len <= 0 || seg_len % DS_CHUNK || !scratch) return IX_ERR_SIZE;
  if ((uintptr_t)scratch & 15) return IX_ERR_ALIGN;
  const int KP = ds_pitch(K), cols = ds_cols(K);
  const long long cells = ds_cells(T, S, seg_len, H);
  float* scr_s = scratch;
  float* scr_a = scr_s + ((cells * K * V + 3) & ~3LL);
  float* qn = scr_a + ((cells * K * K + 3) & ~3LL);
  float* kn = qn + (size_t)T * HK * KP;
  float* kq = kn + (size_t)T * HK * KP;
  float* beta = kq + (size_t)T * HK;
  const int vtiles = (V + cols - 1) / cols, atiles = (K + cols - 1) / cols;
  const DsIn in = {qn, kn, kq, beta, decay, cu_q, state_slot, H, HK, K, V, seg_len,
                   K % 4 == 0 && ((uintptr_t)decay & 15) == 0 ? 1 : 0};
  const size_t smem = ds_smem(K);
  const dim3 join_grid((V + DJ_COLS - 1) / DJ_COLS, H, S);
  const int stages = dj_stages(K, (long long)join_grid.x * H * S);
  const size_t join = dj_smem(K, stages);
  auto join_kern = stages == 4 ? delta_join_staged_kernel<4>
                   : stages == 2 ? delta_join_staged_kernel<2> : delta_join_kernel;
  if (join > 48 * 1024)
    cudaFuncSetAttribute(join_kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)join);
#define DS_ONE(L, Q, LOCAL, TILES)                                                              \
  do {                                                                                          \
    auto kern = delta_segment_kernel<TA, L, Q, LOCAL>;                                          \
    if (smem > 48 * 1024)                                                                       \
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
    ix_launch(kern, dim3((TILES) * nseg, H, S), dim3(DS_THREADS), smem, stream, in, (const TA*)v, \
              ldv, state, out, scr_s, scr_a);                                                   \
  } while (0)
#define DS_LOCAL(L, Q) DS_ONE(L, Q, true, vtiles + atiles)
#define DS_WALK(L, Q) DS_ONE(L, Q, false, vtiles)
  IX_DISPATCH_DTYPE(dtype, TA, {
    ix_launch(delta_prepare_kernel<TA>, dim3(T, (HK + 3) / 4), dim3(128), 0, stream, (const TA*)q,
              ldq, (const TA*)k, ldk, (const TA*)beta_raw, ldb, qn, kn, kq, beta, T, H, HK, K, KP,
              unit_eps, q_scale);
    DS_BY_K(K, DS_LOCAL);
    ix_launch(join_kern, join_grid, dim3(DJ_THREADS), join, stream, scr_s,
              (const float*)scr_a, (const float*)state, cu_q, state_slot, H, K, V, seg_len);
    DS_BY_K(K, DS_WALK);
  });
#undef DS_WALK
#undef DS_LOCAL
#undef DS_ONE
  return ix_launch_status();
}

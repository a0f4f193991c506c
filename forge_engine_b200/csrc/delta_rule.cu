// The gated delta rule: a state per head that is decayed and then corrected towards each key's value.
//
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//     beta = sigmoid(zb),  g = exp(-exp(A) softplus(za + b)),   per head
//
// q, k and v pass a short causal convolution over time and silu, q and k are made unit vectors per
// head (q times dk^(-1/2)); groups of heads share a q/k head.  A head's o is divided by its root
// mean square, weighted and gated.
//
//   delta_prepare   convolutions, silu, unit vectors, beta and log g of a token; the last taps - 1
//                   rows of the convolution's input stay in the request's state.
//   state_walk      (state_recurrence.cuh) short entries.
//   delta_solve / delta_chain / state_out   long entries in chunks.  With c_t the sum of log g from the
//                   chunk's first token up to t and S the state before the chunk, the u of a chunk solve
//                     u_t + sum_(j < t) L_tj u_j = beta_t (v_t - e^(c_t) S^T k_t),
//                     L_tj = beta_t e^(c_t - c_j) k_t . k_j,
//                   a unit lower triangular system.  delta_solve solves it for all chunks side by side, once
//                   for the right side beta v and once for beta e^c k, so that u = U - W S; delta_chain walks
//                   the chunks with two products each (u, and the state it leads to); then
//                     o_t = e^(c_t) S^T q_t + sum_(j <= t) e^(c_t - c_j) (q_t . k_j) u_j.
#include "state_recurrence.cuh"

// ---------------------------------------------------------------------------
// delta_prepare
// ---------------------------------------------------------------------------
struct DeltaPrepare {
  const float* proj;        // [tokens, ld]: q, k, v from column 0, zb and za at b_off, a_off
  long long ld;
  int b_off, a_off;
  const float* conv;        // [taps, channels]
  int taps;
  float* state;             // [rows, taps - 1, channels], oldest first
  const int *slots, *cu_tokens, *token_entry;
  const float *a_log, *dt_bias;     // [heads]
  int kv_heads, dk, heads, dv;
  float* out;               // [tokens, channels]: q, k unit vectors, v
  float* gates;             // [tokens, heads, 2]: beta, log g
  int n_tokens;
};

#define DP_WARPS 4

// One token's channels of one row - a q, k or v head - by a warp: convolution from `input(j)` (the
// inputs j tokens back), silu, and for q and k the unit vector.  `buf` is the warp's own; a lane reads
// back only what it wrote.  V: neighbouring channels a lane takes at a time.
template <int V> __device__ __forceinline__ void dp_load(const float* p, float* v) {
  if constexpr (V == 4) load4(p, v);
  else if constexpr (V == 2) { const float2 a = *reinterpret_cast<const float2*>(p); v[0] = a.x, v[1] = a.y; }
  else v[0] = p[0];
}
template <int V> __device__ __forceinline__ void dp_store(float* p, const float* v) {
  if constexpr (V == 4) store4(p, v);
  else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else p[0] = v[0];
}

template <int V, typename F>
__device__ __forceinline__ void delta_prepare_row(const DeltaPrepare& p, int t, int r, float* buf, F input) {
  const int qk = p.kv_heads * p.dk, channels = 2 * qk + p.heads * p.dv, lane = threadIdx.x & 31;
  const bool unit = r < 2 * p.kv_heads;
  const int base = unit ? r * p.dk : 2 * qk + (r - 2 * p.kv_heads) * p.dv, size = unit ? p.dk : p.dv;
  float* out = p.out + (size_t)t * channels + base;
  float ss = 0.f;
  for (int d = lane * V; d < size; d += 32 * V) {
    float y[V], w[V], x[V];
#pragma unroll
    for (int e = 0; e < V; ++e) y[e] = 0.f;
#pragma unroll 4
    for (int j = p.taps - 1; j >= 0; --j) {
      dp_load<V>(p.conv + (size_t)(p.taps - 1 - j) * channels + base + d, w), dp_load<V>(input(j) + base + d, x);
#pragma unroll
      for (int e = 0; e < V; ++e) y[e] = fmaf(w[e], x[e], y[e]);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) {
      y[e] = y[e] / (1.f + expf(-y[e]));
      ss = fmaf(y[e], y[e], ss);
    }
    dp_store<V>(unit ? buf + d : out + d, y);
  }
  if (!unit) return;
  const float inv = (r < p.kv_heads ? 1.f / sqrtf((float)p.dk) : 1.f) / sqrtf(warp_sum(ss) + 1e-6f);
  for (int d = lane * V; d < size; d += 32 * V) {
    float y[V];
    dp_load<V>(buf + d, y);
#pragma unroll
    for (int e = 0; e < V; ++e) y[e] *= inv;
    dp_store<V>(out + d, y);
  }
}

__device__ __forceinline__ void delta_prepare_gate(const DeltaPrepare& p, int t, int h) {
  const float* src = p.proj + (size_t)t * p.ld;
  float* dst = p.gates + ((size_t)t * p.heads + h) * 2;
  dst[0] = 1.f / (1.f + expf(-src[p.b_off + h]));
  dst[1] = -expf(p.a_log[h]) * sr_softplus(src[p.a_off + h] + p.dt_bias[h]);
}
__device__ __forceinline__ void delta_prepare_gates(const DeltaPrepare& p, int t) {
  for (int h = threadIdx.x; h < p.heads; h += blockDim.x) delta_prepare_gate(p, t, h);
}

template <int V>
__global__ void __launch_bounds__(32 * DP_WARPS) delta_prepare_kernel(DeltaPrepare p, int inner) {
  extern __shared__ __align__(16) float smem[];      // [DP_WARPS][dk]
  pdl_trigger();
  pdl_wait();
  const int back = p.taps - 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.y * DP_WARPS + warp, rows = 2 * p.kv_heads + p.heads;
  float* buf = smem + warp * p.dk;
  if ((int)blockIdx.x < inner) {
    // a token with all its taps inside the step (inner 0: they are delta_prepare_run's)
    const int t = blockIdx.x;
    if (t - p.cu_tokens[p.token_entry[t]] < back) return;
    if (r < rows) delta_prepare_row<V>(p, t, r, buf, [&](int j) { return p.proj + (size_t)(t - j) * p.ld; });
    if (blockIdx.y == 0) delta_prepare_gates(p, t);
    return;
  }
  // an entry's edge: its first taps - 1 tokens, then the state for the next step
  const int entry = blockIdx.x - inner;
  const int first = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - first, edge = min(count, back);
  if (count <= 0) return;
  if (blockIdx.y == 0)
    for (int i = 0; i < edge; ++i) delta_prepare_gates(p, first + i);
  if (r >= rows) return;
  const int qk = p.kv_heads * p.dk, channels = 2 * qk + p.heads * p.dv;
  float* st = p.state + (size_t)p.slots[entry] * back * channels;
  for (int i = 0; i < edge; ++i)
    delta_prepare_row<V>(p, first + i, r, buf, [&](int j) {
      return j <= i ? p.proj + (size_t)(first + i - j) * p.ld : (const float*)st + (size_t)(back + i - j) * channels;
    });
  // the last taps - 1 rows of (state rows, the step's rows), once the warp has read the old ones; a
  // channel is one lane's here, which reads a state row only before it overwrites it
  __syncwarp();
  const int base = r < 2 * p.kv_heads ? r * p.dk : 2 * qk + (r - 2 * p.kv_heads) * p.dv;
  for (int d = lane; d < (r < 2 * p.kv_heads ? p.dk : p.dv); d += 32)
    for (int k = 0; k < back; ++k) {
      const int at = count + k;
      st[(size_t)k * channels + base + d] =
          at < back ? st[(size_t)at * channels + base + d] : p.proj[(size_t)(first + at - back) * p.ld + base + d];
    }
}

// Tokens with all their taps inside the step, DP_RUN of them in a row by a warp for one q, k or v head of
// at most 32 V elements: every input is read once instead of once per tap.  Bound by the bytes in and out
// (2,048 tokens of 4,096 channels: 67 us with a warp per token and head; 24 us this way and 10 us for the entry's edge).
#define DP_RUN 16
template <int V, int TAPS>
__global__ void __launch_bounds__(32 * DP_WARPS) delta_prepare_run_kernel(DeltaPrepare p) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.y * DP_WARPS + warp, t0 = blockIdx.x * DP_RUN, end = min(p.n_tokens, t0 + DP_RUN);
  if (blockIdx.y == 0)
    for (int i = threadIdx.x; i < (end - t0) * p.heads; i += blockDim.x) {
      const int t = t0 + i / p.heads, h = i % p.heads;
      if (t - p.cu_tokens[p.token_entry[t]] >= TAPS - 1) delta_prepare_gate(p, t, h);
    }
  if (r >= 2 * p.kv_heads + p.heads) return;
  const int qk = p.kv_heads * p.dk, channels = 2 * qk + p.heads * p.dv;
  const bool unit = r < 2 * p.kv_heads;
  const int size = unit ? p.dk : p.dv, at = (unit ? r * p.dk : 2 * qk + (r - 2 * p.kv_heads) * p.dv) + lane * V;
  const bool live = lane * V < size;
  const float lead = r < p.kv_heads ? 1.f / sqrtf((float)p.dk) : 1.f;
  float w[TAPS][V], x[TAPS][V];          // x[j]: the input TAPS - 1 - j tokens back
#pragma unroll
  for (int j = 0; j < TAPS; ++j)
#pragma unroll
    for (int e = 0; e < V; ++e) w[j][e] = x[j][e] = 0.f;
  if (live) {
#pragma unroll
    for (int j = 0; j < TAPS; ++j) dp_load<V>(p.conv + (size_t)j * channels + at, w[j]);
#pragma unroll
    for (int j = 1; j < TAPS; ++j)
      if (t0 + j - TAPS >= 0) dp_load<V>(p.proj + (size_t)(t0 + j - TAPS) * p.ld + at, x[j]);
  }
  for (int first = t0; first < end; first += 4) {
    float in[4][V];
    int back[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int e = 0; e < V; ++e) in[u][e] = 0.f;
      const int t = min(first + u, end - 1);
      if (live) dp_load<V>(p.proj + (size_t)t * p.ld + at, in[u]);
      back[u] = t - p.cu_tokens[p.token_entry[t]];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = first + u;
      if (t >= end) break;
#pragma unroll
      for (int e = 0; e < V; ++e) {
#pragma unroll
        for (int j = 0; j + 1 < TAPS; ++j) x[j][e] = x[j + 1][e];
        x[TAPS - 1][e] = in[u][e];
      }
      if (back[u] < TAPS - 1) continue;                // the entry's edge: another kernel's
      float y[V], ss = 0.f;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        y[e] = 0.f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) y[e] = fmaf(w[j][e], x[j][e], y[e]);
        y[e] = y[e] / (1.f + expf(-y[e]));
        ss = fmaf(y[e], y[e], ss);
      }
      if (unit) {
        const float inv = lead / sqrtf(warp_sum(ss) + 1e-6f);
#pragma unroll
        for (int e = 0; e < V; ++e) y[e] *= inv;
      }
      if (live) dp_store<V>(p.out + (size_t)t * channels + at, y);
    }
  }
}

FE_EXPORT int fe_delta_prepare(const float* proj, long long ld, int b_off, int a_off, const float* conv, int taps, float* state,
                               const int* slots, const int* cu_tokens, const int* token_entry, const float* a_log,
                               const float* dt_bias, int kv_heads, int dk, int heads, int dv, float* out, float* gates,
                               int n_tokens, int n_entries, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (taps < 1 || kv_heads < 1 || heads < 1 || dk < 1 || dv < 1 || heads % kv_heads || (taps > 1 && state == nullptr)) return FE_ERR_BAD_SHAPE;
  DeltaPrepare p{proj, ld, b_off, a_off, conv, taps, state, slots, cu_tokens, token_entry, a_log, dt_bias, kv_heads, dk, heads, dv, out, gates, n_tokens};
  const size_t smem = sizeof(float) * (size_t)DP_WARPS * dk;
  const int pieces = (2 * kv_heads + heads + DP_WARPS - 1) / DP_WARPS;
  if (smem > 48 * 1024 || pieces > 65535) return FE_ERR_TOO_LARGE;
  const bool wide = dk % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 &&
                    (((uintptr_t)proj | (uintptr_t)conv | (uintptr_t)state | (uintptr_t)out) & 15) == 0;
  // many tokens: runs of them, then the entries' edges alone.  Below 256 tokens there are too few runs to
  // fill the machine, and a block per token starts all at once.
  const int most = dk > dv ? dk : dv, V = most <= 32 ? 1 : most <= 64 ? 2 : 4;
  int inner = n_tokens;
  if (n_tokens >= 256 && taps >= 2 && taps <= 4 && most <= 128 && (V == 1 || wide || (V == 2 && dk % 2 == 0 && dv % 2 == 0 && ld % 2 == 0 &&
      (((uintptr_t)proj | (uintptr_t)conv | (uintptr_t)out) & 7) == 0))) {
    inner = 0;
    const dim3 runs((n_tokens + DP_RUN - 1) / DP_RUN, pieces);
    int rc = 0;
#define DP_RUNS(V_, TAPS) rc = fe_launch_dependent(delta_prepare_run_kernel<V_, TAPS>, runs, dim3(32 * DP_WARPS), 0, stream, p)
#define DP_RUNS_BY_V(TAPS)        \
  do {                            \
    if (V == 1) DP_RUNS(1, TAPS); \
    else if (V == 2) DP_RUNS(2, TAPS); \
    else DP_RUNS(4, TAPS);        \
  } while (0)
    if (taps == 2) DP_RUNS_BY_V(2);
    else if (taps == 3) DP_RUNS_BY_V(3);
    else DP_RUNS_BY_V(4);
#undef DP_RUNS_BY_V
#undef DP_RUNS
    if (rc) return rc;
  }
  const dim3 grid(inner + (taps > 1 ? n_entries : 0), pieces);
  if (grid.x == 0) return fe_last_error();
  const int rc = wide ? fe_launch_dependent(delta_prepare_kernel<4>, grid, dim3(32 * DP_WARPS), smem, stream, p, inner)
                      : fe_launch_dependent(delta_prepare_kernel<1>, grid, dim3(32 * DP_WARPS), smem, stream, p, inner);
  return rc ? rc : fe_last_error();
}

// ---------------------------------------------------------------------------
// the recurrence
// ---------------------------------------------------------------------------
struct Delta {
  const float* qkv;         // [tokens, channels]
  long long ld;
  int kv_heads, per;        // q/k heads; heads per q/k head
  const float* gates;       // [tokens, heads, 2]
  // chunk-parallel scratch, per (slot, head)
  float* w;                 // [dk][SR_LONG]: W transposed
  float* u;                 // [SR_LONG][dv]: U, then (chain) u
  float* before;            // [dk, dv]: the state before the chunk
  float* decays;            // [SR_LONG + 4]: e^(c_end - c_t) per token, then e^(c_end)

  static constexpr int VECS = 2, SCALARS = 2, EXTRA = 0;
  static constexpr bool SCORES = true, NORMALISER = false;

  __device__ __forceinline__ const float* q_row(const StateRun& p, int head, int token) const {
    return qkv + (size_t)token * ld + (size_t)(head / per) * p.dk;
  }
  __device__ __forceinline__ const float* k_row(const StateRun& p, int head, int token) const {
    return q_row(p, head, token) + (size_t)kv_heads * p.dk;
  }
  __device__ __forceinline__ float beta(const StateRun& p, int head, int token) const { return gates[((size_t)token * p.heads + head) * 2]; }
  __device__ __forceinline__ float log_decay(const StateRun& p, int head, int token) const { return gates[((size_t)token * p.heads + head) * 2 + 1]; }

  __device__ __forceinline__ float* column(const StateRun& p, int slot, int head, int col, size_t* step) const {
    *step = p.dv;
    return p.state + ((size_t)slot * p.heads + head) * p.dk * p.dv + col;
  }
  __device__ __forceinline__ void begin(const StateRun&, int, int, float*) const {}
  __device__ __forceinline__ void end(const StateRun&, int, int, const float*) const {}
  __device__ __forceinline__ void stage(const StateRun& p, int head, int first, int nt, float* vec, int pitch, float* sc) const {
    for (int i = threadIdx.x; i < nt * p.dk; i += blockDim.x) {
      const int t = i / p.dk, d = i - t * p.dk;
      float* dst = vec + t * VECS * pitch + d;
      dst[0] = q_row(p, head, first + t)[d], dst[pitch] = k_row(p, head, first + t)[d];
    }
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
      sc[t * SCALARS] = beta(p, head, first + t);
      sc[t * SCALARS + 1] = expf(log_decay(p, head, first + t));
    }
  }
  template <int KPT>
  __device__ __forceinline__ float step(float (&S)[KPT], const float* vec, int pitch, const float* sc, float value, int s, int ds) const {
    const float *qs = vec + s, *ks = qs + pitch;
    const float g = sc[1];
    float have = 0.f;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      S[i] *= g;
      have = fmaf(S[i], ks[i * ds], have);
    }
    const float u = sc[0] * (value - sr_column_sum(have, ds));
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      S[i] = fmaf(ks[i * ds], u, S[i]);
      acc = fmaf(S[i], qs[i * ds], acc);
    }
    return sr_column_sum(acc, ds);
  }
  __device__ __forceinline__ float scale(const float*, const float*, int) const { return 1.f; }

  // -- chunk form --
  // sums of log g up to the chunk's tokens lane and 32 + lane, by one warp (tokens past the end keep
  // the last sum)
  __device__ __forceinline__ void chunk_sums(const StateRun& p, int head, const ChunkAt& at, double* c) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h) c[h] = lane + 32 * h < at.count ? (double)log_decay(p, head, at.first + lane + 32 * h) : 0.0;
    sr_running_sum(c[0], c[1]);
  }
  __device__ __forceinline__ size_t cell(const StateRun& p, const ChunkAt& at, int head) const { return (size_t)at.slot * p.heads + head; }
  __device__ __forceinline__ Rows queries(const StateRun& p, int head, const ChunkAt& at) const { return Rows{q_row(p, head, at.first), ld}; }
  __device__ __forceinline__ float query_mul() const { return 1.f; }
  __device__ __forceinline__ Rows keys(const StateRun& p, int head, const ChunkAt& at) const { return Rows{k_row(p, head, at.first), ld}; }
  __device__ __forceinline__ Rows others(const StateRun& p, int head, const ChunkAt& at) const {
    return Rows{u + cell(p, at, head) * SR_LONG * p.dv, p.dv};
  }
  __device__ __forceinline__ Rows starts(const StateRun& p, int head, const ChunkAt& at) const {
    return Rows{before + cell(p, at, head) * p.dk * p.dv, p.dv};
  }
  __device__ __forceinline__ void out_begin(const StateRun& p, int head, const ChunkAt& at, double* rt, double* ct, float* ea, float*) const {
    double c[2];
    chunk_sums(p, head, at, c);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = (threadIdx.x & 31) + 32 * h;
      rt[t] = c[h];
      ct[t] = -c[h];
      ea[t] = t < at.count ? expf((float)c[h]) : 0.f;
    }
  }
};

// W and U of one chunk of one head: the triangular system solved for the columns of beta e^c k
// and beta v, sixteen rows at a time.  A block of rows first loses what the rows before it give, then a
// thread per column solves the 16 x 16 triangle in registers and stores the result, also for the blocks
// below.  The products (L itself, and a block's from the rows before it) run on the tensor cores, both
// operands split; what remains is the triangles, one row after the other, and the loads before them.  Solve, chain and
// outputs of 2,048 tokens, 32 heads of 64 channels: 307 us, 371 with tiles of multiply-adds; 3 prompts of 1,000 to 666 tokens,
// heads of 128: 971 and 1,062; outputs' error against 64 bits 1.3e-7 and 1.9e-7, 1.3e-7 and 2.3e-7.
#define DS_THREADS 256
// Columns of the right sides: k in fours, then v, in eights altogether.
__host__ __device__ static inline int ds_columns(int dk, int dv) { return (((dk + 3) & ~3) + dv + 7) & ~7; }
__global__ void __launch_bounds__(DS_THREADS) delta_solve_kernel(const Delta m, const StateRun p) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  ChunkAt at;
  if (!sr_locate(p, &at)) return;
  const int head = blockIdx.x, dk = p.dk, dv = p.dv, tid = threadIdx.x;
  const int v0 = (dk + 3) & ~3, columns = ds_columns(dk, dv), ldx = columns + 8, dk8 = (dk + 7) & ~7;      // columns of k, then of v
  __shared__ double c[SR_LONG];
  __shared__ float bt[SR_LONG], be[SR_LONG];
  float* lt = smem;                          // [SR_LONG columns j][SR_TP rows t]: L transposed
  float* X = lt + SR_LONG * SR_TP;           // [SR_LONG][ldx]
  float* kt = X + SR_LONG * ldx;             // [dk8][SR_TP]; rows past dk are zero
  if (tid < 32) {
    double sums[2];
    m.chunk_sums(p, head, at, sums);
    const double end = __shfl_sync(0xffffffffu, sums[1], 31);
    float* decays = m.decays + m.cell(p, at, head) * (SR_LONG + 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = tid + 32 * h;
      const float beta = t < at.count ? m.beta(p, head, at.first + t) : 0.f;
      c[t] = sums[h];
      bt[t] = beta;
      be[t] = beta * expf((float)sums[h]);
      decays[t] = t < at.count ? expf((float)(end - sums[h])) : 0.f;
    }
    if (tid == 0) decays[SR_LONG] = expf((float)end);
  }
  const Rows keys = m.keys(p, head, at), values{p.v + (size_t)at.first * p.v_ld + (size_t)head * dv, p.v_ld};
  sr_stage_transposed(kt, keys, dk, at.count);
  for (int i = tid; i < (dk8 - dk) * SR_TP; i += DS_THREADS) kt[dk * SR_TP + i] = 0.f;
  __syncthreads();
  // the right sides: rows of beta e^c k and beta v, zero past the last token and between the two
  const int warp = tid >> 5, lane = tid & 31;
  for (int t = warp; t < SR_LONG; t += DS_THREADS / 32) {
    const bool has = t < at.count;
    const float a = be[t], b = bt[t];
    float* x = X + t * ldx;
    for (int d = lane; d < v0; d += 32) x[d] = d < dk ? a * kt[d * SR_TP + t] : 0.f;
    for (int d = lane; d < columns - v0; d += 32) x[v0 + d] = has && d < dv ? b * values.row(t)[d] : 0.f;
  }
  const int fg = lane >> 2, fq = lane & 3;
  {
    const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 16;
    OutTile s;
    s.clear();
    if (n0 <= m0 + 31) s.add(kt + fq * SR_TP + m0 + fg, kt + fq * SR_TP + n0 + fg, SR_TP, dk8);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = m0 + 16 * a + 8 * (i >> 1) + fg, j = n0 + 8 * b + 2 * fq + (i & 1);
          lt[j * SR_TP + t] = j < t ? s.at(a, b, i >> 1, i & 1) * bt[t] * expf((float)(c[t] - c[j])) : 0.f;
        }
  }
  const size_t cell = m.cell(p, at, head);
  for (int r0 = 0; r0 < SR_LONG; r0 += 16) {
    __syncthreads();
    if (r0 > 0) {
      for (int n0 = 8 * warp; n0 < columns; n0 += DS_THREADS / 4) {
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
        const float* l = lt + fq * SR_TP + r0 + fg;
        const float* x = X + fq * ldx + n0 + fg;
#pragma unroll 1
        for (int j = 0; j < r0; j += 16) {
          SplitA fa, fa2;
          SplitB fb, fb2;
          split_load_a(fa, l + j * SR_TP, 1, SR_TP);
          split_load_a(fa2, l + (j + 8) * SR_TP, 1, SR_TP);
          split_load_b(fb, x + j * ldx, ldx);
          split_load_b(fb2, x + (j + 8) * ldx, ldx);
          split_mma(sum, small, fa, fa2, fb, fb2);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float2* x2 = reinterpret_cast<float2*>(X + (r0 + 8 * h + fg) * ldx + n0 + 2 * fq);
          *x2 = make_float2(x2->x - split_join(sum[2 * h], small[2 * h]), x2->y - split_join(sum[2 * h + 1], small[2 * h + 1]));
        }
      }
      __syncthreads();
    }
    for (int i = tid; i < columns; i += DS_THREADS) {
      float x[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) x[t] = X[(r0 + t) * ldx + i];
#pragma unroll
      for (int j = 0; j < 15; ++j) {
        float l[16];
#pragma unroll
        for (int t = 0; t < 16; t += 4)
          if (t + 3 > j) load4(lt + (r0 + j) * SR_TP + r0 + t, l + t);
#pragma unroll
        for (int t = j + 1; t < 16; ++t) x[t] = fmaf(-l[t], x[j], x[t]);
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) X[(r0 + t) * ldx + i] = x[t];
      if (i < dk) {
        float* dst = m.w + (cell * dk + i) * SR_LONG + r0;
#pragma unroll
        for (int t = 0; t < 16; t += 4) store4(dst + t, x + t);
      } else if (i >= v0 && i - v0 < dv) {
        float* dst = m.u + (cell * SR_LONG + r0) * dv + (i - v0);
#pragma unroll
        for (int t = 0; t < 16; ++t) dst[(size_t)t * dv] = x[t];
      }
    }
  }
}

// The chain over an entry's chunks for one head and COLS value columns: u = U - W S, then
// S <- e^(c_end) S + sum_j k_j (e^(c_end - c_j) u_j)^T.  What bounds it is one chunk's two products after the
// other, so they run on the tensor cores with both operands split (mma_split.cuh): a warp takes 16 x 8
// outputs, reads 48 numbers a lane where a 4 x 2 tile of multiply-adds read 192, and a chunk has two
// barriers.  The state's columns stay in registers, as the warps' pieces of the second product, and in shared
// memory for the first; the next chunk's W and keys, and what a lane needs of it besides, are on their way
// while a chunk is worked on.
#define DC_WP (SR_LONG + 8)          // pitches: the rows of a fragment fall into different banks
template <int KD, int COLS>
__global__ void __launch_bounds__(16 * COLS) delta_chain_kernel(const Delta m, const StateRun p, int* status) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  constexpr int KP = 64 * KD + 8, SP = COLS + 8, THREADS = 16 * COLS, WARPS = THREADS / 32;
  const int head = blockIdx.x, entry = blockIdx.y, col0 = blockIdx.z * COLS, tid = threadIdx.x;
  const int first = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - first;
  if (count < p.long_from) return;
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.state_rows) {
    if (tid == 0 && blockIdx.z == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
    return;
  }
  const int dk = p.dk, dv = p.dv, dk8 = (dk + 7) & ~7, half = dk8 * DC_WP + SR_LONG * KP;
  float* S = smem;                           // [64 KD][SP]
  float* us = S + 64 * KD * SP;              // [SR_LONG][SP], weighted
  float* buffers = us + SR_LONG * SP;        // 2 x (W transposed [dk8][DC_WP], keys [SR_LONG][KP])
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int t0 = 16 * (warp & 3) + g, n0 = 8 * (warp >> 2);        // first row and columns of this warp's pieces
  const int col = col0 + n0 + 2 * q;                               // this lane's two columns
  const bool in0 = col < dv, in1 = col + 1 < dv, pair = in1 && (dv & 1) == 0;
  auto load2 = [&](const float* at, float& a, float& b) {
    if (pair) { const float2 x = *reinterpret_cast<const float2*>(at); a = x.x, b = x.y; }
    else { a = in0 ? at[0] : 0.f, b = in1 ? at[1] : 0.f; }
  };
  auto store2 = [&](float* at, float a, float b) {
    if (pair) { *reinterpret_cast<float2*>(at) = make_float2(a, b); }
    else { if (in0) at[0] = a; if (in1) at[1] = b; }
  };
  float* st = p.state + ((size_t)slot * p.heads + head) * dk * dv + col;
  float s[KD][2][2];                         // rows 64 kd + t0, + 8 of the state
#pragma unroll
  for (int kd = 0; kd < KD; ++kd)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int d = 64 * kd + t0 + 8 * h;
      s[kd][h][0] = s[kd][h][1] = 0.f;
      if (d < dk) load2(st + (size_t)d * dv, s[kd][h][0], s[kd][h][1]);
      *reinterpret_cast<float2*>(S + d * SP + n0 + 2 * q) = make_float2(s[kd][h][0], s[kd][h][1]);
    }
  for (int i = tid; i < 2 * half; i += THREADS) buffers[i] = 0.f;      // channels past dk stay zero
  __syncthreads();
  const int chunks = (count + SR_LONG - 1) / SR_LONG;
  const size_t cell0 = (size_t)sr_slot(first, entry, 0) * p.heads + head;
  const Rows keys{m.k_row(p, head, first), m.ld};
  const bool wide = keys.wide(dk);
  auto fetch = [&](int chunk, float* buf) {
    const float* w = m.w + (cell0 + (size_t)chunk * p.heads) * dk * SR_LONG + (tid & 15) * 4;
    float* to = buf + (tid & 15) * 4;
#pragma unroll 4
    for (int d = tid >> 4; d < dk; d += THREADS / 16) sr_copy16(to + d * DC_WP, w + d * SR_LONG);
    const int rows = min(SR_LONG, count - chunk * SR_LONG);
    float* ks = buf + dk8 * DC_WP;
#pragma unroll 4
    for (int t = warp; t < SR_LONG; t += WARPS) {
      float* dst = ks + t * KP;
      if (t >= rows) {
        for (int d = lane; d < dk; d += 32) dst[d] = 0.f;
      } else if (wide) {
        for (int d = 4 * lane; d < dk; d += 128) sr_copy16(dst + d, keys.row(chunk * SR_LONG + t) + d);
      } else {
        for (int d = lane; d < dk; d += 32) sr_copy4(dst + d, keys.row(chunk * SR_LONG + t) + d);
      }
    }
    sr_copy_commit();
  };
  float x[2][2], w[2], keep;                 // U, its weights and the state's decay over the chunk
  auto ask = [&](int chunk) {
    const size_t cell = cell0 + (size_t)chunk * p.heads;
    const float* decays = m.decays + cell * (SR_LONG + 4);
    keep = decays[SR_LONG];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      w[h] = decays[t0 + 8 * h];
      load2(m.u + (cell * SR_LONG + t0 + 8 * h) * dv + col, x[h][0], x[h][1]);
    }
  };
  fetch(0, buffers);
  ask(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const size_t cell = cell0 + (size_t)chunk * p.heads;
    const float* buf = buffers + (chunk & 1) * half;
    if (chunk + 1 == chunks) pdl_trigger();    // state_out's blocks would only lie beside this one's till then
    sr_copy_wait<0>();
    __syncthreads();           // this chunk's tiles have landed, the state is whole; everyone is done with the other buffer
    if (chunk + 1 < chunks) fetch(chunk + 1, buffers + ((chunk + 1) & 1) * half);
    // the state before the chunk, for state_out
    float* before = m.before + cell * dk * dv + col;
#pragma unroll
    for (int kd = 0; kd < KD; ++kd)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int d = 64 * kd + t0 + 8 * h;
        if (d < dk) store2(before + (size_t)d * dv, s[kd][h][0], s[kd][h][1]);
      }
    {
      float sum[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
      const float* a = buf + q * DC_WP + t0;
      const float* b = S + q * SP + n0 + g;
#pragma unroll 8
      for (int d = 0; d < dk8; d += 8) {
        SplitA fa;
        SplitB fb;
        split_load_a(fa, a + d * DC_WP, 1, DC_WP);
        split_load_b(fb, b + d * SP, SP);
        split_mma(sum, small, fa, fb);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        x[h][0] -= split_join(sum[2 * h], small[2 * h]);
        x[h][1] -= split_join(sum[2 * h + 1], small[2 * h + 1]);
        *reinterpret_cast<float2*>(us + (t0 + 8 * h) * SP + n0 + 2 * q) = make_float2(x[h][0] * w[h], x[h][1] * w[h]);
        store2(m.u + (cell * SR_LONG + t0 + 8 * h) * dv + col, x[h][0], x[h][1]);
      }
    }
    const float decay = keep;
    __syncthreads();
    if (chunk + 1 < chunks) ask(chunk + 1);
    const float* b = us + q * SP + n0 + g;
#pragma unroll
    for (int kd = 0; kd < KD; ++kd) {
      float sum[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
      const float* a = buf + dk8 * DC_WP + q * KP + 64 * kd + t0;
#pragma unroll
      for (int t = 0; t < SR_LONG; t += 8) {
        SplitA fa;
        SplitB fb;
        split_load_a(fa, a + t * KP, 1, KP);
        split_load_b(fb, b + t * SP, SP);
        split_mma(sum, small, fa, fb);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        s[kd][h][0] = fmaf(decay, s[kd][h][0], split_join(sum[2 * h], small[2 * h]));
        s[kd][h][1] = fmaf(decay, s[kd][h][1], split_join(sum[2 * h + 1], small[2 * h + 1]));
        *reinterpret_cast<float2*>(S + (64 * kd + t0 + 8 * h) * SP + n0 + 2 * q) = make_float2(s[kd][h][0], s[kd][h][1]);
      }
    }
  }
#pragma unroll
  for (int kd = 0; kd < KD; ++kd)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int d = 64 * kd + t0 + 8 * h;
      if (d < dk) store2(st + (size_t)d * dv, s[kd][h][0], s[kd][h][1]);
    }
}

static size_t delta_solve_smem(int dk, int dv) {
  return sizeof(float) * ((size_t)SR_LONG * SR_TP + (size_t)SR_LONG * (ds_columns(dk, dv) + 8) + (size_t)(dk + 7) / 8 * 8 * SR_TP);
}
// Value columns of a block of delta_chain: few where the heads are small, so that there are more blocks.
static int delta_chain_cols(int dv) { return dv <= 64 ? 16 : 32; }
static size_t delta_chain_smem(int dk, int cols) {
  const size_t kp = (size_t)(dk + 63) / 64 * 64, dk8 = (size_t)(dk + 7) / 8 * 8, sp = cols + 8;
  return sizeof(float) * ((kp + SR_LONG) * sp + 2 * (dk8 * DC_WP + SR_LONG * (kp + 8)));
}
// Keys of up to 176 numbers with 16 columns a block and up to 152 with 32: what shared memory holds of a chunk and the
// next one.  (The instantiations would reach 192.)
static bool delta_chunk_takes(int dk, int dv) {
  return dk <= 192 && chunk_takes(dk, dv, true) && delta_solve_smem(dk, dv) <= 218 * 1024 &&
         delta_chain_smem(dk, delta_chain_cols(dv)) <= 226 * 1024;
}

FE_EXPORT long long fe_delta_rule_scratch(int tokens, int entries, int heads, int dk, int dv, int max_new) {
  const long long need = walk_in_stretches(dk, dv, 0) ? (long long)tokens * heads * dv : 0;
  if (max_new < SR_LONG_FROM || !delta_chunk_takes(dk, dv)) return need;
  return (need + 3) / 4 * 4 + sr_slots(tokens, entries) * heads * ((long long)dk * SR_LONG + (long long)SR_LONG * dv + (long long)dk * dv + SR_LONG + 4);
}

FE_EXPORT int fe_delta_rule(const float* qkv, long long ld, const float* gates, const float* gate, long long gate_ld,
                            const float* norm_w, float eps, float* state, int state_rows, const int* slots,
                            const int* cu_tokens, void* out, int out_dtype, int entries, int kv_heads, int heads, int dk, int dv,
                            int tokens, int max_new, float* scratch, int* status, cudaStream_t stream) {
  if (entries <= 0 || tokens <= 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads || dk < 1 || dv < 1 || heads > 65535 || entries > 65535) return FE_ERR_BAD_SHAPE;
  StateRun p{state, state_rows, slots, cu_tokens, heads, dk, dv, 0, qkv + 2 * kv_heads * dk, ld, norm_w, 0, gate, gate_ld, 0, eps, out, nullptr, 0};
  Delta m{qkv, ld, kv_heads, heads / kv_heads, gates, nullptr, nullptr, nullptr, nullptr};
  if (walk_in_stretches(dk, dv, 0)) {
    p.raw = scratch;
    scratch = scratch ? scratch + ((size_t)tokens * heads * dv + 3) / 4 * 4 : nullptr;
  }
  const bool chunked = max_new >= SR_LONG_FROM && scratch != nullptr && delta_chunk_takes(dk, dv);
  if (chunked) p.long_from = SR_LONG_FROM;
  int rc = launch_walk(m, p, out_dtype, entries, tokens, status, stream);
  if (rc || !chunked) return rc ? rc : fe_last_error();
  const int chunks = (max_new + SR_LONG - 1) / SR_LONG;
  if (chunks > 65535) return FE_ERR_TOO_LARGE;
  const size_t cells = (size_t)sr_slots(tokens, entries) * heads;
  m.w = scratch;
  m.u = m.w + cells * dk * SR_LONG;
  m.decays = m.u + cells * SR_LONG * dv;
  m.before = m.decays + cells * (SR_LONG + 4);
  size_t smem = delta_solve_smem(dk, dv);
  cudaFuncSetAttribute(delta_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  rc = fe_launch_dependent(delta_solve_kernel, dim3(heads, entries, chunks), dim3(DS_THREADS), smem, stream, m, p);
  if (rc) return rc;
  // delta_chain is not launched as a dependent: its blocks, fewer than the SMs or not many more, would take their
  // places while delta_solve's last blocks leave theirs, two on one SM and none on the next (measured with two tf32
  // numbers an operand: 143 us for a chain over 2,048 tokens that took 102 us spread evenly).
  const int cols = delta_chain_cols(dv);
  smem = delta_chain_smem(dk, cols);
  const dim3 chain(heads, entries, (dv + cols - 1) / cols);
#define DC_LAUNCH(KD, COLS)                                                                                       \
  do {                                                                                                            \
    cudaFuncSetAttribute(delta_chain_kernel<KD, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    delta_chain_kernel<KD, COLS><<<chain, 16 * COLS, smem, stream>>>(m, p, status);                               \
    rc = fe_last_error();                                                                                         \
  } while (0)
#define DC_BY_DK(COLS)                 \
  do {                                 \
    if (dk <= 64) DC_LAUNCH(1, COLS);  \
    else if (dk <= 128) DC_LAUNCH(2, COLS); \
    else DC_LAUNCH(3, COLS);           \
  } while (0)
  if (cols == 16) DC_BY_DK(16);
  else DC_BY_DK(32);
#undef DC_BY_DK
#undef DC_LAUNCH
  if (rc) return rc;
  rc = launch_out(m, p, out_dtype, entries, chunks, stream);
  return rc ? rc : fe_last_error();
}

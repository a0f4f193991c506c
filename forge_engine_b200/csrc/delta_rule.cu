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

// An entry's edge: its first taps - 1 tokens, then the state for the next step.
template <int V>
__device__ __forceinline__ void delta_prepare_edge(const DeltaPrepare& p, int entry, int r, float* buf) {
  const int back = p.taps - 1, lane = threadIdx.x & 31, rows = 2 * p.kv_heads + p.heads;
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

template <int V>
__global__ void __launch_bounds__(32 * DP_WARPS) delta_prepare_kernel(DeltaPrepare p, int inner) {
  extern __shared__ __align__(16) float smem[];      // [DP_WARPS][dk]
  pdl_trigger();
  pdl_wait();
  const int back = p.taps - 1, warp = threadIdx.x >> 5;
  const int r = blockIdx.y * DP_WARPS + warp, rows = 2 * p.kv_heads + p.heads;
  float* buf = smem + warp * p.dk;
  if ((int)blockIdx.x < inner) {
    // a token with all its taps inside the step
    const int t = blockIdx.x;
    if (t - p.cu_tokens[p.token_entry[t]] < back) return;
    if (r < rows) delta_prepare_row<V>(p, t, r, buf, [&](int j) { return p.proj + (size_t)(t - j) * p.ld; });
    if (blockIdx.y == 0) delta_prepare_gates(p, t);
    return;
  }
  delta_prepare_edge<V>(p, blockIdx.x - inner, r, buf);
}

// Tokens with all their taps inside the step, DP_RUN of them in a row by a warp for one q, k or v head of
// at most 32 V elements: every input is read once instead of once per tap.  Bound by the bytes in and out
// (2,048 tokens of 4,096 channels: 67 us with a warp per token and head; this way 24 us and 14 us for the entry's edge behind
// them, 25 us with the edges' blocks, the first n_entries, beside them).
#define DP_RUN 16
template <int V, int TAPS>
__global__ void __launch_bounds__(32 * DP_WARPS) delta_prepare_run_kernel(DeltaPrepare p, int n_entries, int wide) {
  extern __shared__ __align__(16) float smem[];      // [DP_WARPS][dk]
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.y * DP_WARPS + warp;
  if ((int)blockIdx.x < n_entries) {
    if (wide) delta_prepare_edge<4>(p, blockIdx.x, r, smem + warp * p.dk);
    else delta_prepare_edge<1>(p, blockIdx.x, r, smem + warp * p.dk);
    return;
  }
  const int t0 = (blockIdx.x - n_entries) * DP_RUN, end = min(p.n_tokens, t0 + DP_RUN);
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
  // many tokens: runs of them, and the entries' edges beside them.  Below 256 tokens there are too few runs to
  // fill the machine, and a block per token starts all at once.
  const int most = dk > dv ? dk : dv, V = most <= 32 ? 1 : most <= 64 ? 2 : 4;
  if (n_tokens >= 256 && taps >= 2 && taps <= 4 && most <= 128 && (V == 1 || wide || (V == 2 && dk % 2 == 0 && dv % 2 == 0 && ld % 2 == 0 &&
      (((uintptr_t)proj | (uintptr_t)conv | (uintptr_t)out) & 7) == 0))) {
    const dim3 runs(n_entries + (n_tokens + DP_RUN - 1) / DP_RUN, pieces);
    int rc = 0;
#define DP_RUNS(V_, TAPS) \
  rc = fe_launch_dependent(delta_prepare_run_kernel<V_, TAPS>, runs, dim3(32 * DP_WARPS), smem, stream, p, n_entries, (int)wide)
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
    return rc ? rc : fe_last_error();
  }
  const dim3 grid(n_tokens + (taps > 1 ? n_entries : 0), pieces);
  if (grid.x == 0) return fe_last_error();
  const int rc = wide ? fe_launch_dependent(delta_prepare_kernel<4>, grid, dim3(32 * DP_WARPS), smem, stream, p, n_tokens)
                      : fe_launch_dependent(delta_prepare_kernel<1>, grid, dim3(32 * DP_WARPS), smem, stream, p, n_tokens);
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
  bf16* w;                  // tiles of W transposed, split in three (mma_split.cuh); rows past dk are zero
  bf16* k;                  // tiles of keys, split; of the first head of those that share them
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

// A tile of the chain, as it lies in memory and in shared memory: three planes of W transposed [dk16][DC_WP] or of keys
// [SR_LONG][dk16 + 8]; the pitches let the rows of a matrix fall into different banks.
#define DC_WP (SR_LONG + 8)
__host__ __device__ static constexpr int dc_tile(int dk16) { return dk16 * DC_WP > SR_LONG * (dk16 + 8) ? dk16 * DC_WP : SR_LONG * (dk16 + 8); }

// W and U of one chunk of one head: the triangular system solved for the columns of beta e^c k
// and beta v, sixteen rows at a time.  A block of rows first loses what the rows before it give, then a
// thread per column solves the 16 x 16 triangle in registers and stores the result, also for the blocks
// below.  The products (L itself, and a block's from the rows before it) run on the tensor cores, both
// operands split; what remains is the triangles, one row after the other, and the loads before them.  Solve, chain and
// outputs of 2,048 tokens, 32 heads of 64 channels: 214 us (307 before a warp's loads of the values went out together, W was
// split here for the chain and sizes of 64 and 128 were known when compiled), 371 with tiles of multiply-adds; 3 prompts of 1,000 to 666 tokens,
// heads of 128: 971 and 1,062; outputs' error against 64 bits 1.3e-7 and 1.9e-7, 1.3e-7 and 2.3e-7.
#define DS_THREADS 256
// Columns of the right sides: k in fours, then v, in eights altogether.
__host__ __device__ static inline int ds_columns(int dk, int dv) { return (((dk + 3) & ~3) + dv + 7) & ~7; }
template <int D>       // head sizes of both sides known when compiled; 0: any
__global__ void __launch_bounds__(DS_THREADS) delta_solve_kernel(const Delta m, const StateRun p) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  ChunkAt at;
  if (!sr_locate(p, &at)) return;
  const int head = blockIdx.x, dk = D ? D : p.dk, dv = D ? D : p.dv, tid = threadIdx.x;
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
  constexpr int ROWS = SR_LONG * 32 / DS_THREADS;       // of a warp: their loads are all on their way before the first is used
  for (int d = lane; d < columns - v0; d += 32) {
    float x[ROWS];
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int t = warp + u * (DS_THREADS / 32);
      x[u] = t < at.count && d < dv ? values.row(t)[d] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int t = warp + u * (DS_THREADS / 32);
      X[t * ldx + v0 + d] = bt[t] * x[u];
    }
  }
  for (int t = warp; t < SR_LONG; t += DS_THREADS / 32)
    for (int d = lane; d < v0; d += 32) X[t * ldx + d] = d < dk ? be[t] * kt[d * SR_TP + t] : 0.f;
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
  const int dk16 = (dk + 15) & ~15, tile = dc_tile(dk16);
  if (head % m.per == 0) {
    const int pairs = dk16 >> 1;
    bf16* dst = m.k + cell * 3 * tile;
    for (int i = tid; i < SR_LONG * pairs; i += DS_THREADS) {
      const int t = i / pairs, d = 2 * (i - t * pairs);
      planes_store2(dst + t * (dk16 + 8) + d, tile, d < dk8 ? kt[d * SR_TP + t] : 0.f, d < dk8 ? kt[(d + 1) * SR_TP + t] : 0.f);
    }
  }
  for (int i = tid; i < 3 * (dk16 - dk) * SR_LONG; i += DS_THREADS) {
    const int part = i / ((dk16 - dk) * SR_LONG), r = (i / SR_LONG) % (dk16 - dk);
    m.w[(cell * 3 + part) * tile + (dk + r) * DC_WP + i % SR_LONG] = __float2bfloat16_rn(0.f);
  }
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
        bf16* dst = m.w + cell * 3 * tile + i * DC_WP + r0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 part[3];
          split_pair(x[8 * h], x[8 * h + 1], part[0].x, part[1].x, part[2].x);
          split_pair(x[8 * h + 2], x[8 * h + 3], part[0].y, part[1].y, part[2].y);
          split_pair(x[8 * h + 4], x[8 * h + 5], part[0].z, part[1].z, part[2].z);
          split_pair(x[8 * h + 6], x[8 * h + 7], part[0].w, part[1].w, part[2].w);
#pragma unroll
          for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(dst + u * tile + 8 * h) = part[u];
        }
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
// outputs.  delta_solve has split W and the keys, which the blocks of a head's columns all read; the state and the
// weighted u are split once by the lanes that hold them.  2,048 tokens, 32 heads of 64: 127 us with every warp
// splitting what it multiplied, 96 us with split tiles, 58 us with whole copies of them and sizes known when compiled.  The state's columns stay in registers, as the warps' pieces of the
// second product, and in shared memory for the first.  Tiles (W and keys of each chunk in turn) go round SLOTS places: the next
// SLOTS - 1 are on their way while one is worked on.
template <int KD, int COLS, int SLOTS, bool WHOLE>
__global__ void __launch_bounds__(16 * COLS) delta_chain_kernel(const Delta m, const StateRun p, int* status) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  constexpr int SP = COLS + 8, THREADS = 16 * COLS;
  const int head = blockIdx.x, entry = blockIdx.y, col0 = blockIdx.z * COLS, tid = threadIdx.x;
  const int first = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - first;
  if (count < p.long_from) return;
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.state_rows) {
    if (tid == 0 && blockIdx.z == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
    return;
  }
  const int dk = WHOLE ? 64 * KD : p.dk, dv = p.dv, dk16 = (dk + 15) & ~15, KP = dk16 + 8, tile = dc_tile(dk16);
  bf16* S = reinterpret_cast<bf16*>(smem);   // [3][dk16][SP]
  bf16* us = S + 3 * dk16 * SP;              // [3][SR_LONG][SP], weighted
  bf16* tiles = us + 3 * SR_LONG * SP;       // SLOTS x 3 planes: W transposed [dk16][DC_WP] or keys [SR_LONG][KP]
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int m0 = 16 * (warp & 3), t0 = m0 + g, n0 = 8 * (warp >> 2);        // first row and columns of this warp's pieces
  const int col = col0 + n0 + 2 * q;                               // this lane's two columns
  const bool in0 = WHOLE || col < dv, in1 = WHOLE || col + 1 < dv, pair = WHOLE || (in1 && (dv & 1) == 0);
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
      if (d < dk16) planes_store2(S + d * SP + n0 + 2 * q, dk16 * SP, s[kd][h][0], s[kd][h][1]);
    }
  const int chunks = (count + SR_LONG - 1) / SR_LONG;
  const size_t cell0 = (size_t)sr_slot(first, entry, 0) * p.heads + head, group0 = cell0 - head % m.per;
  auto fetch = [&](int i) {                  // tile i: W of chunk i / 2, or its keys
    if (i < 2 * chunks) {
      bf16* to = tiles + (i % SLOTS) * 3 * tile;
      const size_t step = (size_t)(i >> 1) * p.heads;
      const bf16* from = (i & 1) == 0 ? m.w + (cell0 + step) * 3 * tile : m.k + (group0 + step) * 3 * tile;
#pragma unroll 4
      for (int at = tid * 8; at < 3 * tile; at += THREADS * 8) sr_copy16(to + at, from + at);
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
#pragma unroll
  for (int i = 0; i + 1 < SLOTS; ++i) fetch(i);
  ask(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const size_t cell = cell0 + (size_t)chunk * p.heads;
    if (chunk + 1 == chunks) pdl_trigger();    // state_out's blocks would only lie beside this one's till then
    sr_copy_wait<SLOTS - 2>();
    __syncthreads();           // W has landed, the state is whole; everyone is done with the keys before
    fetch(2 * chunk + SLOTS - 1);
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
      float sum[4] = {}, small[5][4] = {};
      const bf16* a = tiles + (2 * chunk % SLOTS) * 3 * tile + m0;
      const bf16* b = S + n0;
#pragma unroll 4
      for (int d = 0; d < dk16; d += 16) {
        PlanesA fa;
        PlanesB fb;
        planes_load_a_by_k(fa, a + d * DC_WP, DC_WP, tile);
        planes_load_b_by_k(fb, b + d * SP, SP, dk16 * SP);
        split_mma(sum, small, fa, fb);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        x[h][0] -= split_join(sum[2 * h], small, 2 * h);
        x[h][1] -= split_join(sum[2 * h + 1], small, 2 * h + 1);
        planes_store2(us + (t0 + 8 * h) * SP + n0 + 2 * q, SR_LONG * SP, x[h][0] * w[h], x[h][1] * w[h]);
        store2(m.u + (cell * SR_LONG + t0 + 8 * h) * dv + col, x[h][0], x[h][1]);
      }
    }
    const float decay = keep;
    sr_copy_wait<SLOTS - 2>();
    __syncthreads();           // the keys have landed, u is whole; everyone is done with W
    fetch(2 * chunk + SLOTS);
    if (chunk + 1 < chunks) ask(chunk + 1);
    const bf16* a = tiles + ((2 * chunk + 1) % SLOTS) * 3 * tile + m0;
#pragma unroll
    for (int kd = 0; kd < KD; ++kd) {
      if (64 * kd + m0 >= dk16) break;
      float sum[4] = {}, small[5][4] = {};
#pragma unroll
      for (int t = 0; t < SR_LONG; t += 16) {
        PlanesA fa;
        PlanesB fb;
        planes_load_a_by_k(fa, a + t * KP + 64 * kd, KP, tile);
        planes_load_b_by_k(fb, us + t * SP + n0, SP, SR_LONG * SP);
        split_mma(sum, small, fa, fb);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        s[kd][h][0] = fmaf(decay, s[kd][h][0], split_join(sum[2 * h], small, 2 * h));
        s[kd][h][1] = fmaf(decay, s[kd][h][1], split_join(sum[2 * h + 1], small, 2 * h + 1));
        planes_store2(S + (64 * kd + t0 + 8 * h) * SP + n0 + 2 * q, dk16 * SP, s[kd][h][0], s[kd][h][1]);
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
// Places of its ring of tiles: what shared memory holds of the next chunk.
static int delta_chain_slots(int dk) { return dk <= 64 ? 4 : dk <= 128 ? 3 : 2; }
static size_t delta_chain_smem(int dk, int cols) {
  const int dk16 = (dk + 15) & ~15;
  return sizeof(bf16) * 3 * ((size_t)(dk16 + SR_LONG) * (cols + 8) + (size_t)delta_chain_slots(dk) * dc_tile(dk16));
}
// Keys of up to 176 numbers with 16 columns a block and up to 152 with 32; longer ones are walked.
static bool delta_chunk_takes(int dk, int dv) {
  return dk <= (delta_chain_cols(dv) == 16 ? 176 : 152) && chunk_takes(dk, dv, true) && delta_solve_smem(dk, dv) <= 218 * 1024 &&
         delta_chain_smem(dk, delta_chain_cols(dv)) <= 226 * 1024;
}

FE_EXPORT long long fe_delta_rule_scratch(int tokens, int entries, int heads, int dk, int dv, int max_new) {
  const long long need = walk_in_stretches(dk, dv, 0) ? (long long)tokens * heads * dv : 0;
  if (max_new < SR_LONG_FROM || !delta_chunk_takes(dk, dv)) return need;
  return (need + 3) / 4 * 4 + sr_slots(tokens, entries) * heads *
             (3LL * dc_tile((dk + 15) / 16 * 16) + (long long)SR_LONG * dv + (long long)dk * dv + SR_LONG + 4);
}

FE_EXPORT int fe_delta_rule(const float* qkv, long long ld, const float* gates, const float* gate, long long gate_ld,
                            const float* norm_w, float eps, float* state, int state_rows, const int* slots,
                            const int* cu_tokens, void* out, int out_dtype, int entries, int kv_heads, int heads, int dk, int dv,
                            int tokens, int max_new, float* scratch, int* status, cudaStream_t stream) {
  if (entries <= 0 || tokens <= 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads || dk < 1 || dv < 1 || heads > 65535 || entries > 65535) return FE_ERR_BAD_SHAPE;
  StateRun p{state, state_rows, slots, cu_tokens, heads, dk, dv, 0, qkv + 2 * kv_heads * dk, ld, norm_w, 0, gate, gate_ld, 0, eps, out, nullptr, 0};
  Delta m{qkv, ld, kv_heads, heads / kv_heads, gates, nullptr, nullptr, nullptr, nullptr, nullptr};
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
  const size_t planes = cells * 3 * dc_tile((dk + 15) / 16 * 16);
  m.w = reinterpret_cast<bf16*>(scratch);
  m.k = m.w + planes;
  m.u = scratch + planes;
  m.decays = m.u + cells * SR_LONG * dv;
  m.before = m.decays + cells * (SR_LONG + 4);
  size_t smem = delta_solve_smem(dk, dv);
  const auto solve = dk == 64 && dv == 64 ? delta_solve_kernel<64> : dk == 128 && dv == 128 ? delta_solve_kernel<128> : delta_solve_kernel<0>;
  cudaFuncSetAttribute(solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  rc = fe_launch_dependent(solve, dim3(heads, entries, chunks), dim3(DS_THREADS), smem, stream, m, p);
  if (rc) return rc;
  // delta_chain is not launched as a dependent: its blocks, fewer than the SMs or not many more, would take their
  // places while delta_solve's last blocks leave theirs, two on one SM and none on the next (measured with two tf32
  // numbers an operand: 143 us for a chain over 2,048 tokens that took 102 us spread evenly).
  const int cols = delta_chain_cols(dv);
  smem = delta_chain_smem(dk, cols);
  const dim3 chain(heads, entries, (dv + cols - 1) / cols);
#define DC_LAUNCH_AS(KD, COLS, SLOTS, WHOLE)                                                                                  \
  do {                                                                                                                        \
    cudaFuncSetAttribute(delta_chain_kernel<KD, COLS, SLOTS, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    delta_chain_kernel<KD, COLS, SLOTS, WHOLE><<<chain, 16 * COLS, smem, stream>>>(m, p, status);                             \
    rc = fe_last_error();                                                                                                     \
  } while (0)
  // sizes that fill the warps' pieces: places and bounds known when compiled (2,048 tokens, 32 heads of 64: 96 us, 58 so)
#define DC_LAUNCH(KD, COLS, SLOTS)                                               \
  do {                                                                           \
    if (dk == 64 * KD && dv % COLS == 0) DC_LAUNCH_AS(KD, COLS, SLOTS, true);    \
    else DC_LAUNCH_AS(KD, COLS, SLOTS, false);                                   \
  } while (0)
#define DC_BY_DK(COLS)                       \
  do {                                       \
    if (dk <= 64) DC_LAUNCH(1, COLS, 4);     \
    else if (dk <= 128) DC_LAUNCH(2, COLS, 3); \
    else DC_LAUNCH_AS(3, COLS, 2, false);    \
  } while (0)
  if (cols == 16) DC_BY_DK(16);
  else DC_BY_DK(32);
#undef DC_BY_DK
#undef DC_LAUNCH
#undef DC_LAUNCH_AS
  if (rc) return rc;
  rc = launch_out(m, p, out_dtype, entries, chunks, stream);
  return rc ? rc : fe_last_error();
}

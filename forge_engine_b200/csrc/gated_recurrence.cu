// Linear attention whose forget gate also decides what is written (a gated linear recurrence).
//
// Per head a 32-bit state S [dk, dv]:
//     S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T,      o_t = S_t^T q_t,
//     q = silu(zq),  f = l + (1 - l) sigmoid(zf + b),
// zq, zf, v being columns of one 32-bit projection, l a learned lower bound and b a bias per
// head and channel.  o_t is divided by its root mean square over the head's dv values (eps
// inside the root) and multiplied by one weight vector that all heads share.
//
// gated_recurrence - one block per (head, entry) walks the entry's tokens in order, from and
//   to the request's state row.  Thread (v, s) keeps the rows d = i * DS + s of column v of
//   the state in registers; the DS threads of a column sit side by side in a warp and add
//   their shares of o_t[v] in a butterfly.  Tokens come in chunks of up to 16: all threads
//   first turn the chunk's projections into q, f and v in shared memory (the exponentials
//   run side by side there, not inside the chain), then the chain of the chunk's tokens runs
//   without a block-wide barrier, then a warp per token takes the norm and stores the row.
//   A prompt portion and a single decoded token take the same path; the state is carried in
//   32-bit, and the order of additions depends on dk and DS alone, so how a sequence is cut
//   into steps and what else is in the batch change nothing.  With `long_from` > 0 it leaves
//   entries of that many tokens or more to the three kernels below.
//
// Long entries (prompt portions) run in chunks of 64 tokens side by side, which is exact for a linear
// recurrence: with k_t = 1 - f_t, D(t, s) the product of the forget gates after s up to t, and D(t) that
// from the chunk's first token up to t,
//     o_t = (q_t D(t))^T S_start + sum_{s <= t} A_ts v_s,   A_ts = sum_d q_t D(t, s) k_s,
//     S_end = D(end) S_start + sum_s (D(end, s) k_s) v_s^T.
// gated_recurrence_chunk  - per head and chunk: q_t D(t), A, the chunk's own end state and D(end).
//   The chunk is cut into four sub-chunks of 16 tokens.  Inside one, the 16 x 16 products D(t, s) k_s are
//   built up token by token; between two, D splits into the product from the later one's start up to t,
//   the whole gates of the sub-chunks in between, and the product after s up to the earlier one's end,
//   so that A becomes small matrix products.
// gated_recurrence_scan   - one thread per state element walks the entry's chunks in order: S_start of
//   every chunk (in the place of its end state), and the request's state row after the last.
// gated_recurrence_finish - per chunk [q D | A] [S_start; V] as one 32-bit product from shared memory,
//   then the head's norm and the store.
// All factors are products of gates: there is no division by a decay anywhere (a gate may be as small
// as its lower bound allows), and everything stays 32-bit; against the token-by-token walk only the order
// of additions differs.  What a token costs is 2 dk dv multiply-adds (the walk takes five operations per state
// element and reads two operands of each from shared memory); the products run on the tensor cores with
// both operands split (mma_split.cuh), because the multiply-add units are bound by what shared memory
// delivers to them long before their own rate.
#include "mma_split.cuh"

#define GR_CHUNK 16
#define GR_MAX_KPT 32

struct GatedRecurrence {
  const float* proj;      // [tokens, ld]
  long long ld;
  int q_off, f_off, v_off;
  const float* f_bias;    // [heads * dk] or null
  const float* lower;     // [heads * dk]
  const float* norm_w;    // [dv]
  float eps;
  float* state;           // [rows, heads, dk, dv]
  int state_rows;
  const int* slots;       // [entries]
  const int* cu_tokens;   // [entries + 1]
  void* out;              // [tokens, heads * dv]
  int heads, dk, dv, ds, kpt;
  int long_from;          // above zero: entries of this many tokens or more belong to the chunk-parallel kernels
  // scratch of the chunk-parallel kernels (32-bit)
  int dkp;                // dk rounded up to fours; the added channels are zero
  float* qb;              // [tokens, heads, dkp]
  float* within;          // [chunk slots, heads, 64, 64]: A
  float* chunk_state;     // [chunk slots, heads, dk, dv]: the chunk's own end state, then (scan) its start state
  float* chunk_decay;     // [chunk slots, heads, dk]
};

#define GR_LONG_CHUNK 64
// Chunk c of entry e has a slot of its own: the entries' first tokens are at least a chunk's
// tokens apart per chunk, so floor(first / chunk) + e + c never repeats.
__device__ __forceinline__ int gr_chunk_slot(int first, int entry, int chunk) { return first / GR_LONG_CHUNK + entry + chunk; }

__device__ __forceinline__ void gr_copy16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gr_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void gr_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }
__device__ __forceinline__ void gr_store2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void gr_store2(bf16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }
__device__ __forceinline__ float gr_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

template <typename TO, int KPT>
__global__ void __launch_bounds__(1024) gated_recurrence_kernel(GatedRecurrence p, int* status) {
  extern __shared__ float smem[];
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x, entry = blockIdx.y;
  const int first = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - first;
  if (count <= 0 || (p.long_from > 0 && count >= p.long_from)) return;
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.state_rows) {
    if (threadIdx.x == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
    return;
  }
  const int dk = p.dk, dv = p.dv, DS = p.ds, kpt = p.kpt;
  float* fs = smem;                       // [GR_CHUNK][dk]
  float* qs = fs + GR_CHUNK * dk;         // [GR_CHUNK][dk]
  float* vs = qs + GR_CHUNK * dk;         // [GR_CHUNK][dv]
  float* os = vs + GR_CHUNK * dv;         // [GR_CHUNK][dv]
  const int tid = threadIdx.x;
  const int v = tid / DS, s = tid - v * DS;
  const bool live = v < dv;
  float* st = p.state + (((size_t)slot * p.heads + head) * dk) * dv;
  float S[KPT];
#pragma unroll
  for (int i = 0; i < KPT; ++i) S[i] = (live && i < kpt) ? st[(size_t)(i * DS + s) * dv + v] : 0.f;
  const float* bias = p.f_bias ? p.f_bias + head * dk : nullptr;
  const float* low = p.lower + head * dk;
  const int warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;

  for (int c0 = 0; c0 < count; c0 += GR_CHUNK) {
    const int nt = min(GR_CHUNK, count - c0);
    for (int idx = tid; idx < nt * dk; idx += blockDim.x) {
      const int t = idx / dk, d = idx - t * dk;
      const float* row = p.proj + (size_t)(first + c0 + t) * p.ld;
      const float zq = row[p.q_off + head * dk + d];
      const float zf = row[p.f_off + head * dk + d] + (bias ? bias[d] : 0.f);
      const float l = low[d];
      qs[idx] = zq * gr_sigmoid(zq);
      fs[idx] = l + (1.f - l) * gr_sigmoid(zf);
    }
    for (int idx = tid; idx < nt * dv; idx += blockDim.x) {
      const int t = idx / dv, c = idx - t * dv;
      vs[idx] = p.proj[(size_t)(first + c0 + t) * p.ld + p.v_off + head * dv + c];
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      const float vv = live ? vs[t * dv + v] : 0.f;
      const float* ft = fs + t * dk + s;
      const float* qt = qs + t * dk + s;
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        if (i < kpt) {
          const float f = ft[i * DS];
          S[i] = fmaf(f, S[i], (1.f - f) * vv);
          acc = fmaf(S[i], qt[i * DS], acc);
        }
      }
      for (int o = DS >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (live && s == 0) os[t * dv + v] = acc;
    }
    __syncthreads();
    for (int t = warp; t < nt; t += warps) {
      float ss = 0.f;
      for (int c = lane; c < dv; c += 32) ss = fmaf(os[t * dv + c], os[t * dv + c], ss);
      const float inv = 1.f / sqrtf(warp_sum(ss) / (float)dv + p.eps);
      TO* dst = (TO*)p.out + (size_t)(first + c0 + t) * p.heads * dv + (size_t)head * dv;
      for (int c = lane; c < dv; c += 32) dst[c] = from_float<TO>(os[t * dv + c] * inv * p.norm_w[c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < KPT; ++i)
    if (live && i < kpt) st[(size_t)(i * DS + s) * dv + v] = S[i];
}


#define GR_SUB 16                                // tokens of a sub-chunk
#define GR_SUBS (GR_LONG_CHUNK / GR_SUB)
#define GR_SLICE 128                             // channels (or columns) worked on at a time
#define GR_AP (GR_LONG_CHUNK + 4)

// Sums of the last N of 16 values over the lanes of a warp; lane l gets the sum of value 16 - N + l N / 32.
template <int N>
__device__ __forceinline__ float gr_sums(float (&x)[16], int lane) {
  constexpr int FROM = 16 - N;
  int bit = 16;
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1, bit >>= 1) {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int i = FROM; i < FROM + half; ++i) {
      const float send = upper ? x[i] : x[i + half], keep = upper ? x[i + half] : x[i];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
#pragma unroll
  for (int b = 16 / N; b > 0; b >>= 1) x[FROM] += __shfl_xor_sync(0xffffffffu, x[FROM], b);
  return x[FROM];
}

// R neighbouring channels of a lane: products in pairs.
template <int R> struct GrChannels {
  static constexpr int PAIRS = R / 2;
  uint64_t v[PAIRS];
  __device__ __forceinline__ void load(const float* p) {
    if constexpr (R == 4) { const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(p); v[0] = x.x, v[1] = x.y; }
    else v[0] = *reinterpret_cast<const uint64_t*>(p);
  }
  __device__ __forceinline__ void fill(float x) {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) asm("mov.b64 %0, {%1, %1};" : "=l"(v[i]) : "f"(x));
  }
  __device__ __forceinline__ void times(const GrChannels& o) {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v[i]) : "l"(o.v[i]));
  }
  __device__ __forceinline__ void one_minus(const GrChannels& o) {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      float a, b;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(o.v[i]));
      asm("mov.b64 %0, {%1, %2};" : "=l"(v[i]) : "f"(1.f - a), "f"(1.f - b));
    }
  }
  __device__ __forceinline__ void take(bool which, const GrChannels& o) {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) v[i] = which ? o.v[i] : v[i];
  }
  __device__ __forceinline__ float dot(const GrChannels& o) const {
    uint64_t sum;
    float a, b;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(sum) : "l"(v[0]), "l"(o.v[0]));
    if constexpr (PAIRS == 2) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum) : "l"(v[1]), "l"(o.v[1]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(sum));
    return a + b;
  }
};
template <> struct GrChannels<1> {
  float v;
  __device__ __forceinline__ void load(const float* p) { v = *p; }
  __device__ __forceinline__ void fill(float x) { v = x; }
  __device__ __forceinline__ void times(const GrChannels& o) { v *= o.v; }
  __device__ __forceinline__ void one_minus(const GrChannels& o) { v = 1.f - o.v; }
  __device__ __forceinline__ void take(bool which, const GrChannels& o) { v = which ? o.v : v; }
  __device__ __forceinline__ float dot(const GrChannels& o) const { return v * o.v; }
};

// Inside a sub-chunk: the columns of its tokens 4 PASS .. 4 PASS + 3, two of them by each of its two warps.  Token by
// token from the first of the four on: w, what is left of each token's k, takes the gates, and q w gives the next row.
template <int R, int PASS>
__device__ __forceinline__ void gr_inside(const float* fs, const float* qs, int dp, float* as, int odd, int lane, bool has) {
  const int s0 = 4 * PASS + 2 * odd;
  GrChannels<R> w[2];
  float sums[2][GR_SUB];
  w[0].fill(0.f), w[1].fill(0.f);
#pragma unroll
  for (int t = 0; t < GR_SUB; ++t) {
    sums[0][t] = sums[1][t] = 0.f;
    if (t < 4 * PASS) continue;
    GrChannels<R> f, q;
    f.fill(1.f), q.fill(0.f);
    if (has) f.load(fs + t * dp), q.load(qs + t * dp);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      w[k].times(f);
      if (t < 4 * PASS + 4) {
        GrChannels<R> own;
        own.one_minus(f);
        w[k].take(t == s0 + k, own);
      }
      sums[k][t] = q.dot(w[k]);
    }
  }
  constexpr int N = PASS < 2 ? 16 : PASS == 2 ? 8 : 4;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float sum = gr_sums<N>(sums[k], lane);
    const int t = 16 - N + lane * N / 32;
    if (lane % (32 / N) == 0 && t >= s0 + k) as[t * GR_AP + s0 + k] += sum;
  }
}

// One chunk of a long entry (see the head of this file).  Tokens past the entry's end have f = 1 and
// q = k = v = 0.  Bound by the instructions issued: inside a sub-chunk no row before a column's token is worked out and
// channels go in pairs, and the products between sub-chunks are one round of a warp each without barriers (before, a round and
// two barriers per distance with q rewritten in between).  3 prompts of 1,000 to 666 tokens, 32 heads of 128: 253 us before, 195 now.
// R: channels a lane of the sub-chunks' own blocks holds, in a slice, as few as the head needs.  32 heads of 64, 2,048
// tokens, all kernels: 216 us with two, 225 with four; 32 heads of 16, 1,000 tokens: 77 us with one, 89 with four.
// D: key and value size known when compiled; 0: any.
template <int R, int D>
__global__ void __launch_bounds__(256, 2) gated_recurrence_chunk_kernel(GatedRecurrence p, int aligned) {
  extern __shared__ __align__(16) float smem[];
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x, entry = blockIdx.y, chunk = blockIdx.z;
  const int entry_first = p.cu_tokens[entry], entry_count = p.cu_tokens[entry + 1] - entry_first;
  if (entry_count < p.long_from || chunk * GR_LONG_CHUNK >= entry_count) return;
  const int first = entry_first + chunk * GR_LONG_CHUNK, count = min(GR_LONG_CHUNK, entry_count - chunk * GR_LONG_CHUNK);
  const int dk = D ? D : p.dk, dv = D ? D : p.dv, dkp = (dk + 3) & ~3;
  // pitches: a fragment's rows (q, k) and its columns (v) fall into different banks
  const int dp = min(dkp, GR_SLICE) + 4, vp = min(dv, GR_SLICE) + 8;
  float* fs = smem;                              // [64][dp]: gates, then what is left of k
  float* qs = fs + GR_LONG_CHUNK * dp;           // [64][dp]; when q is done, vs [64][vp]
  float* vs = qs;
  float* as = qs + GR_LONG_CHUNK * max(dp, vp);  // [64][GR_AP]
  float* whole = as + GR_LONG_CHUNK * GR_AP;     // [4][dp]: the gates of a whole sub-chunk
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t at = (size_t)gr_chunk_slot(entry_first, entry, chunk) * p.heads + head;
  for (int i = tid; i < GR_LONG_CHUNK * GR_AP; i += 256) as[i] = 0.f;

  for (int d0 = 0; d0 < dk; d0 += GR_SLICE) {
    const int nd = min(GR_SLICE, dk - d0), ndp = (nd + 3) & ~3;
    __syncthreads();
    // four channels behind the last are read as part of a fragment
    for (int i = tid; i < GR_LONG_CHUNK * 4; i += 256) fs[(i >> 2) * dp + ndp + (i & 3)] = qs[(i >> 2) * dp + ndp + (i & 3)] = 0.f;
    if (aligned) {
      // four channels a thread, all loads of four rows on their way before the first is used
      const int quads = ndp >> 2, step = 256 / 32;      // a warp takes a row (up to 32 quads)
      const int d = lane * 4;
      if (lane < quads) {
        float low[4], bias[4] = {0.f, 0.f, 0.f, 0.f};
        load4(p.lower + head * dk + d0 + d, low);
        if (p.f_bias) load4(p.f_bias + head * dk + d0 + d, bias);
        const float* base = p.proj + (size_t)head * dk + d0 + d;
#pragma unroll
        for (int t0 = 0; t0 < GR_LONG_CHUNK; t0 += 4 * step) {
          float zf[4][4], zq[4][4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int t = t0 + u * step + warp;
            const float* row = base + (size_t)(first + min(t, count - 1)) * p.ld;
            load4(row + p.f_off, zf[u]);
            load4(row + p.q_off, zq[u]);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int t = t0 + u * step + warp;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              zq[u][e] = t < count ? zq[u][e] * gr_sigmoid(zq[u][e]) : 0.f;
              zf[u][e] = t < count ? low[e] + (1.f - low[e]) * gr_sigmoid(zf[u][e] + bias[e]) : 1.f;
            }
            store4(qs + t * dp + d, zq[u]);
            store4(fs + t * dp + d, zf[u]);
          }
        }
      }
    } else {
      for (int i = tid; i < GR_LONG_CHUNK * ndp; i += 256) {
        const int t = i / ndp, d = i - t * ndp;
        float f = 1.f, q = 0.f;
        if (t < count && d < nd) {
          const float* row = p.proj + (size_t)(first + t) * p.ld + (size_t)head * dk + d0 + d;
          const float zq = row[p.q_off], zf = row[p.f_off] + (p.f_bias ? p.f_bias[head * dk + d0 + d] : 0.f);
          const float l = p.lower[head * dk + d0 + d];
          q = zq * gr_sigmoid(zq);
          f = l + (1.f - l) * gr_sigmoid(zf);
        }
        fs[t * dp + d] = f;
        qs[t * dp + d] = q;
      }
    }
    __syncthreads();
    {
      // inside the sub-chunks: two warps each, lanes over the channels
      const int base = (warp >> 1) * GR_SUB, at_lane = base * dp + lane * R;
      const bool has = lane * R < ndp;
      float* own = as + base * GR_AP + base;
      gr_inside<R, 0>(fs + at_lane, qs + at_lane, dp, own, warp & 1, lane, has);
      gr_inside<R, 1>(fs + at_lane, qs + at_lane, dp, own, warp & 1, lane, has);
      gr_inside<R, 2>(fs + at_lane, qs + at_lane, dp, own, warp & 1, lane, has);
      gr_inside<R, 3>(fs + at_lane, qs + at_lane, dp, own, warp & 1, lane, has);
    }
    __syncthreads();
    // q with the gates from its sub-chunk's start on, k with those up to its sub-chunk's end
    for (int i = tid; i < ndp * GR_SUBS; i += 256) {
      const int sub = i / ndp, d = i - sub * ndp;
      float* f = fs + sub * GR_SUB * dp + d;
      float* q = qs + sub * GR_SUB * dp + d;
      float g[GR_SUB], b = 1.f;
#pragma unroll
      for (int t = 0; t < GR_SUB; ++t) {
        g[t] = f[t * dp];
        b *= g[t];
        q[t * dp] *= b;
      }
      whole[sub * dp + d] = b;
      if (d < 4) whole[sub * dp + ndp + d] = 1.f;      // the channels behind the last (see above)
      b = 1.f;
#pragma unroll
      for (int t = GR_SUB - 1; t >= 0; --t) {
        f[t * dp] = (1.f - g[t]) * b;
        b *= g[t];
      }
    }
    __syncthreads();
    // between two sub-chunks: A's six blocks of 16 x 16, a warp each; q takes the gates of the whole sub-chunks in
    // between on its way
    const int fg = lane >> 2, fq = lane & 3;           // this lane's row and column in a fragment
    if (warp < 6) {
      const int to = warp < 1 ? 1 : warp < 3 ? 2 : 3, from = warp - to * (to - 1) / 2;
      const float* q0 = qs + (to * GR_SUB + fg) * dp + fq;
      const float* k0 = fs + (from * GR_SUB + fg) * dp + fq;
      float sum[2][4], small[2][4];
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[b][i] = small[b][i] = 0.f;
      auto gated = [&](SplitA& a, int d) {
        float x[4] = {q0[d], q0[d + 4], q0[8 * dp + d], q0[8 * dp + d + 4]};
        for (int sub = to - 1; sub > from; --sub) {
          const float g0 = whole[sub * dp + d + fq], g1 = whole[sub * dp + d + fq + 4];
          x[0] *= g0, x[1] *= g1, x[2] *= g0, x[3] *= g1;
        }
        split_pair(x[0], x[1], a.part[0][0], a.part[1][0], a.part[2][0]);
        split_pair(x[2], x[3], a.part[0][1], a.part[1][1], a.part[2][1]);
      };
      int d = 0;
#pragma unroll 1
      for (; d + 12 <= ndp; d += 16) {
        SplitA fa, fa2;
        gated(fa, d), gated(fa2, d + 8);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          SplitB fb, fb2;
          split_load_b(fb, k0 + 8 * b * dp + d, 1);
          split_load_b(fb2, k0 + 8 * b * dp + d + 8, 1);
          split_mma(sum[b], small[b], fa, fa2, fb, fb2);
        }
      }
      if (d < ndp) {
        SplitA fa;
        gated(fa, d);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          SplitB fb;
          split_load_b(fb, k0 + 8 * b * dp + d, 1);
          split_mma(sum[b], small[b], fa, fb);
        }
      }
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          as[(to * GR_SUB + fg + 8 * (i >> 1)) * GR_AP + from * GR_SUB + 8 * b + 2 * fq + (i & 1)] += split_join(sum[b][i], small[b][i]);
    }
    // q with the gates from the chunk's start on
    if (lane * 4 < ndp) {
      const int d = lane * 4;
#pragma unroll
      for (int sub = 0; sub < GR_SUBS; ++sub) {
        float g[GR_SUBS][4];
#pragma unroll
        for (int m = 0; m < sub; ++m) load4(whole + m * dp + d, g[m]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int t = sub * GR_SUB + u * 8 + warp;
          if (t >= count) continue;
          float a[4];
          load4(qs + t * dp + d, a);
#pragma unroll
          for (int m = sub - 1; m >= 0; --m)
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] *= g[m][e];
          store4(p.qb + ((size_t)(first + t) * p.heads + head) * dkp + d0 + d, a);
        }
      }
    }
    __syncthreads();
    // k with the gates up to the chunk's end: four tokens and four channels at a time
    const int quads = ndp >> 2;
    for (int i = tid; i < quads * (GR_SUBS - 1) * 4; i += 256) {
      const int d = (i % quads) * 4, t = (i / quads) * 4, sub = t / GR_SUB;
      float b[4] = {1.f, 1.f, 1.f, 1.f};
      for (int m = GR_SUBS - 1; m > sub; --m) {
        float g[4];
        load4(whole + m * dp + d, g);
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] *= g[e];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float k[4];
        load4(fs + (t + u) * dp + d, k);
#pragma unroll
        for (int e = 0; e < 4; ++e) k[e] *= b[e];
        store4(fs + (t + u) * dp + d, k);
      }
    }
    for (int d = tid; d < nd; d += 256) {
      float b = 1.f;
#pragma unroll
      for (int sub = GR_SUBS - 1; sub >= 0; --sub) b *= whole[sub * dp + d];
      p.chunk_decay[at * dk + d0 + d] = b;
    }
    // the chunk's own end state
    for (int v0 = 0; v0 < dv; v0 += GR_SLICE) {
      const int nv = min(GR_SLICE, dv - v0);
      __syncthreads();
      if (aligned) {
        const int c = lane * 4;
        if (c < nv) {
          const float* base = p.proj + p.v_off + (size_t)head * dv + v0 + c;
          float x[8][4];
#pragma unroll
          for (int u = 0; u < 8; ++u) load4(base + (size_t)(first + min(u * 8 + warp, count - 1)) * p.ld, x[u]);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int t = u * 8 + warp;
#pragma unroll
            for (int e = 0; e < 4; ++e) x[u][e] = t < count ? x[u][e] : 0.f;
            store4(vs + t * vp + c, x[u]);
          }
        }
      } else {
        for (int i = tid; i < GR_LONG_CHUNK * nv; i += 256) {
          const int t = i / nv, c = i - t * nv;
          vs[t * vp + c] = t < count ? p.proj[(size_t)(first + t) * p.ld + p.v_off + (size_t)head * dv + v0 + c] : 0.f;
        }
      }
      __syncthreads();
      // a warp takes 32 channels and 32 columns at a time
      const int m0 = (warp >> 1) * 32;
      for (int c0 = (warp & 1) * 32; c0 < nv && m0 < ndp; c0 += 64) {
        float sum[2][4][4], small[2][4][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[a][b][i] = small[a][b][i] = 0.f;
        const float* ka = fs + fq * dp + m0 + fg;
        const float* vb = vs + fq * vp + c0 + fg;
#pragma unroll 1
        for (int t = 0; t < GR_LONG_CHUNK; t += 16) {
          SplitA fa[2], fa2[2];
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            split_load_a(fa[a], ka + t * dp + 16 * a, 1, dp);
            split_load_a(fa2[a], ka + (t + 8) * dp + 16 * a, 1, dp);
          }
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            SplitB fb, fb2;
            split_load_b(fb, vb + t * vp + 8 * b, vp);
            split_load_b(fb2, vb + (t + 8) * vp + 8 * b, vp);
#pragma unroll
            for (int a = 0; a < 2; ++a) split_mma(sum[a][b], small[a][b], fa[a], fa2[a], fb, fb2);
          }
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int d = m0 + 16 * a + 8 * h + fg;
            if (d >= nd) continue;
            float* dst = p.chunk_state + (at * dk + d0 + d) * dv + v0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const int c = c0 + 8 * b + 2 * fq;
              if (c < nv) *reinterpret_cast<float2*>(dst + c) = make_float2(split_join(sum[a][b][2 * h], small[a][b][2 * h]), split_join(sum[a][b][2 * h + 1], small[a][b][2 * h + 1]));
            }
          }
      }
    }
  }
  __syncthreads();
  float* within = p.within + at * GR_LONG_CHUNK * GR_LONG_CHUNK;
  for (int i = tid; i < GR_LONG_CHUNK * GR_LONG_CHUNK; i += 256) within[i] = as[(i / GR_LONG_CHUNK) * GR_AP + i % GR_LONG_CHUNK];
}

// One thread per four neighbouring columns of a state row: the start state of every chunk of a long entry, in
// order, in the place of the chunk's own end state, and the request's state row after the last chunk.
__global__ void __launch_bounds__(128) gated_recurrence_scan_kernel(GatedRecurrence p, int* status) {
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x, entry = blockIdx.y;
  const int first = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - first;
  if (count < p.long_from) return;
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.state_rows) {
    if (threadIdx.x == 0 && blockIdx.z == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
    return;
  }
  const int cell = (blockIdx.z * blockDim.x + threadIdx.x) * 4;
  if (cell >= p.dk * p.dv) return;
  const int d = cell / p.dv;
  const int chunks = (count + GR_LONG_CHUNK - 1) / GR_LONG_CHUNK;
  float* st = p.state + ((size_t)slot * p.heads + head) * p.dk * p.dv + cell;
  const bool wide = ((uintptr_t)p.state & 15) == 0;
  float state[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) state[e] = st[e];
  const size_t stride = (size_t)p.heads * p.dk * p.dv;
  float* cells = p.chunk_state + ((size_t)gr_chunk_slot(first, entry, 0) * p.heads + head) * p.dk * p.dv + cell;
  const float* __restrict__ decay = p.chunk_decay + ((size_t)gr_chunk_slot(first, entry, 0) * p.heads + head) * p.dk + d;
  for (int c = 0; c < chunks; c += 4) {          // four chunks' loads at a time
    float own[4][4], keep[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int at = min(c + u, chunks - 1);
      load4(cells + at * stride, own[u]);
      keep[u] = decay[(size_t)at * p.heads * p.dk];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c + u >= chunks) break;
      store4(cells + (c + u) * stride, state);
#pragma unroll
      for (int e = 0; e < 4; ++e) state[e] = fmaf(keep[u], state[e], own[u][e]);
    }
  }
  if (wide) {
    store4(st, state);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) st[e] = state[e];
  }
}

// o = [q D | A] [S_start; V] for the 64 tokens of a chunk, then the head's norm.  Both operands pass
// through shared memory in stretches of 32 rows of the right one; a warp takes 32 tokens and 32 columns of a
// pass of 128 columns (dv is a multiple of 4).  Where dv takes more than one pass the rows wait in shared
// memory for the norm.
#define GR_FK 32
#define GR_FX (GR_FK + 4)
__host__ __device__ static inline int gr_finish_pitch(int dv) { return ((dv < GR_SLICE ? dv : GR_SLICE) + 31) / 32 * 32 + 8; }
__host__ __device__ static inline int gr_finish_stages(int dv) { return dv <= GR_SLICE ? 3 : 2; }
template <typename TO, int D>
__global__ void __launch_bounds__(256, 2) gated_recurrence_finish_kernel(GatedRecurrence p, int v_aligned) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float part[4][GR_LONG_CHUNK];
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x, entry = blockIdx.y, chunk = blockIdx.z;
  const int entry_first = p.cu_tokens[entry], entry_count = p.cu_tokens[entry + 1] - entry_first;
  if (entry_count < p.long_from || chunk * GR_LONG_CHUNK >= entry_count) return;
  const int first = entry_first + chunk * GR_LONG_CHUNK, count = min(GR_LONG_CHUNK, entry_count - chunk * GR_LONG_CHUNK);
  const int dk = D ? D : p.dk, dv = D ? D : p.dv, dkp = (dk + 3) & ~3;
  const int pitch = gr_finish_pitch(dv), stages = gr_finish_stages(dv);
  const int stage_floats = GR_LONG_CHUNK * GR_FX + GR_FK * pitch;
  float* os = smem + stages * stage_floats;          // [64][dv], only where dv > 128
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fg = lane >> 2, fq = lane & 3;
  const int m0 = (warp >> 2) * 32, n0 = (warp & 3) * 32;
  const size_t at = (size_t)gr_chunk_slot(entry_first, entry, chunk) * p.heads + head;
  const float* start = p.chunk_state + at * dk * dv;
  const float* values = p.proj + (size_t)first * p.ld + p.v_off + (size_t)head * dv;
  const int q_steps = (dkp + GR_FK - 1) / GR_FK, steps = q_steps + (count + GR_FK - 1) / GR_FK;
  // what this thread copies of a stretch: eight numbers of a row of the left operand, every eighth four of a row
  // of the right one
  const int xt = tid >> 2, xk = (tid & 3) * 8, yk = tid >> 3, yc = (tid & 7) * 4;
  const bool row = xt < count;
  const float* x_q = p.qb + ((size_t)(first + (row ? xt : 0)) * p.heads + head) * dkp + xk;
  const float* x_a = p.within + at * GR_LONG_CHUNK * GR_LONG_CHUNK + xt * GR_LONG_CHUNK + xk;

  auto stage = [&](int step, int v0, int nv) {
    float* xs = smem + (step % stages) * stage_floats;
    float* ys = xs + GR_LONG_CHUNK * GR_FX + yk * pitch + yc;
    const bool state = step < q_steps;
    const int k0 = (state ? step : step - q_steps) * GR_FK;
    const float* src = (state ? x_q : x_a) + k0;
    float* to = xs + xt * GR_FX + xk;
    gr_copy16(to, src, row && (!state || k0 + xk < dkp));
    gr_copy16(to + 4, src + 4, row && (!state || k0 + xk + 4 < dkp));
    const bool valid = state ? k0 + yk < dk : k0 + yk < count;
    const float* from = !valid ? start : (state ? start + (size_t)(k0 + yk) * dv : values + (size_t)(k0 + yk) * p.ld) + v0 + yc;
#pragma unroll
    for (int j = 0; j < GR_SLICE / 32; ++j) {
      if (yc + 32 * j >= nv) break;
      if (state || v_aligned) {
        gr_copy16(ys + 32 * j, valid ? from + 32 * j : from, valid);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) ys[32 * j + e] = valid ? from[32 * j + e] : 0.f;
      }
    }
  };

  for (int v0 = 0; v0 < dv; v0 += GR_SLICE) {
    const int nv = min(GR_SLICE, dv - v0);
    float sum[2][4][4], small[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[a][b][i] = small[a][b][i] = 0.f;
    __syncthreads();
    for (int s = 0; s + 1 < stages; ++s) {
      if (s < steps) stage(s, v0, nv);
      gr_commit();
    }
    for (int step = 0; step < steps; ++step) {
      if (stages == 3) gr_wait<1>();
      else gr_wait<0>();
      __syncthreads();               // this stretch has landed; everyone is done with the one before it
      if (step + stages - 1 < steps) stage(step + stages - 1, v0, nv);
      gr_commit();
      if (step >= q_steps) {
        // What is too loud to be split joins by multiply-adds, and only the tokens that see it: its products with
        // the zeros of A would not be zero.
        float* ys = smem + (step % stages) * stage_floats + GR_LONG_CHUNK * GR_FX;
        bool loud = false;
        const int quads = nv >> 2;
        for (int i = tid; i < GR_FK * quads; i += 256) {
          float x[4];
          load4(ys + (i / quads) * pitch + (i % quads) * 4, x);
          loud |= split_loud(x[0]) || split_loud(x[1]) || split_loud(x[2]) || split_loud(x[3]);
        }
        if (__syncthreads_or(loud)) {
          const float* xs = ys - GR_LONG_CHUNK * GR_FX;
#pragma unroll
          for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int t = m0 + 16 * a + 8 * (i >> 1) + fg, c = n0 + 8 * b + 2 * fq + (i & 1);
                if (c >= nv) continue;
#pragma unroll 1
                for (int s = 0; s < GR_FK && s + GR_FK * (step - q_steps) <= t; ++s)
                  if (split_loud(ys[s * pitch + c])) sum[a][b][i] = fmaf(xs[t * GR_FX + s], ys[s * pitch + c], sum[a][b][i]);
              }
          __syncthreads();
          for (int i = tid; i < GR_FK * nv; i += 256) {
            float& x = ys[(i / nv) * pitch + i % nv];
            if (split_loud(x)) x = 0.f;
          }
          __syncthreads();
        }
      }
      // the first 32 tokens come before all tokens of the second stretch of V: A is zero there
      if (n0 < nv && (m0 > 0 || step <= q_steps)) {
        const float* xs = smem + (step % stages) * stage_floats + (m0 + fg) * GR_FX + fq;
        const float* ys = smem + (step % stages) * stage_floats + GR_LONG_CHUNK * GR_FX + fq * pitch + n0 + fg;
#pragma unroll 1
        for (int k = 0; k < GR_FK; k += 16) {
          SplitA fa[2], fa2[2];
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            split_load_a(fa[a], xs + 16 * a * GR_FX + k, GR_FX, 1);
            split_load_a(fa2[a], xs + 16 * a * GR_FX + k + 8, GR_FX, 1);
          }
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            SplitB fb, fb2;
            split_load_b(fb, ys + k * pitch + 8 * b, pitch);
            split_load_b(fb2, ys + (k + 8) * pitch + 8 * b, pitch);
#pragma unroll
            for (int a = 0; a < 2; ++a) split_mma(sum[a][b], small[a][b], fa[a], fa2[a], fb, fb2);
          }
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[a][b][i] = n0 + 8 * b + 2 * fq < nv ? split_join(sum[a][b][i], small[a][b][i]) : 0.f;
    if (dv > GR_SLICE) {
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (n0 + 8 * b + 2 * fq < nv)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              *reinterpret_cast<float2*>(os + (m0 + 16 * a + 8 * h + fg) * dv + v0 + n0 + 8 * b + 2 * fq) =
                  make_float2(sum[a][b][2 * h], sum[a][b][2 * h + 1]);
      continue;
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float sq = 0.f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          sq = fmaf(sum[a][b][2 * h], sum[a][b][2 * h], sq);
          sq = fmaf(sum[a][b][2 * h + 1], sum[a][b][2 * h + 1], sq);
        }
        sq += __shfl_xor_sync(0xffffffffu, sq, 1);
        sq += __shfl_xor_sync(0xffffffffu, sq, 2);
        if (fq == 0) part[warp & 3][m0 + 16 * a + 8 * h + fg] = sq;
      }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = m0 + 16 * a + 8 * h + fg;
        if (t >= count) continue;
        const float inv = 1.f / sqrtf((part[0][t] + part[1][t] + part[2][t] + part[3][t]) / (float)dv + p.eps);
        TO* dst = (TO*)p.out + ((size_t)(first + t) * p.heads + head) * dv;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = n0 + 8 * b + 2 * fq;
          if (c >= nv) continue;
          gr_store2(dst + c, sum[a][b][2 * h] * inv * p.norm_w[c], sum[a][b][2 * h + 1] * inv * p.norm_w[c + 1]);
        }
      }
  }
  if (dv <= GR_SLICE) return;
  __syncthreads();
  for (int r = warp; r < count; r += 8) {
    float sq = 0.f;
    for (int c = lane; c < dv; c += 32) sq = fmaf(os[r * dv + c], os[r * dv + c], sq);
    const float inv = 1.f / sqrtf(warp_sum(sq) / (float)dv + p.eps);
    TO* dst = (TO*)p.out + (size_t)(first + r) * p.heads * dv + (size_t)head * dv;
    for (int c = lane; c < dv; c += 32) dst[c] = from_float<TO>(os[r * dv + c] * inv * p.norm_w[c]);
  }
}

// Threads of a column: the largest power of two up to 8 (4 where the block stays at 128
// threads or more: then a warp's state rows are whole 32-byte sectors) that divides dk, keeps
// the block within 1,024 threads and a thread within GR_MAX_KPT rows.  0: no such number.
static int gr_column_threads(int dk, int dv) {
  const int prefer[] = {4, 8, 2, 1, 16, 32};
  for (int pass = 0; pass < 2; ++pass) {
    for (int ds : prefer) {
      if (dk % ds || (long long)dv * ds > 1024 || dk / ds > GR_MAX_KPT) continue;
      if (pass == 0 && (dv * ds < 128 || dk / ds > 16)) continue;
      return ds;
    }
  }
  return 0;
}

// Shared memory of the chunk kernels.
static size_t gr_chunk_smem(int dk, int dv) {
  const int dkp = (dk + 3) & ~3, dp = (dkp < GR_SLICE ? dkp : GR_SLICE) + 4, vp = (dv < GR_SLICE ? dv : GR_SLICE) + 8;
  return sizeof(float) * ((size_t)GR_LONG_CHUNK * (dp + (dp > vp ? dp : vp) + GR_AP) + GR_SUBS * dp);
}
static size_t gr_finish_smem(int dv) {
  return sizeof(float) * ((size_t)gr_finish_stages(dv) * (GR_LONG_CHUNK * GR_FX + GR_FK * gr_finish_pitch(dv)) +
                          (dv > GR_SLICE ? (size_t)GR_LONG_CHUNK * dv : 0));
}

// 32-bit floats of scratch the chunk-parallel kernels need for a step of `tokens` tokens in
// `entries` entries (0: these sizes run token by token whatever the entries' lengths).
FE_EXPORT long long fe_gated_recurrence_scratch(int tokens, int entries, int heads, int dk, int dv) {
  if (dv % 4 != 0 || gr_finish_smem(dv) > 220 * 1024 || gr_column_threads(dk, dv) == 0) return 0;
  const long long slots = tokens / GR_LONG_CHUNK + entries + 1, dkp = (dk + 3) & ~3;
  return slots * heads * ((long long)dk * dv + GR_LONG_CHUNK * GR_LONG_CHUNK + dkp) + (long long)tokens * heads * dkp;
}

// Tokens from which on an entry runs chunk by chunk.
FE_EXPORT int fe_gated_recurrence_long_from() { return 2 * GR_LONG_CHUNK; }

// scratch: null, or fe_gated_recurrence_scratch floats; then entries of fe_gated_recurrence_long_from
// tokens or more (max_new is the most tokens any entry brings) run chunk by chunk
FE_EXPORT int fe_gated_recurrence(const float* proj, long long ld, int q_off, int f_off, int v_off, const float* f_bias,
                                  const float* lower, const float* norm_w, float eps, float* state, int state_rows,
                                  const int* slots, const int* cu_tokens, void* out, int out_dtype, int entries, int heads,
                                  int dk, int dv, int tokens, int max_new, float* scratch, int* status,
                                  cudaStream_t stream) {
  if (entries <= 0) return 0;
  if (heads < 1 || dk < 1 || dv < 1 || heads > 65535 || entries > 65535) return FE_ERR_BAD_SHAPE;
  const int ds = gr_column_threads(dk, dv);
  if (ds == 0) return FE_ERR_BAD_SHAPE;
  const int kpt = dk / ds;
  GatedRecurrence p{proj, ld, q_off, f_off, v_off, f_bias, lower, norm_w, eps, state, state_rows, slots, cu_tokens, out,
                    heads, dk, dv, ds, kpt, 0, (dk + 3) & ~3, nullptr, nullptr, nullptr, nullptr};
  const bool chunked = scratch != nullptr && max_new >= fe_gated_recurrence_long_from() &&
                       fe_gated_recurrence_scratch(tokens, entries, heads, dk, dv) > 0;
  if (chunked) {
    const long long chunk_slots = tokens / GR_LONG_CHUNK + entries + 1;
    p.long_from = fe_gated_recurrence_long_from();
    // every part starts on a 16-byte boundary
    p.chunk_state = scratch;
    p.within = p.chunk_state + (size_t)chunk_slots * heads * dk * dv;
    p.qb = p.within + (size_t)chunk_slots * heads * GR_LONG_CHUNK * GR_LONG_CHUNK;
    p.chunk_decay = p.qb + (size_t)tokens * heads * p.dkp;
  }
  const int threads = (dv * ds + 31) / 32 * 32;
  const size_t smem = sizeof(float) * (size_t)GR_CHUNK * 2 * (dk + dv);
  if (smem > 200 * 1024) return FE_ERR_TOO_LARGE;
  int rc = FE_ERR_BAD_DTYPE;
#define GR_LAUNCH(TO, KPT)                                                                                            \
  do {                                                                                                                \
    if (smem > 48 * 1024)                                                                                             \
      cudaFuncSetAttribute(gated_recurrence_kernel<TO, KPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    rc = fe_launch_dependent(gated_recurrence_kernel<TO, KPT>, dim3(heads, entries), dim3(threads), smem, stream, p,  \
                             status);                                                                                 \
  } while (0)
#define GR_BY_KPT(TO)                        \
  do {                                       \
    if (kpt <= 4) GR_LAUNCH(TO, 4);          \
    else if (kpt <= 8) GR_LAUNCH(TO, 8);     \
    else if (kpt <= 16) GR_LAUNCH(TO, 16);   \
    else GR_LAUNCH(TO, 32);                  \
  } while (0)
  if (out_dtype == FE_DTYPE_F32) GR_BY_KPT(float);
  else if (out_dtype == FE_DTYPE_BF16) GR_BY_KPT(bf16);
#undef GR_BY_KPT
#undef GR_LAUNCH
  if (rc || !chunked) return rc ? rc : fe_last_error();
  const int chunks = (max_new + GR_LONG_CHUNK - 1) / GR_LONG_CHUNK;
  if (chunks > 65535) return FE_ERR_TOO_LARGE;
  const size_t chunk_smem = gr_chunk_smem(dk, dv);
  // heads of 64 and of 128 on both sides: places and bounds known when compiled (3 prompts of 1,000 to 666
  // tokens, 32 heads of 128: chunk kernel 195 us, 169 so; outputs 126 and 114)
  const int whole = dk == dv && (dk == 64 || dk == 128) ? dk : 0;
  auto chunk_kernel = whole == 64 ? gated_recurrence_chunk_kernel<2, 64> : whole == 128 ? gated_recurrence_chunk_kernel<4, 128>
                      : dk <= 32 ? gated_recurrence_chunk_kernel<1, 0> : dk <= 64 ? gated_recurrence_chunk_kernel<2, 0> : gated_recurrence_chunk_kernel<GR_SLICE / 32, 0>;
  if (chunk_smem > 48 * 1024) cudaFuncSetAttribute(chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chunk_smem);
  const int v_aligned = ((uintptr_t)proj & 15) == 0 && ld % 4 == 0 && v_off % 4 == 0;
  const int aligned = v_aligned && q_off % 4 == 0 && f_off % 4 == 0 && dk % 4 == 0 && (((uintptr_t)lower | (uintptr_t)f_bias) & 15) == 0;
  rc = fe_launch_dependent(chunk_kernel, dim3(heads, entries, chunks), dim3(256), chunk_smem, stream, p, aligned);
  if (rc) return rc;
  rc = fe_launch_dependent(gated_recurrence_scan_kernel, dim3(heads, entries, (dk * dv + 511) / 512), dim3(128), 0, stream,
                           p, status);
  if (rc) return rc;
  const size_t finish_smem = gr_finish_smem(dv);
#define GR_FINISH(TO)                                                                                                          \
  do {                                                                                                                         \
    auto finish = whole == 64 ? gated_recurrence_finish_kernel<TO, 64> : whole == 128 ? gated_recurrence_finish_kernel<TO, 128> \
                                                                       : gated_recurrence_finish_kernel<TO, 0>;                \
    if (finish_smem > 48 * 1024) cudaFuncSetAttribute(finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)finish_smem);  \
    rc = fe_launch_dependent(finish, dim3(heads, entries, chunks), dim3(256), finish_smem, stream, p, v_aligned);              \
  } while (0)
  if (out_dtype == FE_DTYPE_F32) GR_FINISH(float);
  else GR_FINISH(bf16);
#undef GR_FINISH
  return rc ? rc : fe_last_error();
}

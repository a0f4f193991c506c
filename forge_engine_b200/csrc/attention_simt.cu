// Causal grouped-query attention over cache pages in plain 32-bit arithmetic.
//
// The plain form upstream uses for prefill is softmax(q k^T * scale + mask) v with the
// softmax in 32-bit (src/forge_engine/qwen3.py:187-206); its decode kernel walks the
// pages position by position with an online softmax in 32-bit
// (src/forge_engine/kernels/cuda_paged.py:276-347).  These kernels are the general form
// of both: any number of new tokens per request, keys read from pages (the new
// tokens' keys have been written before they run), optional window.  They are the true
// 32-bit attention and the fallback for shapes the tensor-core kernels refuse.
//
// attention_simt_span: single tokens (decoding, or a caller that names no entries).  A block takes
//   the query heads of one kv head (up to 16) over one span of 128 key positions, whose keys and
//   values pass through a ring in shared memory; attention_simt_merge folds a token's spans in
//   order.  Bound by the bytes of keys and values; the spans are what keeps the chip busy at few
//   requests.
// attention_simt_tile: entries of several tokens.  A block takes 32 rows (token, query head) of one
//   kv head over all their keys in tiles of 64, as two small FFMA products from shared memory; where that leaves
//   the chip idle, over a share of their spans, and attention_simt_fold folds a row's spans.  Bound by instructions (heads of 128:
//   two blocks of 8 warps an SM issue in 53 % of the cycles; with 4 warps of twice the rows 30 %).
//
// A row's bits depend on nothing but its token and the keys it sees: not on what else is in the batch, nor on
// how its portion was cut.  Both kernels take a span's keys, counted from position 0, in thirty-twos with one
// running maximum, sum over positions (or elements of a head: even and odd ones apart) in ascending order,
// and fold the spans one after the other (fold_factors).  us, 16 heads of 128, before (4 warps a block, all spans of a row by one block, one
// head's tiles after the other's, the value product without pairs of columns) and now: 500 tokens 158 / 104, 2,048 1,243 / 806, 200 after
// 3,000 696 / 302; 32 heads of 64 111 / 92, 985 / 862, 461 / 307; 40 of 64 in bfloat16 104 / 98, 1,102 / 1,061, 455 / 368.
#include "attention_common.cuh"

#include <algorithm>

namespace {

constexpr int SPAN = 128;          // key positions of a block of the span kernel
constexpr int SPAN_KEYS = 32;      // of one stage of its ring
constexpr int SPAN_STAGES = 3;
constexpr int SPAN_THREADS = 128;
constexpr int TILE_ROWS = 32, TILE_KEYS = 64;
constexpr int P_PITCH = TILE_KEYS + 4;

struct Simt {
  const void* q;
  int q_stride;
  PagedKV cache;
  const int* positions;
  const int* token_entry;
  const int* cu_tokens;     // null: every token is a unit of its own
  int units, window;
  float scale;
  void* out;
  int num_q_heads, groups, spans, row_tiles;
  int unit0;                // of this launch: the units go through the workspace in slices
  float* partial;           // [unit of the slice][kv head][row tile][span][row][D + 2]
  int n_tokens;
  int share;                // blocks of a row tile and kv head (1: all spans by one block)
  int* status;
};

__device__ __forceinline__ void copy16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint64_t scale2(uint64_t x, float by) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(twice(by)));
  return r;
}
__device__ __forceinline__ float half2_of(uint64_t x, int which) { return __uint_as_float((unsigned)(which ? x >> 32 : x)); }
__device__ __forceinline__ float sum2(uint64_t acc) {
  return __uint_as_float((unsigned)acc) + __uint_as_float((unsigned)(acc >> 32));
}
__device__ __forceinline__ void pairs4(const float* p, uint64_t (&out)[2]) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  out[0] = v.x;
  out[1] = v.y;
}
__device__ __forceinline__ void pairs4(const bf16* p, uint64_t (&out)[2]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  out[0] = (uint64_t)(raw.x << 16) | ((uint64_t)(raw.x & 0xffff0000u) << 32);
  out[1] = (uint64_t)(raw.y << 16) | ((uint64_t)(raw.y & 0xffff0000u) << 32);
}

// Sums (or maxima) of N (four or eight) numbers over 16 neighbouring lanes, for all of them, in the order of warp_sum's last
// four steps: half of the numbers go to the partner at a time, and come back whole.
template <bool MAX, int N>
__device__ __forceinline__ void reduce_all(float (&x)[N], int lane) {
  int bit = 8;
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1, bit >>= 1) {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? x[i] : x[i + half], keep = upper ? x[i + half] : x[i];
      const float got = __shfl_xor_sync(0xffffffffu, send, bit);
      x[i] = MAX ? fmaxf(keep, got) : keep + got;
    }
  }
  float mine = x[0];
#pragma unroll
  for (int b = 8 / N; b > 0; b >>= 1) {
    const float got = __shfl_xor_sync(0xffffffffu, mine, b);
    mine = MAX ? fmaxf(mine, got) : mine + got;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = __shfl_sync(0xffffffffu, mine, (lane & 16) | (i * (16 / N)));
}

// A span (maximum m) joins those before it (maximum top): their sums take `old`, its own `mine`.
__device__ __forceinline__ void fold_factors(float& top, float m, float& old, float& mine) {
  const float t = fmaxf(top, m);
  old = top == -INFINITY ? 0.f : expf(top - t);
  mine = m == -INFINITY ? 0.f : expf(m - t);
  top = t;
}

// Where key position `key` of an entry lies, in elements of the cache; -1 (and a status bit) without a page.
__device__ __forceinline__ long long key_offset(const PagedKV& c, const int* table, int kvh, int key, int* status) {
  const int logical = key / c.page_size;
  const int page = logical < c.max_pages ? table[logical] : -1;
  if (page < 0 || page >= c.num_pages) {
    atomicOr(status, FE_STATUS_BAD_PAGE);
    return -1;
  }
  return (long long)kv_offset(c, page, kvh, key - logical * c.page_size);
}

// KEYS keys from `first` on (those in [lo, hi] are needed), as they lie in memory: k rows with 16
// bytes of padding, v rows without.  ok[i]: whether key i counts.
template <typename T, int KEYS, int THREADS>
__device__ __forceinline__ void stage_keys(const Simt& p, const int* table, int kvh, int first, int lo, int hi, T* ks, T* vs, int* ok) {
  constexpr int CH = 16 / (int)sizeof(T), TPK = THREADS / KEYS;     // threads of a key
  const int D = p.cache.head_dim, i = threadIdx.x / TPK, part = threadIdx.x % TPK;
  const int key = first + i;
  const long long off = key >= lo && key <= hi ? key_offset(p.cache, table, kvh, key, p.status) : -1;
  if (part == 0) ok[i] = off >= 0;
  const T* k = (const T*)p.cache.k + (off < 0 ? 0 : off);
  const T* v = (const T*)p.cache.v + (off < 0 ? 0 : off);
  for (int d = part * CH; d < D; d += TPK * CH) {
    copy16(ks + i * (D + CH) + d, k + d, off >= 0);
    copy16(vs + i * D + d, v + d, off >= 0);
  }
}

template <typename T, int R, int DMAX>
__global__ void __launch_bounds__(SPAN_THREADS) attention_simt_span_kernel(const Simt p) {
  constexpr int CH = 16 / (int)sizeof(T), PER = (DMAX + SPAN_THREADS - 1) / SPAN_THREADS;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) float ps[R][SPAN_KEYS];
  __shared__ float corr[R];
  __shared__ int ok[SPAN_STAGES][SPAN_KEYS];
  pdl_trigger();
  pdl_wait();
  const int D = p.cache.head_dim, unit = p.unit0 + (int)blockIdx.z, span = blockIdx.x, kvh = blockIdx.y / p.row_tiles, tile = blockIdx.y % p.row_tiles;
  int token = unit, entry;
  if (p.cu_tokens != nullptr) {
    token = p.cu_tokens[unit];
    if (p.cu_tokens[unit + 1] - token != 1) return;
    entry = unit;
  } else {
    entry = p.token_entry[unit];
  }
  const int pos = p.positions[token];
  const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
  const int begin = span * SPAN, end = min(begin + SPAN, pos + 1);
  if (span == 0 && pos >= p.spans * SPAN && threadIdx.x == 0) atomicOr(p.status, FE_STATUS_BAD_PAGE);   // past the block table
  if (end <= max(begin, lo)) return;
  const int rows = min(R, p.groups - tile * R);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* qs = (float*)smem;                                     // [R][D]
  T* ks = (T*)(qs + R * D);                                     // [stage][key][D + CH]
  T* vs = ks + SPAN_STAGES * SPAN_KEYS * (D + CH);              // [stage][key][D]
  const int* table = p.cache.block_table + (size_t)entry * p.cache.max_pages;
  const int first = max(begin, lo) / SPAN_KEYS * SPAN_KEYS, steps = (end - first + SPAN_KEYS - 1) / SPAN_KEYS;
#pragma unroll
  for (int s = 0; s < SPAN_STAGES - 1; ++s) {
    if (s < steps)
      stage_keys<T, SPAN_KEYS, SPAN_THREADS>(p, table, kvh, first + s * SPAN_KEYS, lo, end - 1, ks + s * SPAN_KEYS * (D + CH),
                                             vs + s * SPAN_KEYS * D, ok[s]);
    commit();
  }
  const int head0 = kvh * p.groups + tile * R;
  const T* q = (const T*)p.q + (size_t)token * p.q_stride + (size_t)head0 * D;
  for (int i = threadIdx.x; i < R * D; i += SPAN_THREADS) qs[i] = i < rows * D ? to_float(q[i]) : 0.f;

  float m[(R + 3) / 4], l[(R + 3) / 4], acc[R][PER];
#pragma unroll
  for (int i = 0; i < (R + 3) / 4; ++i) m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < PER; ++j) acc[i][j] = 0.f;

  for (int step = 0; step < steps; ++step) {
    const int s = step % SPAN_STAGES;
    wait<SPAN_STAGES - 2>();
    __syncthreads();               // this stage has landed; everyone is done with the one before it
    const int next = step + SPAN_STAGES - 1, to = next % SPAN_STAGES;
    if (next < steps)
      stage_keys<T, SPAN_KEYS, SPAN_THREADS>(p, table, kvh, first + next * SPAN_KEYS, lo, end - 1, ks + to * SPAN_KEYS * (D + CH),
                                             vs + to * SPAN_KEYS * D, ok[to]);
    commit();
    const T* krow = ks + (s * SPAN_KEYS + lane) * (D + CH);
#pragma unroll
    for (int i = 0; i < (R + 3) / 4; ++i) {
      const int r = warp + 4 * i;
      if (r < rows) {
        uint64_t dot = 0;
        const float* qrow = qs + r * D;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          uint64_t a[2], b[2];
          pairs4(qrow + d, a);
          pairs4(krow + d, b);
          fma2(dot, a[0], b[0]);
          fma2(dot, a[1], b[1]);
        }
        const float score = ok[s][lane] ? __fmul_rn(sum2(dot), p.scale) : -INFINITY;
        const float top = fmaxf(m[i], warp_max(score));
        const float e = score == -INFINITY ? 0.f : expf(score - top);
        const float c = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
        l[i] = fmaf(l[i], c, warp_sum(e));
        m[i] = top;
        ps[r][lane] = e;
        if (lane == 0) corr[r] = c;
      }
    }
    __syncthreads();
    const T* vt = vs + s * SPAN_KEYS * D;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int d = threadIdx.x + j * SPAN_THREADS;
      if (d < D) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r < rows) acc[r][j] *= corr[r];
#pragma unroll 2
        for (int key = 0; key < SPAN_KEYS; key += 4) {
          float v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = to_float(vt[(key + e) * D + d]);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (r < rows) {
              const float4 e = *reinterpret_cast<const float4*>(&ps[r][key]);
              acc[r][j] = fmaf(e.x, v[0], acc[r][j]);
              acc[r][j] = fmaf(e.y, v[1], acc[r][j]);
              acc[r][j] = fmaf(e.z, v[2], acc[r][j]);
              acc[r][j] = fmaf(e.w, v[3], acc[r][j]);
            }
          }
        }
      }
    }
  }
  float* part = p.partial + ((((size_t)blockIdx.z * gridDim.y + blockIdx.y) * p.spans + span) * R) * (D + 2);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (r < rows) {
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int d = threadIdx.x + j * SPAN_THREADS;
        if (d < D) part[r * (D + 2) + d] = acc[r][j];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < (R + 3) / 4; ++i) {
    const int r = warp + 4 * i;
    if (r < rows && lane == 0) {
      part[r * (D + 2) + D] = m[i];
      part[r * (D + 2) + D + 1] = l[i];
    }
  }
}

// One block per (query head, unit): its spans in ascending order.
template <typename T>
__global__ void __launch_bounds__(128) attention_simt_merge_kernel(const Simt p, int R) {
  pdl_trigger();
  pdl_wait();
  const int D = p.cache.head_dim, unit = p.unit0 + (int)blockIdx.x, head = blockIdx.y;
  int token = unit;
  if (p.cu_tokens != nullptr) {
    token = p.cu_tokens[unit];
    if (p.cu_tokens[unit + 1] - token != 1) return;
  }
  const int pos = p.positions[token], lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
  // a position past the block table has no spans beyond it
  const int from = lo / SPAN, to = min(pos / SPAN, p.spans - 1);
  const int kvh = head / p.groups, within = head - kvh * p.groups;
  const size_t stride = (size_t)R * (D + 2);
  const float* part = p.partial + (((size_t)blockIdx.x * (p.cache.num_kv_heads * p.row_tiles) + kvh * p.row_tiles + within / R) * p.spans) * stride +
                      (size_t)(within % R) * (D + 2);
  T* out = (T*)p.out + ((size_t)token * p.num_q_heads + head) * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float num = 0.f, den = 0.f, top = -INFINITY;
#pragma unroll 4
    for (int s = from; s <= to; ++s) {
      float old, mine;
      fold_factors(top, part[s * stride + D], old, mine);
      num = fmaf(part[s * stride + d], mine, __fmul_rn(num, old));
      den = fmaf(part[s * stride + D + 1], mine, __fmul_rn(den, old));
    }
    out[d] = from_float<T>(den > 0.f ? num / den : 0.f);
  }
}

// Which entry of several tokens row tile `index` of the launch belongs to, and which of its tiles it is: a warp counts 32
// entries at a time.  False past the last tile.
__device__ __forceinline__ bool find_tile(const Simt& p, int index, int& entry, int& tile, int& tiles) {
  const int lane = threadIdx.x & 31;
  for (int base = 0, seen = 0; base < p.units; base += 32) {
    const int e = base + lane;
    const int count = e < p.units ? p.cu_tokens[e + 1] - p.cu_tokens[e] : 0;
    const int mine = count > 1 ? (count * p.groups + TILE_ROWS - 1) / TILE_ROWS : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const unsigned past = __ballot_sync(0xffffffffu, index < seen + upto);
    if (past) {
      const int owner = __ffs(past) - 1;
      entry = base + owner;
      tiles = __shfl_sync(0xffffffffu, mine, owner);
      tile = index - seen - (__shfl_sync(0xffffffffu, upto, owner) - tiles);
      return true;
    }
    seen += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// SPLIT: `share` blocks take a row tile of a kv head, each every share-th span of the keys that its rows see, and leave the spans'
// maxima and sums to attention_simt_fold_kernel.
// Whole tiles: the kv heads of a row tile one after the other, so that the tiles with the most keys start first in all of them (one
// head's tiles after the other: 1,000 tokens of 16 heads of 128 324 us, 223 so; 32 heads of 64 314 and 256).  Shares of a tile lie tile by tile.
template <typename T, int DMAX, bool SPLIT, int THREADS>
__global__ void __launch_bounds__(THREADS, DMAX == 256 && sizeof(T) == 4 ? 1 : THREADS == 256 ? 2 : 3) attention_simt_tile_kernel(const Simt p) {
  constexpr int RT = TILE_ROWS / (THREADS / 16);               // rows of a thread
  constexpr int CH = 16 / (int)sizeof(T), CG = DMAX / 64;      // groups of four output columns of a thread
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int ok[TILE_KEYS];
  pdl_trigger();
  pdl_wait();
  const int D = p.cache.head_dim, nkv = p.cache.num_kv_heads;
  const unsigned per = nkv * (SPLIT ? p.share : 1), tiles_all = gridDim.x / per;
  const int part = (int)(SPLIT ? blockIdx.x / tiles_all : blockIdx.x % per), kvh = part % nkv, which = part / nkv;
  int entry = 0, tile = 0, tiles = 0;
  if (!find_tile(p, (int)(SPLIT ? blockIdx.x % tiles_all : blockIdx.x / per), entry, tile, tiles)) return;
  const int token0 = p.cu_tokens[entry], count = p.cu_tokens[entry + 1] - token0;
  const int total = count * p.groups;
  const int row0 = (tiles - 1 - tile) * TILE_ROWS;    // the tiles with the most keys first
  const int qpitch = D + 4;
  float* qs = (float*)smem;                                     // [row][D + 4]
  float* ps = qs + TILE_ROWS * qpitch;                          // [row][key]
  T* ks = (T*)(ps + TILE_ROWS * P_PITCH);                       // [key][D + CH]
  T* vs = ks + TILE_KEYS * (D + CH);                            // [key][D]
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int* table = p.cache.block_table + (size_t)entry * p.cache.max_pages;
  const int low = p.positions[token0 + row0 / p.groups], last = p.positions[token0 + (min(row0 + TILE_ROWS, total) - 1) / p.groups];
  const int lo = p.window > 0 ? max(0, low - p.window + 1) : 0;
  if (SPLIT && which == 0 && last >= p.spans * SPAN && threadIdx.x == 0) atomicOr(p.status, FE_STATUS_BAD_PAGE);   // past the block table
  const int stop = SPLIT ? min(last / SPAN, p.spans - 1) : 0;
  int span = SPLIT ? lo / SPAN + which : 0;
  if (span > stop) return;
  for (int i = threadIdx.x; i < TILE_ROWS * D; i += THREADS) {
    const int r = i / D, d = i - r * D, row = row0 + r;
    const int token = token0 + row / p.groups, head = kvh * p.groups + row % p.groups;
    qs[r * qpitch + d] = row < total ? to_float(((const T*)p.q)[(size_t)token * p.q_stride + (size_t)head * D + d]) : 0.f;
  }
  int from[RT], upto[RT];              // the positions this thread's rows see
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int row = row0 + ty * RT + i;
    upto[i] = row < total ? p.positions[token0 + row / p.groups] : -1;
    from[i] = p.window > 0 ? max(0, upto[i] - p.window + 1) : 0;
  }
  int column[CG];                      // columns past the head's last are its last ones again, and are not stored
#pragma unroll
  for (int g = 0; g < CG; ++g) column[g] = min(tx * 4 + 64 * g, D - 4);
  for (; span <= stop; span += p.share) {
    const int high = SPLIT ? min(last, span * SPAN + SPAN - 1) : last;
    // of the span at hand, and of the spans before it
    float m[RT], l[RT], top[SPLIT ? 1 : RT], den[SPLIT ? 1 : RT], num[SPLIT ? 1 : RT][CG][4];
    uint64_t acc[RT][CG][2];           // two neighbouring columns each
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
      if (!SPLIT) top[i] = -INFINITY, den[i] = 0.f;
#pragma unroll
      for (int g = 0; g < CG; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[i][g][e / 2] = 0;
          if (!SPLIT) num[i][g][e] = 0.f;
        }
    }
    for (int first = max(lo, SPLIT ? span * SPAN : 0) / TILE_KEYS * TILE_KEYS; first <= high; first += TILE_KEYS) {
      __syncthreads();
      stage_keys<T, TILE_KEYS, THREADS>(p, table, kvh, first, lo, high, ks, vs, ok);
      commit();
      wait<0>();
      __syncthreads();
      uint64_t dot[RT][4];
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dot[i][j] = 0;
#pragma unroll 4
      for (int d = 0; d < D; d += 4) {
        uint64_t a[RT][2], b[4][2];
#pragma unroll
        for (int i = 0; i < RT; ++i) pairs4(qs + (ty * RT + i) * qpitch + d, a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) pairs4(ks + (tx + 16 * j) * (D + CH) + d, b[j]);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) fma2(dot[i][j], a[i][e], b[j][e]);
      }
      // by row and thirty-two of keys: maxima, corrections of what came before, sums
      float score[RT][4], most[2 * RT], corr[2][RT];
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = first + tx + 16 * j;
          score[i][j] = ok[tx + 16 * j] && key >= from[i] && key <= upto[i] ? __fmul_rn(sum2(dot[i][j]), p.scale) : -INFINITY;
          if (j & 1) most[2 * i + j / 2] = fmaxf(score[i][j - 1], score[i][j]);
        }
      reduce_all<true>(most, threadIdx.x & 31);
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float now = fmaxf(m[i], most[2 * i + h]);
          corr[h][i] = m[i] == -INFINITY ? 0.f : expf(m[i] - now);
          m[i] = now;
          float e[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            e[j] = score[i][2 * h + j] == -INFINITY ? 0.f : expf(score[i][2 * h + j] - now);
            ps[(ty * RT + i) * P_PITCH + 32 * h + 16 * j + tx] = e[j];
          }
          most[2 * i + h] = e[0] + e[1];
        }
      reduce_all<false>(most, threadIdx.x & 31);
#pragma unroll
      for (int i = 0; i < RT; ++i) l[i] = fmaf(fmaf(l[i], corr[0][i], most[2 * i]), corr[1][i], most[2 * i + 1]);
      __syncwarp();                    // a row's probabilities are written and read by the same warp
      // Where some row of the tile does not see some key, that key's value is left out for it: a
      // zero probability would not keep an infinity out.
      const bool edge = first < max(0, p.window > 0 ? last - p.window + 1 : 0) || first + TILE_KEYS - 1 > low;
      for (int key = 0; key < TILE_KEYS; key += 4) {
        if (key % 32 == 0) {
#pragma unroll
          for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int g = 0; g < CG; ++g)
#pragma unroll
              for (int e = 0; e < 2; ++e) acc[i][g][e] = scale2(acc[i][g][e], key == 0 ? corr[0][i] : corr[1][i]);
        }
        float e[RT][4];
#pragma unroll
        for (int i = 0; i < RT; ++i) load4(ps + (ty * RT + i) * P_PITCH + key, e[i]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint64_t v[CG][2];
#pragma unroll
          for (int g = 0; g < CG; ++g) pairs4(vs + (key + u) * D + column[g], v[g]);
          auto add = [&](int i) {
            const uint64_t both = twice(e[i][u]);
#pragma unroll
            for (int g = 0; g < CG; ++g)
#pragma unroll
              for (int c = 0; c < 2; ++c) fma2(acc[i][g][c], both, v[g][c]);
          };
          if (!edge) {
#pragma unroll
            for (int i = 0; i < RT; ++i) add(i);
          } else {
#pragma unroll
            for (int i = 0; i < RT; ++i)
              if (first + key + u >= from[i] && first + key + u <= upto[i]) add(i);
          }
        }
      }
      if constexpr (!SPLIT) if ((first + TILE_KEYS) % SPAN == 0 || first + TILE_KEYS > high) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          float old, mine;
          fold_factors(top[i], m[i], old, mine);
          den[i] = fmaf(l[i], mine, __fmul_rn(den[i], old));
          m[i] = -INFINITY;
          l[i] = 0.f;
#pragma unroll
          for (int g = 0; g < CG; ++g)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              num[i][g][e] = fmaf(half2_of(acc[i][g][e / 2], e & 1), mine, __fmul_rn(num[i][g][e], old));
              if (e & 1) acc[i][g][e / 2] = 0;
            }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int row = row0 + ty * RT + i;
      if (row >= total) continue;
      if constexpr (SPLIT) {
        const size_t rows = (size_t)p.n_tokens * p.groups, at = ((size_t)span * nkv + kvh) * rows + (size_t)token0 * p.groups + row;
        float* sums = p.partial + at * D;
#pragma unroll
        for (int g = 0; g < CG; ++g)
          if (tx * 4 + 64 * g < D) *reinterpret_cast<ulonglong2*>(sums + tx * 4 + 64 * g) = make_ulonglong2(acc[i][g][0], acc[i][g][1]);
        if (tx == 0) *reinterpret_cast<float2*>(p.partial + (size_t)p.spans * nkv * rows * D + 2 * at) = make_float2(m[i], l[i]);
        continue;
      }
      T* out = (T*)p.out + ((size_t)(token0 + row / p.groups) * p.num_q_heads + kvh * p.groups + row % p.groups) * D;
#pragma unroll
      for (int g = 0; g < CG; ++g) {
        const int d = tx * 4 + 64 * g;
        if (d < D) {
          float o[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c] = den[SPLIT ? 0 : i] > 0.f ? num[SPLIT ? 0 : i][g][c] / den[SPLIT ? 0 : i] : 0.f;
          store4(out + d, o);
        }
      }
    }
  }
}

// What the split tile kernel left, a warp a row (token, query head): its spans in ascending order, as the tile kernel folds them.
template <typename T>
__global__ void __launch_bounds__(256) attention_simt_fold_kernel(const Simt p) {
  pdl_trigger();
  pdl_wait();
  const int D = p.cache.head_dim, lane = threadIdx.x & 31, index = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int token = index / p.num_q_heads, head = index % p.num_q_heads;
  if (token >= p.n_tokens) return;
  const int entry = p.token_entry[token];
  if (p.cu_tokens[entry + 1] - p.cu_tokens[entry] <= 1) return;
  const int pos = p.positions[token], lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
  const int from = lo / SPAN, to = min(pos / SPAN, p.spans - 1), kvh = head / p.groups;
  const size_t rows = (size_t)p.n_tokens * p.groups, row = (size_t)token * p.groups + head % p.groups;
  const float* ml = p.partial + (size_t)p.spans * p.cache.num_kv_heads * rows * D;
  T* out = (T*)p.out + ((size_t)token * p.num_q_heads + head) * D;
  for (int d = lane * 4; d < D; d += 128) {
    float num[4] = {0.f, 0.f, 0.f, 0.f}, den = 0.f, top = -INFINITY;
#pragma unroll 4
    for (int s = from; s <= to; ++s) {
      const size_t at = ((size_t)s * p.cache.num_kv_heads + kvh) * rows + row;
      const float2 has = *reinterpret_cast<const float2*>(ml + 2 * at);
      float part[4], old, mine;
      load4(p.partial + at * D + d, part);
      fold_factors(top, has.x, old, mine);
#pragma unroll
      for (int e = 0; e < 4; ++e) num[e] = fmaf(part[e], mine, __fmul_rn(num[e], old));
      den = fmaf(has.y, mine, __fmul_rn(den, old));
    }
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = den > 0.f ? num[e] / den : 0.f;
    store4(out + d, o);
  }
}

template <typename K, typename... A>
int launch(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  if (smem > 48 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
  }
  return fe_launch_dependent(kernel, grid, dim3(threads), smem, stream, args...);
}

int rows_of(int groups) { return groups <= 2 ? 2 : groups <= 4 ? 4 : groups <= 8 ? 8 : 16; }

// Floats of a unit's partial results, and how many units go through the workspace at once: all of them up to
// 128 MB (48 requests of 16 heads of 128 at 32,768 positions), then slices of them one after the other, so that one
// long request among many does not ask for its spans that many times.
constexpr long long SIMT_WORKSPACE = 1ll << 25;
long long unit_floats(int num_q_heads, int num_kv_heads, int head_dim, long long spans) {
  const int groups = num_q_heads / num_kv_heads, R = rows_of(groups);
  return (long long)num_kv_heads * ((groups + R - 1) / R) * spans * R * (head_dim + 2);
}
int units_at_once(int units, long long floats) {
  const long long most = SIMT_WORKSPACE / floats;
  return (int)(most < 1 ? 1 : most > 65535 ? (units < 65535 ? units : 65535) : most < units ? most : units);
}
long long spans_of(int max_pages, int page_size) {
  const long long spans = ((long long)max_pages * page_size + SPAN - 1) / SPAN;
  return spans < 1 ? 1 : spans;
}

template <typename T, int DMAX>
int run_spans(Simt p, cudaStream_t stream) {
  const int R = rows_of(p.groups), D = p.cache.head_dim;
  const size_t smem = (size_t)R * D * 4 + SPAN_STAGES * SPAN_KEYS * ((size_t)2 * D * sizeof(T) + 16);
  const int slice = units_at_once(p.units, unit_floats(p.num_q_heads, p.cache.num_kv_heads, D, p.spans));
  int code = 0;
  for (; p.unit0 < p.units && code == 0; p.unit0 += slice) {
    const int units = p.units - p.unit0 < slice ? p.units - p.unit0 : slice;
    const dim3 grid(p.spans, p.cache.num_kv_heads * p.row_tiles, units);
    if (R == 2) code = launch(attention_simt_span_kernel<T, 2, DMAX>, grid, SPAN_THREADS, smem, stream, p);
    else if (R == 4) code = launch(attention_simt_span_kernel<T, 4, DMAX>, grid, SPAN_THREADS, smem, stream, p);
    else if (R == 8) code = launch(attention_simt_span_kernel<T, 8, DMAX>, grid, SPAN_THREADS, smem, stream, p);
    else code = launch(attention_simt_span_kernel<T, 16, DMAX>, grid, SPAN_THREADS, smem, stream, p);
    if (code == 0) code = launch(attention_simt_merge_kernel<T>, dim3(units, p.num_q_heads), 128, 0, stream, p, R);
  }
  return code;
}

// Whether entries of several tokens are cut into spans of their keys: while their row tiles are fewer than 340 blocks (the
// chip holds 296, two an SM; 444 with heads of 64) and what the spans leave fits the workspace.  us, whole / in spans, 16 heads of 128: 250 tokens
// (136 blocks) 54 / 50, 500 (264) 105 / 104, 600 (312) 136 / 124, 700 (360) 150 / 157, 850 (432) 182 / 220; 100 after 5,000 cached ones
// (64) 740 / 275, 300 after 900 (160) 249 / 181, 700 after 400 (360) 242 / 278.  32 heads of 64: 250 tokens (264) 51 / 46, 500 (512)
// 93 / 112; 24 heads of 64 and one kv head: 500 (376) 92 / 85, 600 (451) 111 / 113; 40 in bfloat16: 250 (316) 54 / 54, 300 after 900 (378) 202 / 224.
long long tile_floats(int n_tokens, int num_q_heads, int num_kv_heads, int head_dim, long long spans, int units) {
  const long long tiles = ((long long)n_tokens * (num_q_heads / num_kv_heads) + TILE_ROWS - 1) / TILE_ROWS + units;
  const long long floats = (long long)n_tokens * num_q_heads * spans * (head_dim + 2);
  return spans < 2 || tiles * num_kv_heads >= 340 || floats > SIMT_WORKSPACE || spans * num_kv_heads > 65535 ? 0 : floats;
}

template <typename T, bool SPLIT>
int run_tiles(Simt p, cudaStream_t stream) {
  const int D = p.cache.head_dim;
  const size_t smem = (size_t)4 * TILE_ROWS * (D + 4 + P_PITCH) + (size_t)TILE_KEYS * (2 * D * sizeof(T) + 16);
  // tiles of all entries one after the other; an entry's last one may be short
  const long long heads = p.cache.num_kv_heads, tiles = ((long long)p.n_tokens * p.groups + TILE_ROWS - 1) / TILE_ROWS + p.units;
  // Blocks that share a tile: about eight times what the chip holds altogether, and no more than there are spans in a window.  How
  // many spans a tile has is known on the device; a block for each that the block table has room for took 190 us for a prompt of
  // 60 tokens beside a request of 32,768 (16 heads of 128; 28 now), and 81 for 100 tokens with a window of 256 (49).  With 600
  // blocks 200 tokens after 3,000 of 16 heads of 128 took 330 us, 1,200 304, 2,400 322, 4,700 331; 40 tokens beside 50 decoding
  // requests, 16 heads of 96, 153, 135, 111 and 111.
  p.share = 1;
  if (SPLIT) {
    long long share = std::min<long long>(p.spans, (8 * 296 + tiles * heads - 1) / (tiles * heads));
    if (p.window > 0) share = std::min<long long>(share, ((long long)p.window + TILE_ROWS / p.groups + SPAN) / SPAN + 1);
    p.share = (int)share;
  }
  if (tiles * heads * p.share > 0x7fffffffLL) return FE_ERR_TOO_LARGE;
  const dim3 grid((unsigned)(tiles * heads * p.share));
  // Threads: what a block holds in shared memory leaves three blocks an SM with up to 32 KB of keys and values (heads of 64, of 128 in
  // bfloat16); four warps of four rows a thread then read less for a multiply-add than eight of two.  Otherwise two blocks fit, and eight
  // warps hide more.  us, 128 / 256 threads: 2,048 tokens of 32 heads of 64 991 / 1,094, 40 heads of 64 in bfloat16 1,167 / 1,528, of 128
  // 1,692 / 1,997; 16 heads of 128 1,261 (other changes besides) / 955.
  constexpr int SMALL = 128, LARGE = 256, MID = sizeof(T) == 2 ? SMALL : LARGE;
  int code;
  if (D <= 64) code = launch(attention_simt_tile_kernel<T, 64, SPLIT, SMALL>, grid, SMALL, smem, stream, p);
  else if (D <= 128) code = launch(attention_simt_tile_kernel<T, 128, SPLIT, MID>, grid, MID, smem, stream, p);
  else code = launch(attention_simt_tile_kernel<T, 256, SPLIT, LARGE>, grid, LARGE, smem, stream, p);
  if (code || !SPLIT) return code;
  const long long rows = (long long)p.n_tokens * p.num_q_heads;
  return launch(attention_simt_fold_kernel<T>, dim3((unsigned)((rows + 7) / 8)), 256, 0, stream, p);
}

template <typename T>
int run(const Simt& p, int n_tokens, int max_new, cudaStream_t stream) {
  // units that bring several tokens, then those that bring one; a step of one prompt has none of these
  if (p.cu_tokens != nullptr && max_new > 1) {
    const bool split = tile_floats(n_tokens, p.num_q_heads, p.cache.num_kv_heads, p.cache.head_dim, p.spans, p.units) > 0;
    const int code = split ? run_tiles<T, true>(p, stream) : run_tiles<T, false>(p, stream);
    if (code) return code;
    if (p.units == 1 && n_tokens > 1) return 0;
  }
  return p.cache.head_dim <= 128 ? run_spans<T, 128>(p, stream) : run_spans<T, 256>(p, stream);
}

}  // namespace

// For `units` single tokens whose block tables are `max_pages` wide: how many of them are worked on at
// once, and the floats of workspace those take.
FE_EXPORT int fe_attention_simt_units(int units, int num_q_heads, int num_kv_heads, int head_dim, int max_pages, int page_size) {
  if (units <= 0 || num_kv_heads <= 0 || num_q_heads <= 0 || num_q_heads % num_kv_heads) return 0;
  return units_at_once(units, unit_floats(num_q_heads, num_kv_heads, head_dim, spans_of(max_pages, page_size)));
}
FE_EXPORT long long fe_attention_simt_scratch(int units, int num_q_heads, int num_kv_heads, int head_dim, int max_pages, int page_size) {
  const int slice = fe_attention_simt_units(units, num_q_heads, num_kv_heads, head_dim, max_pages, page_size);
  return slice == 0 ? 0 : slice * unit_floats(num_q_heads, num_kv_heads, head_dim, spans_of(max_pages, page_size));
}

// The floats of workspace that entries of several tokens take (0: none), for `n_tokens` tokens of `units` entries.
FE_EXPORT long long fe_attention_simt_tile_scratch(int n_tokens, int units, int num_q_heads, int num_kv_heads, int head_dim, int max_pages,
                                                   int page_size) {
  if (num_kv_heads <= 0 || num_q_heads <= 0 || num_q_heads % num_kv_heads) return 0;
  return tile_floats(n_tokens, num_q_heads, num_kv_heads, head_dim, spans_of(max_pages, page_size), units);
}

// `cu_tokens` [units + 1] says which tokens each unit (an entry: row u of the block table, positions
// in order) brings, at most `max_new`; null: every token is a unit and `token_entry` names its row.
FE_EXPORT int fe_attention_simt(const void* q, int q_stride, int dtype, const void* k_cache,
                                const void* v_cache, const int* block_table, int max_pages,
                                int page_size, int num_pages, const int* positions,
                                const int* token_entry, const int* cu_tokens, int units, int max_new,
                                int window, float scale, void* out,
                                int num_q_heads, int num_kv_heads, int head_dim, int n_tokens,
                                float* workspace, int* status, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (head_dim % 8 || head_dim > 256 || head_dim < 8) return FE_ERR_BAD_SHAPE;
  if (num_kv_heads <= 0 || num_q_heads % num_kv_heads || num_q_heads > 65535) return FE_ERR_BAD_SHAPE;
  if (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) return FE_ERR_BAD_ALIGN;
  if (cu_tokens == nullptr) units = n_tokens;
  PagedKV cache{k_cache, v_cache, block_table, max_pages, page_size, num_pages, num_kv_heads, head_dim};
  const int groups = num_q_heads / num_kv_heads, R = rows_of(groups);
  const long long spans = spans_of(max_pages, page_size);
  const int row_tiles = (groups + R - 1) / R;
  if (spans > 0x7fffffff || (long long)num_kv_heads * row_tiles > 65535) return FE_ERR_TOO_LARGE;
  Simt p{q, q_stride, cache, positions, token_entry, cu_tokens, units, window, scale, out, num_q_heads, groups,
         (int)spans, row_tiles, 0, workspace, n_tokens, 1, status};
  if (dtype == FE_DTYPE_F32) return run<float>(p, n_tokens, max_new, stream);
  if (dtype == FE_DTYPE_BF16) return run<bf16>(p, n_tokens, max_new, stream);
  return FE_ERR_BAD_DTYPE;
}

// Next-token choice from rows of 32-bit logits: argmax, or temperature -> top-k ->
// top-p -> min-p -> softmax -> one draw, in the order of upstream's filter
// (src/forge_engine/sampling.py:49-140).  One block per row; nothing is sorted:
// the k-th largest value and the nucleus boundary are found by a 4-pass radix
// search over an order-preserving integer image of the shifted logits, with counts
// and fixed-point probability mass per digit, so that the result does not depend on
// the order in which threads arrive.  Groups of warps count into histograms of their own
// in shared memory (a vocabulary's keys fall into a handful of digits in the first pass: one
// shared histogram would serialise 150,000 atomic adds on five addresses), and the
// histograms are added up after each pass.
//
// Ties: among values equal to the k-th largest, the lowest indices are kept (exactly
// k survive).  Values equal to the nucleus boundary are all kept.
// A block keeps its slice of the row, shifted and divided by the temperature, in shared memory where
// it fits, so that only the first pass reads the logits; the digit that a pass decides on is found
// by a warp.  (16 rows of 151,936, top-k 50 and top-p 0.95: 199 us with the slice read from L2 in
// every pass and a single thread walking the 256 digits.)
// With a top-k of up to 512 the passes are not taken: a bound from the threads' maxima leaves a few hundred elements, and
// one block decides among them without a barrier of the cluster (the same 16 rows 93 us by passes, 34 this way; top-k 200 94 and
// 38, 512 95 and 47; 64 rows 179 and 63; 16 rows of 32,000 43 and 26).  More than 1,024 elements above the bound (ties, or
// the largest all in one block's slice) go through the passes.
// The draw: u = uniform(seed, counter) from a counter hash (see fe_uniform below and
// its Python twin), target = u * sum(weights of survivors), first index whose running
// sum in index order exceeds target.
#include "common.cuh"

#include <atomic>

#define FE_STATUS_BAD_LOGITS 16
#define SMP_THREADS 1024
#define MASS_SCALE 1099511627776.0f  // 2^40
#define SMP_GROUPS 8                 // histogram copies; warp w counts into copy w % 8

__host__ __device__ inline unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// 24 random bits -> [0, 1).  The same two lines in Python give the same number.
__host__ __device__ inline float fe_uniform(unsigned long long seed, unsigned long long counter) {
  const unsigned long long h = splitmix64(splitmix64(seed) ^ (counter * 0xD1342543DE82EF95ull));
  return (float)(h >> 40) * (1.0f / 16777216.0f);
}

__device__ __forceinline__ unsigned int float_key(float x) {
  const unsigned int u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct Survive {
  unsigned int thr_key;  // keep key > thr_key
  int tie_cut;           // keep key == thr_key only for index <= tie_cut
  float min_w;           // keep exp(x) >= min_w
};

__device__ __forceinline__ bool survives(const Survive& s, unsigned int key, int index, float w) {
  if (w < s.min_w) return false;
  return key > s.thr_key || (key == s.thr_key && index <= s.tie_cut);
}

// Exclusive scan of one value per thread in thread order; total returned to everyone.
template <typename V>
__device__ V block_exclusive_scan(V v, V* scratch /* 33 */, V* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    V w = scratch[lane];
    V winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    scratch[lane] = winc - w;
    if (lane == 31) scratch[32] = winc;
  }
  __syncthreads();
  *total = scratch[32];
  return scratch[warp] + inc - v;
}

// ---- the blocks of a row's cluster ----
// A row is cut into `parts` contiguous slices of the vocabulary, one per block of a
// thread-block cluster (1 block: no cluster).  What the blocks have to agree on - the
// maximum, histograms, counts, sums - every block leaves in its own shared memory, and after
// one cluster barrier every block reads all of them in block order, so that all reach the
// same decision.  Buffers alternate between two copies: a block can be at most one
// exchange ahead of the slowest reader.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned int peer_address(const void* mine, int rank) {
  unsigned int remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(remote) : "r"((unsigned int)__cvta_generic_to_shared(mine)), "r"(rank));
  return remote;
}
__device__ __forceinline__ unsigned int peer_u32(const void* mine, int rank) {
  unsigned int v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_address(mine, rank)) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long peer_u64(const void* mine, int rank) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(peer_address(mine, rank)) : "memory");
  return v;
}

// Place of logit i of a slice in shared memory: threads that walk neighbouring stretches of a power of
// two meet in different banks.
__host__ __device__ __forceinline__ int slice_at(int i) { return i + (i >> 5); }

// Digit in which the count of the largest keys reaches `want`, by one warp; *left: how many of that digit
// are wanted.  Digit 0 where all of them together do not.
__device__ __forceinline__ int digit_of_count(const unsigned int* n, int want, int* left) {
  const int lane = threadIdx.x & 31, top = 255 - 8 * lane;      // this lane's digits top .. top - 7
  int sum = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) sum += (int)n[top - b];
  int upto = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  int remaining = want - (upto - sum), digit = -1;
  if (remaining > 0) {
    for (int b = 0; b < 8 && digit < 0; ++b) {
      const int have = (int)n[top - b];
      if (have >= remaining || top - b == 0) digit = top - b;
      else remaining -= have;
    }
  }
  const unsigned found = __ballot_sync(0xffffffffu, digit >= 0);
  const int owner = found ? __ffs(found) - 1 : 31;
  *left = __shfl_sync(0xffffffffu, remaining, owner);
  return max(0, __shfl_sync(0xffffffffu, digit, owner));
}

// The smallest digit with keys whose mass above it (`above` and that of the larger digits) is at most
// `limit`, by one warp; the largest digit with keys where there is none.  *mass: the mass above it.
__device__ __forceinline__ int digit_of_mass(const unsigned int* n, const unsigned long long* m, unsigned long long above,
                                             unsigned long long limit, unsigned long long* mass) {
  const int lane = threadIdx.x & 31, top = 255 - 8 * lane;
  unsigned long long sum = 0ull;
  int largest = -1;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (n[top - b] == 0u) continue;
    sum += m[top - b];
    if (largest < 0) largest = top - b;
  }
  unsigned long long upto = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  unsigned long long here = above + (upto - sum), chosen_above = here;
  int chosen = -1;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (n[top - b] == 0u) continue;
    if (here <= limit) { chosen = top - b; chosen_above = here; }
    here += m[top - b];
  }
  const unsigned fits = __ballot_sync(0xffffffffu, chosen >= 0), any = __ballot_sync(0xffffffffu, largest >= 0);
  if (fits) {
    const int owner = 31 - __clz(fits);
    *mass = __shfl_sync(0xffffffffu, chosen_above, owner);
    return __shfl_sync(0xffffffffu, chosen, owner);
  }
  *mass = above;
  return any ? __shfl_sync(0xffffffffu, largest, __ffs(any) - 1) : 0;
}

// What a row is sampled with.
struct SampleRow {
  float temperature, top_p, min_p;
  int top_k;
  unsigned long long seed, counter;
};
// Up to SMP_ROWS_BY_VALUE rows travel as an argument of the kernel (no copy to the device goes ahead of it), more as arrays there.
#define SMP_ROWS_BY_VALUE 64
struct SampleParams {
  const float* temperature;     // null: 0
  const int* top_k;
  const float* top_p;
  const float* min_p;
  const unsigned long long* seeds;
  const unsigned long long* counters;
  int by_value;
  SampleRow rows[SMP_ROWS_BY_VALUE];
  __device__ __forceinline__ SampleRow of(int row) const {
    if (by_value) return rows[row];
    return SampleRow{temperature ? temperature[row] : 0.f, top_p ? top_p[row] : 1.f, min_p ? min_p[row] : 0.f, top_k ? top_k[row] : 0,
                     seeds ? seeds[row] : 0ull, counters ? counters[row] : 0ull};
  }
};

#define FEW_MOST 512                 // a top-k up to which the largest keys are collected

// Top-k, top-p, min-p and the draw among `n` <= 1,024 elements that hold the row's k largest, in index order (s: shifted
// logits, index: their places): the element drawn, or -1.  Thread t holds element t; `room`: 16 KB.  One block; the sums
// are added up as by a cluster of `parts` blocks whose threads walk stretches of the row.
__device__ int choose_of_few(const float* s_in, const int* index_in, int n, int k, float p, float mp, float u, int vocab, int parts,
                             unsigned char* room, unsigned long long* scan_u, float* scan_f, int* scan_i, int* red_i) {
  unsigned long long* mass = reinterpret_cast<unsigned long long*>(room);        // [512] of the k survivors
  float* s_of = reinterpret_cast<float*>(mass + FEW_MOST);                        // [512]
  float* w_of = s_of + FEW_MOST;
  int* index_of = reinterpret_cast<int*>(w_of + FEW_MOST);
  int* lives = index_of + FEW_MOST;
  float* walked = reinterpret_cast<float*>(lives + FEW_MOST);                     // [1024] sums of a block's threads
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // top-k: the k-th largest key, bit by bit; of the keys equal to it the first in index order
  {
    const bool have = tid < n;
    const float s = have ? s_in[tid] : 0.f;
    const unsigned int key = have ? float_key(s) : 0u;
    unsigned int threshold = 0u;
#pragma unroll 1
    for (int bit = 31; bit >= 0; --bit) {
      const unsigned int trial = threshold | (1u << bit);
      if (__syncthreads_count(have && key >= trial) >= k) threshold = trial;
    }
    const int ties = k - __syncthreads_count(have && key > threshold);
    int total;
    const int before = block_exclusive_scan<int>(have && key == threshold ? 1 : 0, scan_i, &total);
    const bool keep = have && (key > threshold || (key == threshold && before < ties));
    const int at = block_exclusive_scan<int>(keep ? 1 : 0, scan_i, &total);
    if (keep) { s_of[at] = s; index_of[at] = index_in[tid]; }
    n = total;
    __syncthreads();
  }
  const bool have = tid < n;
  const float s = have ? s_of[tid] : 0.f, w = have ? expf(s) : 0.f;
  const int index = have ? index_of[tid] : 0;
  const unsigned int key = float_key(s);
  bool live = have;
  // top-p: the smallest key whose mass of strictly larger survivors is at most p of all
  if (p < 1.f) {
    const unsigned long long own = have ? (unsigned long long)(w * MASS_SCALE) : 0ull;
    if (have) mass[tid] = own;
    unsigned long long total;
    block_exclusive_scan<unsigned long long>(own, scan_u, &total);
    const unsigned long long limit = (unsigned long long)((double)p * (double)total);
    unsigned long long above = 0ull;
    if (have)
      for (int j = 0; j < n; ++j)
        if (float_key(s_of[j]) > key) above += mass[j];
    unsigned int boundary = have && above <= limit ? key : 0xffffffffu;
    boundary = __reduce_min_sync(0xffffffffu, boundary);
    __syncthreads();
    if (lane == 0) red_i[warp] = (int)boundary;
    __syncthreads();
    boundary = __reduce_min_sync(0xffffffffu, (unsigned int)red_i[lane]);
    live = live && key >= boundary;
  }
  if (mp > 0.f) live = live && !(w < mp);
  if (have) { w_of[tid] = w; lives[tid] = live ? 1 : 0; }
  // the draw in index order: the first element of every (block, thread) stretch adds up the stretch
  const int chunk = (vocab + parts - 1) / parts;
  auto owner_of = [&](int i) {
    const int block = i / chunk, first = block * chunk, last = min(vocab, first + chunk);
    return block * SMP_THREADS + (i - first) / ((last - first + SMP_THREADS - 1) / SMP_THREADS);
  };
  const int owner = have ? owner_of(index) : -1;
  __syncthreads();
  const bool leads = have && (tid == 0 || owner_of(index_of[tid - 1]) != owner);
  float sum = 0.f;
  int end = tid, last = -1;
  if (leads) {
    do {
      if (lives[end]) { sum += w_of[end]; last = end; }
      ++end;
    } while (end < n && owner_of(index_of[end]) == owner);
  }
  float total = 0.f, before = 0.f;
  for (int r = 0; r < parts; ++r) {
    const bool here = leads && owner / SMP_THREADS == r;
    walked[tid] = 0.f;
    __syncthreads();
    if (here) walked[owner % SMP_THREADS] = sum;
    __syncthreads();
    const float mine = walked[tid];
    float block_total;
    const float upto = block_exclusive_scan<float>(mine, scan_f, &block_total);
    walked[tid] = upto + total;
    __syncthreads();
    if (here) before = walked[owner % SMP_THREADS];
    total += block_total;
    __syncthreads();
  }
  const float target = u * total;
  int best = last >= 0 && before <= target ? owner : -1;
  best = __reduce_max_sync(0xffffffffu, best);
  if (lane == 0) red_i[warp] = best;
  __syncthreads();
  best = __reduce_max_sync(0xffffffffu, red_i[lane]);
  __syncthreads();
  if (tid == 0) red_i[0] = -1;
  __syncthreads();
  if (leads && owner == best) {
    float c = before;
    int pick = last;
    for (int j = tid; j < end; ++j) {
      if (!lives[j]) continue;
      c += w_of[j];
      if (target < c) { pick = j; break; }
    }
    red_i[0] = index_of[pick];
  }
  __syncthreads();
  return red_i[0];
}

__global__ void __launch_bounds__(SMP_THREADS)
sample_kernel(const float* __restrict__ logits, int vocab, const __grid_constant__ SampleParams params,
              int* __restrict__ out, int* status, int keep_slice) {
  extern __shared__ float slice[];                   // with keep_slice: this block's shifted logits
  __shared__ float red_v[32];
  __shared__ int red_i[32];
  __shared__ unsigned int hist_n[2][256];            // this block's counts per digit (two copies, see above)
  __shared__ unsigned long long hist_m[2][256];      // ... and masses
  __shared__ unsigned int all_n[256];                // the row's counts per digit
  __shared__ unsigned long long all_m[256];
  __shared__ unsigned long long group_m[SMP_GROUPS * 256];
  __shared__ unsigned int group_n[SMP_GROUPS * 256];
  __shared__ unsigned long long share[2][2];         // scalars handed to the other blocks
  __shared__ unsigned long long scan_u[33];
  __shared__ float scan_f[33];
  __shared__ int scan_i[33];
  __shared__ unsigned int sh_prefix;
  __shared__ unsigned long long sh_mass_above;
  __shared__ int sh_remaining;
  __shared__ int sh_pick;

  const int parts = gridDim.x, part = blockIdx.x, row = blockIdx.y;
  const float* x = logits + (size_t)row * vocab;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = warp % SMP_GROUPS;
  const int chunk = (vocab + parts - 1) / parts;
  const int lo = min(vocab, part * chunk), hi = min(vocab, lo + chunk);   // this block's slice
  int turn = 0;                                                            // which copy the next exchange uses

  // ---- argmax, lowest index on ties; NaN and +inf are reported ----
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  bool bad = false;
#pragma unroll 4
  for (int i = lo + tid; i < hi; i += SMP_THREADS) {
    const float v = x[i];
    if (keep_slice) slice[slice_at(i - lo)] = v;
    if (v != v || v == INFINITY) bad = true;
    if (v > best) { best = v; best_i = i; }
  }
  const float own_max = best;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
  }
  if (lane == 0) { red_v[warp] = best; red_i[warp] = best_i; }
  if (bad) atomicOr(status, FE_STATUS_BAD_LOGITS);
  __syncthreads();
  if (warp == 0) {
    best = red_v[lane];
    best_i = red_i[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (lane == 0) { share[turn][0] = __float_as_uint(best); share[turn][1] = (unsigned long long)(unsigned int)best_i; }
  }
  cluster_sync();
  float row_max = -INFINITY;
  int arg = 0x7fffffff;
  for (int r = 0; r < parts; ++r) {       // slices are in index order: the first of equal maxima wins
    const float v = __uint_as_float((unsigned int)peer_u64(&share[turn][0], r));
    const int at = (int)(unsigned int)peer_u64(&share[turn][1], r);
    if (v > row_max || (v == row_max && at < arg)) { row_max = v; arg = at; }
  }
  turn ^= 1;
  if (arg == 0x7fffffff) arg = 0;
  const SampleRow wish = params.of(row);
  const float temp = wish.temperature;
  if (temp <= 0.f || row_max == -INFINITY) {
    if (tid == 0 && part == 0) out[row] = arg;
    cluster_sync();        // nobody leaves while another block may still read its shared memory
    return;
  }
  const float inv_t = 1.f / temp, p = wish.top_p, mp = wish.min_p, u = fe_uniform(wish.seed, wish.counter);
  const int k = wish.top_k;

  // ---- few wanted: the largest keys alone ----
  // Two lower bounds of the row's k-th largest key (their upper 20 bits): the best block's k-th largest of its threads'
  // maxima, and the worst block's (k / blocks)-th largest.  What reaches the larger of the two is collected in
  // index order in the first block, which decides among it: the same survivors, and the same sums in the same
  // order, as the passes over the whole row below.
  if (keep_slice && k > 0 && k <= FEW_MOST && k < vocab) {
    const unsigned int top_key = float_key((own_max - row_max) * inv_t);
    const int fair = (k + parts - 1) / parts;
    unsigned int bound = 0u, fair_bound = 0u;
#pragma unroll 1
    for (int bit = 31; bit >= 12; --bit) {
      const unsigned int trial = bound | (1u << bit), fair_trial = fair_bound | (1u << bit);
      if (__syncthreads_count(top_key >= trial) >= k) bound = trial;
      if (__syncthreads_count(top_key >= fair_trial) >= fair) fair_bound = fair_trial;
    }
    if (tid == 0) { share[turn][0] = bound; share[turn][1] = fair_bound; }
    cluster_sync();
    for (int r = 0; r < parts; ++r) {
      bound = max(bound, (unsigned int)peer_u64(&share[turn][0], r));
      fair_bound = min(fair_bound, (unsigned int)peer_u64(&share[turn][1], r));
    }
    bound = max(bound, fair_bound);
    turn ^= 1;
    const int seg = (hi - lo + SMP_THREADS - 1) / SMP_THREADS;
    const int begin = min(hi, lo + tid * seg), end = min(hi, begin + seg);
    int mine = 0, total;
    for (int i = begin; i < end; ++i) mine += float_key((slice[slice_at(i - lo)] - row_max) * inv_t) >= bound;
    int at = block_exclusive_scan<int>(mine, scan_i, &total);
    if (tid == 0) share[turn][0] = (unsigned long long)(unsigned int)total;
    cluster_sync();
    int all = 0;
    for (int r = 0; r < parts; ++r) {
      const int theirs = (int)(unsigned int)peer_u64(&share[turn][0], r);
      if (r < part) at += theirs;
      all += theirs;
    }
    turn ^= 1;
    if (all <= SMP_THREADS) {
      float* few_s = reinterpret_cast<float*>(group_n);        // [1024] shifted logits, [1024] indices
      int* few_i = reinterpret_cast<int*>(group_n) + SMP_THREADS;
      if (mine > 0) {
        const unsigned int to_s = peer_address(few_s, 0), to_i = peer_address(few_i, 0);
        for (int i = begin; i < end; ++i) {
          const float s = (slice[slice_at(i - lo)] - row_max) * inv_t;
          if (float_key(s) < bound) continue;
          asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to_s + 4u * (unsigned)at), "f"(s) : "memory");
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to_i + 4u * (unsigned)at), "r"(i) : "memory");
          ++at;
        }
      }
      cluster_sync();
      if (part == 0) {
        const int pick = choose_of_few(few_s, few_i, all, k, p, mp, u, vocab, parts, reinterpret_cast<unsigned char*>(group_m), scan_u, scan_f,
                                       scan_i, red_i);
        if (tid == 0) out[row] = pick < 0 ? arg : pick;
      }
      return;
    }
  }
  Survive keep{0u, 0x7fffffff, 0.f};
  if (keep_slice) {
    for (int i = lo + tid; i < hi; i += SMP_THREADS) slice[slice_at(i - lo)] = (slice[slice_at(i - lo)] - row_max) * inv_t;
    __syncthreads();
  }
#define SHIFTED(i) (keep_slice ? slice[slice_at((i) - lo)] : (x[i] - row_max) * inv_t)
  // after the blocks' histograms are complete: add them up over the cluster, in block order
#define GATHER_HISTOGRAMS(WITH_MASS)                                                                  \
  do {                                                                                                \
    if (tid < 256) {                                                                                  \
      unsigned int n = 0u;                                                                            \
      unsigned long long m = 0ull;                                                                    \
      for (int w = 0; w < SMP_GROUPS; ++w) {                                                          \
        n += group_n[w * 256 + tid];                                                                  \
        if (WITH_MASS) m += group_m[w * 256 + tid];                                                   \
      }                                                                                               \
      hist_n[turn][tid] = n;                                                                          \
      if (WITH_MASS) hist_m[turn][tid] = m;                                                           \
    }                                                                                                 \
    cluster_sync();                                                                                   \
    if (tid < 256) {                                                                                  \
      unsigned int n = 0u;                                                                            \
      unsigned long long m = 0ull;                                                                    \
      for (int r = 0; r < parts; ++r) {                                                               \
        n += peer_u32(&hist_n[turn][tid], r);                                                         \
        if (WITH_MASS) m += peer_u64(&hist_m[turn][tid], r);                                          \
      }                                                                                               \
      all_n[tid] = n;                                                                                 \
      if (WITH_MASS) all_m[tid] = m;                                                                  \
    }                                                                                                 \
    turn ^= 1;                                                                                        \
    __syncthreads();                                                                                  \
  } while (0)

  // ---- top-k: radix search for the k-th largest key ----
  if (k > 0 && k < vocab) {
    if (tid == 0) { sh_prefix = 0u; sh_remaining = k; }
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int b = tid; b < SMP_GROUPS * 256; b += SMP_THREADS) group_n[b] = 0u;
      __syncthreads();
      const unsigned int prefix = sh_prefix;
      const unsigned int mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
      if (shift == 24) {
        // first pass: every key takes part and they fall into a handful of digits; lanes of
        // a warp that hit the same digit add together, one atomic per digit and warp step
        for (int base = lo; base < hi; base += SMP_THREADS) {
          const int i = base + tid;
          const unsigned int digit = i < hi ? (float_key(SHIFTED(i)) >> 24) : 0xffffffffu;
          const unsigned int peers = __match_any_sync(0xffffffffu, digit);
          if (digit != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&group_n[group * 256 + digit], (unsigned int)__popc(peers));
        }
      } else {
        for (int i = lo + tid; i < hi; i += SMP_THREADS) {
          const unsigned int key = float_key(SHIFTED(i));
          if ((key & mask) == prefix) atomicAdd(&group_n[group * 256 + ((key >> shift) & 255u)], 1u);
        }
      }
      __syncthreads();
      GATHER_HISTOGRAMS(false);
      if (warp == 0) {
        int left;
        const int digit = digit_of_count(all_n, sh_remaining, &left);
        __syncwarp();
        if (lane == 0) {
          sh_prefix = prefix | ((unsigned int)digit << shift);
          sh_remaining = left;  // how many of the chosen digit are still wanted
        }
      }
      __syncthreads();
    }
    keep.thr_key = sh_prefix;
    const int want_ties = sh_remaining;
    // the want_ties lowest indices among keys equal to the threshold survive
    const int seg = (hi - lo + SMP_THREADS - 1) / SMP_THREADS;
    const int begin = min(hi, lo + tid * seg), end = min(hi, begin + seg);
    int mine = 0;
    for (int i = begin; i < end; ++i) mine += float_key(SHIFTED(i)) == keep.thr_key;
    int total;
    int before = block_exclusive_scan<int>(mine, scan_i, &total);
    if (tid == 0) { share[turn][0] = (unsigned long long)(unsigned int)total; sh_pick = 0x7fffffff; }
    cluster_sync();
    int all_total = 0;
    for (int r = 0; r < parts; ++r) {
      const int theirs = (int)(unsigned int)peer_u64(&share[turn][0], r);
      if (r < part) before += theirs;
      all_total += theirs;
    }
    turn ^= 1;
    if (all_total > want_ties && before < want_ties && before + mine >= want_ties) {
      int seen = before;
      for (int i = begin; i < end; ++i) {
        if (float_key(SHIFTED(i)) == keep.thr_key && ++seen == want_ties) { sh_pick = i; break; }
      }
    }
    __syncthreads();
    if (tid == 0) share[turn][0] = (unsigned long long)(unsigned int)sh_pick;
    cluster_sync();
    int cut = 0x7fffffff;
    for (int r = 0; r < parts; ++r) cut = min(cut, (int)(unsigned int)peer_u64(&share[turn][0], r));
    turn ^= 1;
    keep.tie_cut = cut;
    __syncthreads();
  }

  // ---- top-p: smallest key whose mass of strictly larger survivors is <= top_p * Z ----
  if (p < 1.f) {
    if (tid == 0) { sh_prefix = 0u; sh_mass_above = 0ull; }
    unsigned long long limit = 0ull;
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int b = tid; b < SMP_GROUPS * 256; b += SMP_THREADS) { group_n[b] = 0u; group_m[b] = 0ull; }
      __syncthreads();
      const unsigned int prefix = sh_prefix;
      const unsigned int mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
      unsigned long long local_total = 0ull;
      if (shift == 24) {
        // first pass: the survivors fall into a handful of digits.  Lanes that hit the same
        // digit add their masses together (in two 20-bit halves, so that 32 of them fit the
        // 32-bit warp reduction) and one of them does the atomics
        for (int base = lo; base < hi; base += SMP_THREADS) {
          const int i = base + tid;
          unsigned int digit = 0xffffffffu;
          unsigned long long mass = 0ull;
          if (i < hi) {
            const float s = SHIFTED(i);
            const unsigned int key = float_key(s);
            const float w = expf(s);
            if (survives(keep, key, i, w)) {
              mass = (unsigned long long)(w * MASS_SCALE);      // at most 2^40
              local_total += mass;
              digit = key >> 24;
            }
          }
          const unsigned int peers = __match_any_sync(0xffffffffu, digit);
          const unsigned int low = __reduce_add_sync(peers, (unsigned int)(mass & 0xfffffull));
          const unsigned int high = __reduce_add_sync(peers, (unsigned int)(mass >> 20));
          if (digit != 0xffffffffu && lane == __ffs(peers) - 1) {
            atomicAdd(&group_n[group * 256 + digit], (unsigned int)__popc(peers));
            atomicAdd(&group_m[group * 256 + digit], ((unsigned long long)high << 20) + low);
          }
        }
      } else {
        for (int i = lo + tid; i < hi; i += SMP_THREADS) {
          const float s = SHIFTED(i);
          const unsigned int key = float_key(s);
          if ((key & mask) != prefix) continue;
          const float w = expf(s);
          if (!survives(keep, key, i, w)) continue;
          atomicAdd(&group_n[group * 256 + ((key >> shift) & 255u)], 1u);
          atomicAdd(&group_m[group * 256 + ((key >> shift) & 255u)], (unsigned long long)(w * MASS_SCALE));
        }
      }
      if (shift == 24) {
        unsigned long long total;
        block_exclusive_scan<unsigned long long>(local_total, scan_u, &total);
        if (tid == 0) share[turn][1] = total;     // read after the barrier inside the gather below
      }
      __syncthreads();
      const int shared_turn = turn;
      GATHER_HISTOGRAMS(true);
      if (shift == 24) {
        unsigned long long total = 0ull;
        for (int r = 0; r < parts; ++r) total += peer_u64(&share[shared_turn][1], r);
        limit = (unsigned long long)((double)p * (double)total);
      }
      if (warp == 0) {
        unsigned long long above;
        const int digit = digit_of_mass(all_n, all_m, sh_mass_above, limit, &above);
        __syncwarp();
        if (lane == 0) {
          sh_prefix = prefix | ((unsigned int)digit << shift);
          sh_mass_above = above;
        }
      }
      __syncthreads();
    }
    const unsigned int boundary = sh_prefix;
    if (boundary > keep.thr_key) { keep.thr_key = boundary; keep.tie_cut = 0x7fffffff; }
    __syncthreads();
  }

  // ---- min-p: drop p_i < min_p * p_max  <=>  exp(x_i) < min_p (the largest has exp 1) ----
  if (mp > 0.f) keep.min_w = mp;

  // ---- draw in index order ----
  const int seg = (hi - lo + SMP_THREADS - 1) / SMP_THREADS;
  const int begin = min(hi, lo + tid * seg), end = min(hi, begin + seg);
  float mine = 0.f;
  int last_survivor = -1;
  for (int i = begin; i < end; ++i) {
    const float s = SHIFTED(i);
    const float w = expf(s);
    if (survives(keep, float_key(s), i, w)) { mine += w; last_survivor = i; }
  }
  float block_total;
  float before = block_exclusive_scan<float>(mine, scan_f, &block_total);
  if (tid == 0) share[turn][0] = __float_as_uint(block_total);
  cluster_sync();
  float total = 0.f, earlier = 0.f;
  for (int r = 0; r < parts; ++r) {
    const float theirs = __uint_as_float((unsigned int)peer_u64(&share[turn][0], r));
    if (r == part) earlier = total;         // the sum of the slices before this one, in block order
    total += theirs;
  }
  turn ^= 1;
  before += earlier;
  const float target = u * total;
  // the last thread (in index order over the whole row) that has survivors and starts at or below target
  int cand = (last_survivor >= 0 && before <= target) ? part * SMP_THREADS + tid : -1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cand = max(cand, __shfl_xor_sync(0xffffffffu, cand, o));
  __syncthreads();
  if (lane == 0) red_i[warp] = cand;
  __syncthreads();
  if (warp == 0) {
    cand = red_i[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cand = max(cand, __shfl_xor_sync(0xffffffffu, cand, o));
    if (lane == 0) share[turn][0] = (unsigned long long)(unsigned int)cand;
  }
  cluster_sync();
  int owner = -1;
  for (int r = 0; r < parts; ++r) owner = max(owner, (int)(unsigned int)peer_u64(&share[turn][0], r));
  turn ^= 1;
  if (owner < 0) {
    if (tid == 0 && part == 0) out[row] = arg;
  } else if (part * SMP_THREADS + tid == owner) {
    float c = before;
    int pick = last_survivor;
    for (int i = begin; i < end; ++i) {
      const float s = SHIFTED(i);
      const float w = expf(s);
      if (!survives(keep, float_key(s), i, w)) continue;
      c += w;
      if (target < c) { pick = i; break; }
    }
    out[row] = pick;
  }
  cluster_sync();          // nobody leaves while another block may still read its shared memory
#undef GATHER_HISTOGRAMS
#undef SHIFTED
}

// Shared memory of a block's slice, and the most of it that fits an SM beside the histograms' 35 KB.
#define SMP_SLICE_MOST (190 * 1024)
static size_t slice_bytes(int vocab, int parts) { return ((size_t)slice_at((vocab + parts - 1) / parts) + 1) * sizeof(float); }

// Clusters of `parts` blocks that run at once.  A block has an SM to itself (1,024 threads of 62 registers), and a
// cluster's blocks lie in one group of SMs: 148, 74, 33 and 15 clusters of 1, 2, 4 and 8 on a whole B200.
static int resident_clusters(int parts) {
  static std::atomic<int> known[16][4];
  int device = 0, slot = parts == 1 ? 0 : parts == 2 ? 1 : parts == 4 ? 2 : 3;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 16) return 148 / parts;
  int count = known[device][slot].load(std::memory_order_relaxed);
  if (count > 0) return count;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(parts, 1);
  config.blockDim = dim3(SMP_THREADS);
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = parts;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&count, sample_kernel, &config) != cudaSuccess || count < 1) {
    cudaGetLastError();
    count = 148 / parts;
  }
  known[device][slot].store(count, std::memory_order_relaxed);
  return count;
}

// How many blocks share a row: the number for which the rounds of clusters that run at once, times what a
// block's slice takes, is least.  The times are those of the passes over the row (no top-k, or one past 512): a slice takes 30 us and
// 1.4 us per 1,000 logits where it is kept in shared memory, 45 and 1.85 where every pass reads it again, from L2 (3.3 where the
// rows at hand do not fit there); top-k 50 and top-p 0.95 by passes.  Measured so, 1 / 2 / 4 / 8 blocks a row, us: 8 rows of
// 151,936 330 / 187 / 88 / 64, 16 rows 326 / 187 / 86 / 122, 40 rows 327 / 186 / 168 / 185, 64 rows 328 / 188 /
// 172 / 302, 128 rows 333 / 368 / 336 / 544; 40 rows of 32,000 70 / 51 / 76 / 118, 256 rows 135 / 191 / 300 / 663; 64 rows
// of 300,000 611 / 337 / 372 / 436, 128 rows 1047 / 715 / 757 / 815.  A top-k of up to 512, decided among the largest logits, has its
// least time at the same number or within 2 us of it: 1 row of 151,936 351 / 200 / 36 / 34, 8 rows 368 / 221 / 56 / 52, 16 rows 366 / 206 /
// 36 / 52, 40 rows 366 / 206 / 58 / 73, 64 rows 368 / 212 / 69 / 110, 128 rows 394 / 409 / 124 / 190; of 32,000 1 row 32 / 28 / 26 / 28,
// 16 rows 32 / 28 / 28 / 42, 40 rows 32 / 28 / 40 / 58, 64 rows 32 / 28 / 48 / 83, 256 rows 58 / 97 / 149 / 276 (one and two blocks keep no
// slice of 151,936 in shared memory and take the passes).
static int sample_parts(int rows, int vocab) {
  int best = 1;
  double least = 0.0;
  for (int parts = 1; parts <= 8 && (parts == 1 || vocab >= parts * 4096); parts *= 2) {
    const int resident = resident_clusters(parts), rounds = (rows + resident - 1) / resident;
    const double slice = (double)((vocab + parts - 1) / parts);
    const bool in_l2 = (double)(rows < resident ? rows : resident) * vocab * 4.0 < 110e6;
    const double time = rounds * (slice_bytes(vocab, parts) <= SMP_SLICE_MOST ? 30.0 + 1.4e-3 * slice
                                                                              : 45.0 + (in_l2 ? 1.85e-3 : 3.3e-3) * slice);
    if (parts == 1 || time < least) best = parts, least = time;
  }
  return best;
}

// What the rule above decides, for its test.
FE_EXPORT int fe_sample_parts(int rows, int vocab) { return sample_parts(rows, vocab); }

static int launch_sample(const float* logits, int rows, int vocab, const SampleParams& params, bool drawn, int* out, int* status,
                         cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0) return FE_ERR_BAD_SHAPE;
  if (rows > 65535) return FE_ERR_TOO_LARGE;
  // A row's vocabulary over up to 8 blocks (one cluster) of at least 4,096 logits each.
  int parts = 1;
  size_t smem = 0;
  if (!drawn) {
    while (parts < 8 && rows * parts * 2 <= 296 && vocab >= parts * 2 * 4096) parts *= 2;
  } else {
    parts = sample_parts(rows, vocab);
    if (slice_bytes(vocab, parts) <= SMP_SLICE_MOST) smem = slice_bytes(vocab, parts);
  }
  if (smem > 0) {
    const cudaError_t set = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (set != cudaSuccess) return (int)set;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(parts, rows);
  config.blockDim = dim3(SMP_THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = parts;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = parts > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&config, sample_kernel, logits, vocab, params, out, status, smem > 0 ? 1 : 0);
  if (e != cudaSuccess) return (int)e;
  return fe_last_error();
}

FE_EXPORT int fe_sample(const float* logits, int rows, int vocab, const float* temperature,
                        const int* top_k, const float* top_p, const float* min_p,
                        const unsigned long long* seeds, const unsigned long long* counters,
                        int* out, int* status, cudaStream_t stream) {
  SampleParams params{temperature, top_k, top_p, min_p, seeds, counters, 0, {}};
  return launch_sample(logits, rows, vocab, params, temperature != nullptr, out, status, stream);
}

// The same with the rows' parameters in host memory, SampleRow after SampleRow; at most SMP_ROWS_BY_VALUE of them.
FE_EXPORT int fe_sample_rows(const float* logits, int rows, int vocab, const SampleRow* wishes, int* out, int* status, cudaStream_t stream) {
  if (rows > SMP_ROWS_BY_VALUE) return FE_ERR_TOO_LARGE;
  SampleParams params{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 1, {}};
  for (int r = 0; r < rows; ++r) params.rows[r] = wishes[r];
  return launch_sample(logits, rows, vocab, params, true, out, status, stream);
}

// Host copy of the uniform, for the Python twin's self-check.
FE_EXPORT float fe_uniform_host(unsigned long long seed, unsigned long long counter) {
  return fe_uniform(seed, counter);
}

// 32-bit products of deep rows on the 5th-generation tensor cores (part of gemm_simt.cu).
//
// Every operand is split into three bfloat16 numbers on its way to shared memory: x = a + b + c, each rounded to
// nearest of what the ones before left, so that nothing of the 24 bits of a number from 2^-110 on is lost (of smaller ones
// what lies below 2^-133, where bfloat16 ends).  x y is taken as
// (ab + ba + bb + ac + ca) + aa; the three products left out are 2^-25 of x y and below.  The products of 64 k are
// summed in tensor memory, the small ones first; what a stretch of 64 gives is added to the 32-bit sum outside, rounded
// to nearest, because the tensor core cuts off what falls below the 24 bits of its sum.  Of the eight parts of k
// (stretches s * 8 / stretches) each has a sum of its own, and the parts' sums are added in order: so blocks of a cluster can take
// a part each, and a row's bits depend neither on how many rows the call has, nor on the tile, nor on the blocks a
// tile is cut into.
//
//   block:          128 rows of w x NT rows of x.  16 warps (8 with up to 32 rows) read 64 k of both operands into registers a
//                   stretch ahead, split them into the three planes of a stage (128-byte swizzle) and, while the tensor
//                   cores work on it, add up what they left of the stretch before; one warp issues the 24 tcgen05.mma
//                   of a stretch.
//   tensor memory:  an accumulator of NT columns for every stage, and the sum of the parts behind.
//
// What bounds it: with 128 rows of x the instructions that split (a stretch takes 3,100 cycles, of which its products need
// 1,536); with 16 a stretch's chain of load, split, 24 products of 35 cycles each to issue, and sum (2,200 cycles).
// 500 x 4,096 x 1,024 takes 43 us, 500 x 1,024 x 3,072 36 (multiply-adds: 118 and 111).  Relative error against 64 bits, random normal
// operands, depth 256 / 1,024 / 3,072: 0.9e-7, 1.0e-7 and 1.1e-7 (of it along the result -0.6e-7); one chain of 32-bit
// multiply-adds 2.9e-7, 5.7e-7 and 9.9e-7.
//
// A sum that is not finite, or not zero and below 2^-70, is taken again as one chain of multiply-adds: so infinities, numbers
// that round to infinity and rows of numbers that bfloat16 does not hold give what they give there.  (Numbers about 2^-118 are
// off by 9e-6 of themselves in three parts, about 2^-126 by 2e-3.  What they lose moves a sum from 2^-70 on by less than 2^-24 of
// it while the other operand's numbers add up to less than 2^40; where all numbers are below 2^-134 the sum is zero.)
// A warp takes the chains of eight rows of x together.  1,024 x 32,000 x 1,024: 0.54 ms finite, 0.65 with a NaN in one row, 0.80 in
// one column, 8.2 in every row (every lane its own chains, one after the other: 0.66, 1.5 and 124; multiply-adds alone 1.44).
#pragma once
#include "tcgen05.cuh"

#define GST_K 64
#define GST_PARTS 8
#define GST_L2 2             // stretches of w asked for ahead
#define GST_MIN_K 256        // depth from which on 32-bit operands go this way
#define GST_SMALL 8.4703295e-22f     // 2^-70

namespace {

__device__ __forceinline__ void gst_split(float x, float y, unsigned& a, unsigned& b, unsigned& c) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(a) : "f"(y), "f"(x));
  x -= __uint_as_float(a << 16), y -= __uint_as_float(a & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b) : "f"(y), "f"(x));
  x -= __uint_as_float(b << 16), y -= __uint_as_float(b & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(c) : "f"(y), "f"(x));
}

// Sixteen bytes, in the order of the program: x is written by the kernel before this one, and a load that may move could
// pass the wait for it.
__device__ __forceinline__ float4 gst_load(const char* from) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(from) : "memory");
  return v;
}

// One operand's rows of a block: thread t has four k, piece t % 16, of rows t / 16, t / 16 + WORKERS / 16, ...; a stretch is on its way
// in registers.  Rows that do not exist are the last one again: what they give is not stored.
template <int ROWS, int WORKERS>
struct SplitRows {
  static constexpr int STEP = WORKERS / 16, PIECES = (ROWS + STEP - 1) / STEP;
  unsigned from[PIECES];   // bytes from the operand's first row
  unsigned at;             // of the first piece in a plane
  float4 raw[PIECES];
  __device__ __forceinline__ void begin(long long ld, int rows) {
    const int row = threadIdx.x >> 4, piece = threadIdx.x & 15;
#pragma unroll
    for (int j = 0; j < PIECES; ++j) from[j] = (unsigned)(min(row + STEP * j, rows - 1) * ld + piece * 4) * 4u;
    at = (unsigned)(row * 128 + (((piece >> 1) ^ (row & 7)) << 4) + (piece & 1) * 8);
  }
  // Stretch of 64 k at `base` (the operand's first row from that k on), `left` of them in the row: pieces behind its end
  // read the last one (no branch round a load: registers that two places load are waited for where the places meet).
  __device__ __forceinline__ void load(const float* base, int left) {
    const int piece = (int)(threadIdx.x & 15) * 4;
    const char* src = reinterpret_cast<const char*>(base) + (long long)min(0, left - 4 - piece) * 4;
#pragma unroll
    for (int j = 0; j < PIECES; ++j) raw[j] = gst_load(src + from[j]);
  }
  // The planes at `planes`, from what is held; `left` as it was loaded with.
  __device__ __forceinline__ void put(unsigned char* planes, int left) {
    if (left < GST_K && (int)(threadIdx.x & 15) * 4 >= left) {
#pragma unroll
      for (int j = 0; j < PIECES; ++j) raw[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
      if (ROWS % STEP != 0 && (int)(threadIdx.x >> 4) + STEP * j >= ROWS) break;
      unsigned a[2], b[2], c[2];
      gst_split(raw[j].x, raw[j].y, a[0], b[0], c[0]);
      gst_split(raw[j].z, raw[j].w, a[1], b[1], c[1]);
      unsigned char* to = planes + at + j * (STEP * 128);
      *reinterpret_cast<uint2*>(to) = make_uint2(a[0], a[1]);
      *reinterpret_cast<uint2*>(to + ROWS * 128) = make_uint2(b[0], b[1]);
      *reinterpret_cast<uint2*>(to + 2 * ROWS * 128) = make_uint2(c[0], c[1]);
    }
  }
};

// Eight columns of this thread's row of tensor memory.
__device__ __forceinline__ void gst_tmem_load(unsigned taddr, float (&v)[8]) {
  unsigned r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void gst_tmem_store8(unsigned taddr, const float* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
               "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
}

// The chains of multiply-adds that take the place of sums (bits of `which`): N rows of x, `step` apart from
// `row` on (the last one again where the product has no more), with this lane's row of w.  A warp takes them together: a row of w
// is then read once for N chains, and they fill one another's waits.
template <int N>
__device__ __noinline__ void gst_chains(const Product& p, int row, int step, int col, unsigned which) {
  const float* x = (const float*)p.x + (size_t)blockIdx.z * p.batch_x;
  const float* w = (const float*)p.w + (size_t)blockIdx.z * p.batch_w + (size_t)min(col, p.o - 1) * p.k;
  float sum[N];
#pragma unroll
  for (int j = 0; j < N; ++j) sum[j] = 0.f;
  for (int i = 0; i < p.k; i += 4) {
    const float4 b = *reinterpret_cast<const float4*>(w + i);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float4 a = *reinterpret_cast<const float4*>(x + (size_t)min(row + j * step, p.n - 1) * p.ldx + i);
      sum[j] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum[j]))));
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (which >> j & 1u) gs_store(p, sum[j], row + j * step, col);
}

// Stores a sum, or says that it has to be taken again.
__device__ __forceinline__ unsigned gst_finish(const Product& p, float v, int row, int col, bool ok) {
  if (row >= p.n || col >= p.o) return 0u;
  if (ok && !(v == 0.f || (fabsf(v) >= GST_SMALL && isfinite(v)))) return 1u;
  gs_store(p, ok ? v : __int_as_float(0x7fffffff), row, col);
  return 0u;
}

__host__ __device__ constexpr int gst_stage_bytes(int nt) { return 3 * (128 + nt) * 128; }
// Threads that read, split and add up: with few rows of x half as many, so that (up to 16 rows: 110 KB a block) two blocks share an SM.
__host__ __device__ constexpr int gst_workers(int nt) { return nt <= 32 ? 256 : 512; }
__host__ __device__ constexpr int gst_stages(int nt) { return nt == 64 ? 3 : 2; }
__host__ __device__ constexpr int gst_smem(int nt) { return gst_stages(nt) * gst_stage_bytes(nt) + 1024 + 128; }
// an accumulator a stage and the parts' sum, a power of two
__host__ __device__ constexpr int gst_tmem_cols(int nt) { return 4 * nt; }

// By a whole warp, the lane with `leads` issues: the operands of the instruction then lie in uniform registers (issued
// from a branch of one lane each product takes about 90 cycles to issue, 45 of them moves).
template <bool FIRST>
__device__ __forceinline__ void gst_mma(unsigned acc, uint64_t a, uint64_t b, unsigned idesc, unsigned leads) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 q, %4, 0;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(acc), "l"(a), "l"(b), "r"(idesc), "r"(leads), "n"(FIRST ? 0 : 1) : "memory");
}
// The 24 products of a stretch: 64 k of both operands' planes at `stage` into the columns at `acc`.
template <int NT>
__device__ __forceinline__ void gst_multiply(const unsigned char* stage, unsigned acc, uint64_t* done, unsigned leads) {
  const unsigned idesc = tc5::umma_idesc(NT);
  uint64_t a[3], b[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    a[q] = tc5::umma_desc(stage + q * (128 * 128));
    b[q] = tc5::umma_desc(stage + 3 * (128 * 128) + q * (NT * 128));
  }
  // 16 k are 32 bytes further along the swizzled row: 2 in units of 16 bytes
#pragma unroll
  for (int kk = 0; kk < 8; kk += 2) {
    if (kk == 0) gst_mma<true>(acc, a[2], b[0], idesc, leads);
    else gst_mma<false>(acc, a[2] + kk, b[0] + kk, idesc, leads);
    gst_mma<false>(acc, a[0] + kk, b[2] + kk, idesc, leads);
    gst_mma<false>(acc, a[1] + kk, b[1] + kk, idesc, leads);
    gst_mma<false>(acc, a[1] + kk, b[0] + kk, idesc, leads);
    gst_mma<false>(acc, a[0] + kk, b[1] + kk, idesc, leads);
  }
#pragma unroll
  for (int kk = 0; kk < 8; kk += 2) gst_mma<false>(acc, a[0] + kk, b[0] + kk, idesc, leads);
  if (leads) tc5::umma_commit(done);
  __syncwarp();
}

template <int NT>
__global__ void __launch_bounds__(gst_workers(NT) + 32, NT <= 16 ? 2 : 1) gemm_split_kernel(const __grid_constant__ Product p, int cuts, int ahead, const Fault fault) {
  constexpr int WORKERS = gst_workers(NT);
  constexpr int COLS = NT * 128 / WORKERS, STEP = 8;          // columns of a thread, and of a piece of them
  constexpr int STAGES = gst_stages(NT);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * gst_stage_bytes(NT));   // [STAGES] the planes of a stage are written
  uint64_t* done = full + STAGES;                                                       // [STAGES] its products are summed
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(done + STAGES);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % cuts, col0 = (blockIdx.x / cuts) * 128, row0 = blockIdx.y * NT;
  const int stretches = (p.k + GST_K - 1) / GST_K;
  // parts first .. last - 1 and their stretches
  const int first = rank * (GST_PARTS / cuts), last = first + GST_PARTS / cuts;
  const int s_begin = (int)((long long)stretches * first / GST_PARTS), s_end = (int)((long long)stretches * last / GST_PARTS);
  const int count = s_end - s_begin;
  const float* w = (const float*)p.w + (size_t)blockIdx.z * p.batch_w + (size_t)col0 * p.k;
  const float* x = (const float*)p.x + (size_t)blockIdx.z * p.batch_x + (size_t)row0 * p.ldx;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) tc5::mbar_init(&full[s], WORKERS / 32), tc5::mbar_init(&done[s], 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc5::smem_u32(tmem_slot)),
                 "r"(gst_tmem_cols(NT)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // With `ahead` w is not the result of an earlier kernel that may still run, and does not wait for it: the first stages of w are
  // split, and L2 is asked for the first stretches (a row each thread.  2 stretches: 4 x 32,000 x 1,024 55 us, 8 58, all 61, none 57).
  if (ahead && blockIdx.y == 0 && threadIdx.x < 128 && col0 + (int)threadIdx.x < p.o && count > 0) {
    const int k_begin = s_begin * GST_K, bytes = (min(p.k, min(s_end, s_begin + GST_L2) * GST_K) - k_begin) * 4;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + (size_t)threadIdx.x * p.k + k_begin), "r"(bytes) : "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;
  pdl_trigger();         // after the allocation: a block of the next kernel that held the columns would wait for this one's end
  if (!ahead) pdl_wait();

  bool ok = true;
  unsigned again = 0u;       // sums of this thread that are taken again, at the end
  if (warp == WORKERS / 32) {
    unsigned leads;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leads));
    int s = 0, issued = 0;
    unsigned phase = 0;
    for (int i = 0; i < count; ++i) {
      const bool here = tc5::mbar_wait(&full[s], phase, abort_flag, fault.wait_limit);
      if (!__all_sync(0xffffffffu, here)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      gst_multiply<NT>(smem + s * gst_stage_bytes(NT), tmem + s * NT, &done[s], leads);
      issued = i + 1;
      if (++s == STAGES) s = 0, phase ^= 1u;
    }
    // nothing may be in flight when the tensor memory is given back, also after a wait that ran out
    if (issued > 0) {
      int ended = 0;
      for (unsigned t = 0; t < tc5::WAIT_LIMIT && !ended; ++t) ended = tc5::mbar_try_wait(&done[(issued - 1) % STAGES], ((issued - 1) / STAGES) & 1);
    }
    __syncwarp();
    if (ahead) pdl_wait();
  } else {
    const int quarter = warp & 3, column = (warp >> 2) * COLS;
    const unsigned mine = tmem + ((unsigned)(quarter * 32) << 16) + column;
    SplitRows<128, WORKERS> a;
    SplitRows<NT, WORKERS> b;
    a.begin(p.k, min(128, p.o - col0));
    b.begin(p.ldx, min(NT, p.n - row0));
    float acc[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
    const int split_ahead = ahead ? min(count, STAGES) : 0;
    // stretch i of this block's, and past the last one that again
    auto k_of = [&](int i) { return (s_begin + min(i, count - 1)) * GST_K; };
    if (count > 0) a.load(w + k_of(0), p.k - k_of(0));
    for (int i = 0; i < split_ahead; ++i) {
      a.put(smem + i * gst_stage_bytes(NT), p.k - k_of(i));
      a.load(w + k_of(i + 1), p.k - k_of(i + 1));
    }
    if (ahead) pdl_wait();
    if (count > 0) b.load(x + k_of(0), p.k - k_of(0));
    // The lanes of a warp part where a row ends, where a value is not finite and where one of them speaks for all; what the whole
    // warp executes together (tensor memory, cluster barriers) stands behind a __syncwarp or a vote.
    __syncwarp();
    int part = first, part_end = (int)((long long)stretches * (first + 1) / GST_PARTS);
    // the sum of the parts before `part` lies behind the accumulators (with two blocks' parts and more: the part before)
    auto close_parts = [&](int stretch) {
      while (part < last - 1 && stretch == part_end) {
#pragma unroll
        for (int c = 0; c < COLS; c += STEP) {
          if (part > first) {
            float sum[STEP];
            gst_tmem_load(mine + STAGES * NT + c, sum);
#pragma unroll
            for (int e = 0; e < STEP; ++e) acc[c + e] = sum[e] + acc[c + e];
          }
        }
#pragma unroll
        for (int c = 0; c < COLS; c += 8) gst_tmem_store8(mine + STAGES * NT + c, acc + c);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
        ++part;
        part_end = (int)((long long)stretches * (part + 1) / GST_PARTS);
      }
    };
    close_parts(s_begin);
    auto hand_over = [&](int i, int s) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();        // one arrival a warp
      if (lane == 0 && (fault.skip_stretch < 0 || (s_begin + i) / 2 != fault.skip_stretch)) gs_arrive(&full[s]);
    };
    for (int i = 0; i < split_ahead; ++i) {
      b.put(smem + i * gst_stage_bytes(NT) + 3 * 128 * 128, p.k - k_of(i));
      b.load(x + k_of(i + 1), p.k - k_of(i + 1));
      hand_over(i, i);
    }
    int s = split_ahead % STAGES;
    for (int i = split_ahead; i < count + STAGES; ++i) {
      if (i >= STAGES) {
        // the products of stretch i - STAGES are summed: its stage is free, and so is its accumulator once it is read
        ok = tc5::mbar_wait(&done[s], (i / STAGES + 1) & 1, abort_flag, fault.wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < COLS; c += STEP) {
          float v[STEP];
          gst_tmem_load(mine + s * NT + c, v);
#pragma unroll
          for (int e = 0; e < STEP; ++e) acc[c + e] += v[e];
        }
        close_parts(s_begin + i - STAGES + 1);
      }
      if (i < count) {
        unsigned char* stage = smem + s * gst_stage_bytes(NT);
        a.put(stage, p.k - k_of(i));
        a.load(w + k_of(i + 1), p.k - k_of(i + 1));
        b.put(stage + 3 * 128 * 128, p.k - k_of(i));
        b.load(x + k_of(i + 1), p.k - k_of(i + 1));
        hand_over(i, s);
      }
      if (++s == STAGES) s = 0;
    }
    if (!ok && lane == 0 && p.status) atomicOr(p.status, FE_STATUS_WAIT_TIMEOUT);
    __syncwarp();
    if (cuts == 1) {
      const int col = col0 + quarter * 32 + lane;
#pragma unroll
      for (int c = 0; c < COLS; c += 8) {
        float sum[8];
        __syncwarp();        // lanes past the last column have left the stores
        gst_tmem_load(mine + STAGES * NT + c, sum);
#pragma unroll
        for (int e = 0; e < 8; ++e) again |= gst_finish(p, sum[e] + acc[c + e], row0 + column + c + e, col, ok) << (c + e);
      }
    } else {
      // the parts of this block, [part][row of x][row of w], over the stages that nobody reads any more
      float* stash = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
#pragma unroll
      for (int c = 0; c < COLS; c += 8) {
        if (last - first > 1) {
          float before[8];
          gst_tmem_load(mine + STAGES * NT + c, before);
#pragma unroll
          for (int e = 0; e < 8; ++e) stash[(column + c + e) * 128] = before[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) stash[((last - first - 1) * NT + column + c + e) * 128] = acc[c + e];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (cuts > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int per = GST_PARTS / cuts, share = NT / cuts;
    bool all_ok = true;
    unsigned stash[GST_PARTS];
    for (int r = 0; r < cuts; ++r) {
      unsigned flag, value;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(flag) : "r"(tc5::smem_u32(abort_flag)), "r"(r));
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(value) : "r"(flag) : "memory");
      all_ok = all_ok && value == 0;
    }
#pragma unroll
    for (int q = 0; q < GST_PARTS; ++q) {
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(stash[q]) : "r"(tc5::smem_u32(smem)), "r"(q / per));
      stash[q] += (unsigned)((q % per) * NT * 512);
    }
    if (warp < WORKERS / 32) {
      for (int at = threadIdx.x, j = 0; at < share * 128; at += WORKERS, ++j) {
        const int token = rank * share + (at >> 7), feature = at & 127;
        float v[GST_PARTS];
#pragma unroll
        for (int q = 0; q < GST_PARTS; ++q)
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[q]) : "r"(stash[q] + (unsigned)((token * 128 + feature) * 4)) : "memory");
#pragma unroll
        for (int q = 1; q < GST_PARTS; ++q) v[0] += v[q];
        again |= gst_finish(p, v[0], row0 + token, col0 + feature, all_ok) << j;
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // the stashes stay until they are read
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  if (warp == WORKERS / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(gst_tmem_cols(NT)));
  } else if (__any_sync(0xffffffffu, again != 0u)) {
    // Here, where no register is needed for anything else (called from among the stores: 1,024 x 32,000 x 1,024 651 us instead of
    // 533 with finite sums).  A thread's sums are neighbouring columns of its piece, or every STRIDE-th row of the block's share.
    constexpr int AT_ONCE = 8, STRIDE = WORKERS / 128;
    const bool whole = cuts == 1;
    const int row = row0 + (whole ? (warp >> 2) * COLS : rank * (NT / cuts) + (int)(threadIdx.x >> 7)), step = whole ? 1 : STRIDE;
    for (int j = 0; j < COLS; j += AT_ONCE) {
      const unsigned which = again >> j & ((1u << AT_ONCE) - 1u);
      if (__any_sync(0xffffffffu, which != 0u)) gst_chains<AT_ONCE>(p, row + j * step, step, col0 + (int)(threadIdx.x & 127), which);
    }
  }
}

}  // namespace

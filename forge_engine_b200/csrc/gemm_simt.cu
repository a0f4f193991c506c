// y[n, o] = sum_k x[n, k] * w[o, k] (+ bias[o]) (+ y[n, o])   -- in 32 bits.
//
// This is the matrix product of the true 32-bit path and of any tensor whose
// checkpoint dtype is float32.  Both operands are K-major, like nn.Linear's
// [out, in] weight (src/forge_engine/qwen3.py:113-122).  Deep products of 32-bit operands go to the tensor
// cores (gemm_split.cuh); for the others each output element is summed over k in ascending order by one
// thread, in both kernels below.  Which of the two does not depend on the number of rows, so a row's result
// does not depend on how many other rows are in the call, nor on the tile.
// (A row's bits do depend on which of the two it is: from 256 numbers on, where both operands are 32 bits and lie on 16 bytes,
// rows and strides too and below 2^22 numbers, the tensor cores; a layer's products are all of one kind.)
//
// Tiles of both operands lie in shared memory as they lie in memory, rows of k with 16 bytes
// of padding, so that a 16-byte read of 4 k by eight neighbouring rows touches every bank once.
// What bounds the products is the 128 bytes a cycle that shared memory delivers to registers
// (an operand read by several lanes at once counts for each of them): a thread's tile of
// TM x TN outputs reads TM + TN numbers for TM TN multiply-adds.
#include "tcgen05.cuh"

#include <algorithm>

namespace {

__device__ __forceinline__ void gs_copy16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc5::smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void gs_copy4(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc5::smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void gs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void gs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }
// The barrier counts this thread once all its copies so far have landed.
__device__ __forceinline__ void gs_arrive_copied(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc5::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void gs_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc5::smem_u32(bar)) : "memory");
}

struct Product {
  const void* x;
  const void* w;
  const float* bias;
  void* y;
  int y_dtype, n, o, k, accumulate;
  int* status;           // null: none
  long long ldx, ldy, batch_x, batch_w, batch_y;   // blockIdx.z: one product of a batch (a head)
};

__device__ __forceinline__ void gs_store(const Product& p, float v, int r, int c) {
  if (p.bias) v += p.bias[c];
  const size_t at = (size_t)blockIdx.z * p.batch_y + (size_t)r * p.ldy + c;
  if (p.y_dtype == FE_DTYPE_F32) {
    float* dst = (float*)p.y + at;
    *dst = p.accumulate ? v + *dst : v;
  } else {
    bf16* dst = (bf16*)p.y + at;
    *dst = from_float<bf16>(p.accumulate ? v + to_float(*dst) : v);
  }
}

// Usually tc5::WAIT_LIMIT and no stretch; see fe_gemm_simt_set_test_fault.
struct Fault {
  unsigned wait_limit;
  int skip_stretch;
};
Fault g_test_fault{tc5::WAIT_LIMIT, -1};

}  // namespace

#include "gemm_split.cuh"

namespace {

// Many rows: TY x TX threads keep TM x TN outputs each; thread (ty, tx) the rows ty + TY i and the
// columns tx + TX j of the block's tile.
#define GS_BK 32
#define GS_STAGES 3
#define GS_PITCH (GS_BK + 4)

// What a thread copies of one operand's stages: rows row, row + STEP, ... of ROWS, one piece of each; zeros
// stand where a row or a k does not exist.  A piece is 16 bytes with VEC: rows start on 16-byte boundaries and
// k is a multiple of 16 bytes.  Otherwise it is one number, a warp's 32 of them neighbours.  Tiles hold 32-bit
// numbers: 32-bit operands go there by cp.async, bfloat16 ones through registers, asked for a stage earlier (read
// from shared memory as they were, they would be widened once per output: 500 x 1,024 x 3,072 with
// bfloat16 rows, weights or both 213, 220 and 240 us, 187, 184 and 208 this way).
template <typename T, int ROWS, int THREADS, bool VEC>
struct Stager {
  static constexpr bool HELD = sizeof(T) == 2;
  static constexpr int CH = VEC ? 16 / (int)sizeof(T) : 1, PER_ROW = GS_BK / CH;
  static constexpr int STEP = THREADS / PER_ROW, COPIES = (ROWS + STEP - 1) / STEP;
  const T* base;         // something to point at where nothing is read
  const T* src;
  long long step;
  int kk, rows;          // rows of this thread's that exist
  float* dst;
  uint4 held[HELD && VEC ? COPIES : 1];
  T one[HELD && !VEC ? COPIES : 1];
  __device__ __forceinline__ Stager(float* tile, const T* from, long long ld, int row0, int limit) : base(from) {
    const int row = threadIdx.x / PER_ROW;
    kk = (threadIdx.x % PER_ROW) * CH;
    src = base + (size_t)min(row0 + row, limit - 1) * ld + kk;
    step = STEP * ld;
    const int have = min(limit - row0, ROWS) - row;
    rows = have <= 0 ? 0 : (have + STEP - 1) / STEP;
    dst = tile + row * GS_PITCH + kk;
  }
  // 32-bit operands: stage `stage` is on its way.  bfloat16 ones: held for put().
  __device__ __forceinline__ void get(int stage, int k0, int k) {
    float* to = dst + stage * (ROWS * GS_PITCH);
    const T* from = src + k0;
#pragma unroll
    for (int u = 0; u < COPIES; ++u) {
      if (ROWS % STEP == 0 || (int)threadIdx.x / PER_ROW + u * STEP < ROWS) {
        const bool valid = u < rows && k0 + kk < k;
        if constexpr (HELD && VEC) held[u] = valid ? *reinterpret_cast<const uint4*>(from) : make_uint4(0u, 0u, 0u, 0u);
        else if constexpr (HELD) one[u] = valid ? *from : from_float<T>(0.f);
        else if constexpr (VEC) gs_copy16(to + u * STEP * GS_PITCH, valid ? from : base, valid);
        else gs_copy4(to + u * STEP * GS_PITCH, valid ? from : base, valid);
      }
      from += step;
    }
  }
  __device__ __forceinline__ void put(int stage) const {
    if constexpr (HELD) {
      float* to = dst + stage * (ROWS * GS_PITCH);
#pragma unroll
      for (int u = 0; u < COPIES; ++u) {
        if (ROWS % STEP == 0 || (int)threadIdx.x / PER_ROW + u * STEP < ROWS) {
          if constexpr (VEC) {
            const unsigned w[4] = {held[u].x, held[u].y, held[u].z, held[u].w};
#pragma unroll
            for (int e = 0; e < 2; ++e)
              *reinterpret_cast<float4*>(to + u * STEP * GS_PITCH + 4 * e) =
                  make_float4(__uint_as_float(w[2 * e] << 16), __uint_as_float(w[2 * e] & 0xffff0000u),
                              __uint_as_float(w[2 * e + 1] << 16), __uint_as_float(w[2 * e + 1] & 0xffff0000u));
          } else {
            to[u * STEP * GS_PITCH] = to_float(one[u]);
          }
        }
      }
    }
  }
};

template <typename TX_, typename TW_, int TM, int TN, int TY, int TX, bool VEC>
__global__ void __launch_bounds__(TY * TX) gemm_simt_tile_kernel(const Product p) {
  constexpr int BM = TM * TY, BN = TN * TX, THREADS = TY * TX;
  constexpr int PX = GS_PITCH, PW = GS_PITCH;
  extern __shared__ __align__(16) unsigned char smem[];
  float* xs = (float*)smem;
  float* ws = xs + GS_STAGES * BM * PX;
  pdl_trigger();
  pdl_wait();
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
  Stager<TX_, BM, THREADS, VEC> x_in(xs, (const TX_*)p.x + (size_t)blockIdx.z * p.batch_x, p.ldx, row0, p.n);
  Stager<TW_, BN, THREADS, VEC> w_in(ws, (const TW_*)p.w + (size_t)blockIdx.z * p.batch_w, p.k, col0, p.o);
  const int ty = threadIdx.x / TX, tx = threadIdx.x % TX;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  const int steps = (p.k + GS_BK - 1) / GS_BK;
#pragma unroll
  for (int s = 0; s < GS_STAGES - 1; ++s) {
    if (s < steps) {
      x_in.get(s, s * GS_BK, p.k);
      w_in.get(s, s * GS_BK, p.k);
      if (s == 0) x_in.put(0), w_in.put(0);
    }
    gs_commit();
  }
  int stage = 0;
  for (int step = 0; step < steps; ++step) {
    gs_wait<GS_STAGES - 2>();
    __syncthreads();
    const int next = step + GS_STAGES - 1, after = stage + 1 == GS_STAGES ? 0 : stage + 1;
    if (step + 1 < steps) x_in.put(after), w_in.put(after);       // what is held of the stage after this one
    if (next < steps) {
      const int to = stage == 0 ? GS_STAGES - 1 : stage - 1;
      x_in.get(to, next * GS_BK, p.k);
      w_in.get(to, next * GS_BK, p.k);
    }
    gs_commit();
    const float* xt = xs + stage * BM * PX + ty * PX;
    const float* wt = ws + stage * BN * PW + tx * PW;
    float a[2][TM][4], b[2][TN][4];          // the next four k are read while these four are summed
#pragma unroll
    for (int i = 0; i < TM; ++i) load4(xt + i * TY * PX, a[0][i]);
#pragma unroll
    for (int j = 0; j < TN; ++j) load4(wt + j * TX * PW, b[0][j]);
#pragma unroll
    for (int u = 0; u < GS_BK / 4; ++u) {
      if (u + 1 < GS_BK / 4) {
#pragma unroll
        for (int i = 0; i < TM; ++i) load4(xt + i * TY * PX + 4 * (u + 1), a[(u + 1) & 1][i]);
#pragma unroll
        for (int j = 0; j < TN; ++j) load4(wt + j * TX * PW + 4 * (u + 1), b[(u + 1) & 1][j]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[u & 1][i][e], b[u & 1][j][e], acc[i][j]);
    }
    stage = after;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = row0 + ty + TY * i;
    if (r >= p.n) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int c = col0 + tx + TX * j;
      if (c < p.o) gs_store(p, acc[i][j], r, c);
    }
  }
}

// Few rows (decoding): a block streams COLS rows of w through a ring that four warps fill; the lanes of
// the other warps lie over LC columns and 32 / LC groups of R rows.  Bound by the stream of w, by what
// shared memory delivers, and by the chain of k dependent additions per output (4 cycles each).
#define GSK_KT 128
#define GSK_MAX_STAGES 8
#define GSK_LOADERS 4
template <typename TX, typename TW, int COLS, int LC, int R>
__global__ void __launch_bounds__(32 * (GSK_LOADERS + 8)) gemm_simt_rows_kernel(const Product p, int stages, const Fault fault) {
  constexpr int PX = GSK_KT + 16 / (int)sizeof(TX), PW = GSK_KT + 16 / (int)sizeof(TW);
  constexpr int ROWS = R * (32 / LC);           // rows of x a warp takes
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[GSK_MAX_STAGES], empty[GSK_MAX_STAGES];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, workers = (blockDim.x >> 5) - GSK_LOADERS;
  const int rows = (workers / (COLS / LC)) * ROWS;
  TW* ws = (TW*)smem;
  TX* xs = (TX*)(smem + (size_t)stages * COLS * PW * sizeof(TW));
  const int col0 = blockIdx.x * COLS;
  const int steps = (p.k + GSK_KT - 1) / GSK_KT;
  pdl_trigger();
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < stages; ++s) {
      tc5::mbar_init(&full[s], 32 * GSK_LOADERS);
      tc5::mbar_init(&empty[s], workers);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  if (warp >= workers) {
    // a thread copies one 16-byte piece of rows at, at + step, ...
    constexpr int CW = 16 / (int)sizeof(TW), CX = 16 / (int)sizeof(TX);
    constexpr int PW_ROW = GSK_KT / CW, PX_ROW = GSK_KT / CX;
    constexpr int SW = 32 * GSK_LOADERS / PW_ROW, SX = 32 * GSK_LOADERS / PX_ROW;
    const int id = (int)threadIdx.x - 32 * workers;
    const int wr = id / PW_ROW, wk = (id % PW_ROW) * CW, xr = id / PX_ROW, xk = (id % PX_ROW) * CX;
    const int cols = min(COLS, p.o - col0);
    const TW* w = (const TW*)p.w + (size_t)blockIdx.z * p.batch_w + (size_t)(col0 + min(wr, cols - 1)) * p.k + wk;
    const TX* x = (const TX*)p.x + (size_t)blockIdx.z * p.batch_x + (size_t)min(xr, p.n - 1) * p.ldx + xk;
    const long long w_step = (long long)SW * p.k, x_step = SX * p.ldx;
    int s = 0;
    unsigned phase = 1;
    for (int step = 0; step < steps; ++step) {
      const int k0 = step * GSK_KT;
      if (step >= stages) {
        int ok = 1;
        if (lane == 0) ok = tc5::mbar_wait(&empty[s], phase, &abort_flag, fault.wait_limit) ? 1 : 0;
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
      }
      const TW* from = w + k0;
      TW* to = ws + (s * COLS + wr) * PW + wk;
      const bool w_in = k0 + wk < p.k;
#pragma unroll
      for (int u = 0; u < (COLS + SW - 1) / SW; ++u) {
        if (w_in && wr + u * SW < cols) gs_copy16(to, from, true);
        from += w_step;
        to += SW * PW;
      }
      const TX* xfrom = x + k0;
      TX* xto = xs + (s * rows + xr) * PX + xk;
      if (k0 + xk < p.k)
        for (int r = xr; r < p.n; r += SX) {
          gs_copy16(xto, xfrom, true);
          xfrom += x_step;
          xto += SX * PX;
        }
      if (step != fault.skip_stretch) gs_arrive_copied(&full[s]);
      if (++s == stages) s = 0, phase ^= 1u;
    }
    gs_commit();
    gs_wait<0>();          // no copy is in flight when the block ends, also after a wait that ran out
  } else {
    const int lc = (warp % (COLS / LC)) * LC + lane % LC, mine = (warp / (COLS / LC)) * ROWS + (lane / LC) * R;
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.f;
    bool ok = true;
    int s = 0;
    unsigned phase = 0;
    for (int step = 0; step < steps; ++step) {
      const int kt = min(GSK_KT, p.k - step * GSK_KT);
      ok = tc5::mbar_wait(&full[s], phase, &abort_flag, fault.wait_limit);
      if (!ok) break;
      const TW* wt = ws + (s * COLS + lc) * PW;
      const TX* xt = xs + (s * rows + mine) * PX;
      if (kt == GSK_KT) {
        float a[2][R][8], b[2][8];            // the next eight k are read while these eight are summed
        load4(wt, b[0]), load4(wt + 4, b[0] + 4);
#pragma unroll
        for (int i = 0; i < R; ++i) load4(xt + i * PX, a[0][i]), load4(xt + i * PX + 4, a[0][i] + 4);
#pragma unroll
        for (int u = 0; u < GSK_KT / 8; ++u) {
          if (u + 1 < GSK_KT / 8) {
            load4(wt + 8 * (u + 1), b[(u + 1) & 1]), load4(wt + 8 * (u + 1) + 4, b[(u + 1) & 1] + 4);
#pragma unroll
            for (int i = 0; i < R; ++i)
              load4(xt + i * PX + 8 * (u + 1), a[(u + 1) & 1][i]), load4(xt + i * PX + 8 * (u + 1) + 4, a[(u + 1) & 1][i] + 4);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(a[u & 1][i][e], b[u & 1][e], acc[i]);
        }
      } else {
        for (int kk = 0; kk < kt; kk += 4) {
          float b[4];
          load4(wt + kk, b);
#pragma unroll
          for (int i = 0; i < R; ++i) {
            float a[4];
            load4(xt + i * PX + kk, a);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i] = fmaf(a[e], b[e], acc[i]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) gs_arrive(&empty[s]);
      if (++s == stages) s = 0, phase ^= 1u;
    }
    if (!ok && lane == 0 && p.status) atomicOr(p.status, FE_STATUS_WAIT_TIMEOUT);
    if (col0 + lc < p.o) {
      // after a wait that ran out the outputs are NaN
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (mine + i < p.n) gs_store(p, ok ? acc[i] : __int_as_float(0x7fffffff), mine + i, col0 + lc);
    }
  }
}

template <typename K, typename... A>
int launch_sized(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  if (smem > 48 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
  }
  return fe_launch_dependent(kernel, grid, dim3(threads), smem, stream, args...);
}

template <typename TX_, typename TW_, int TM, int TN, int TY, int TX, bool VEC>
int launch_tile(const Product& p, int batch, cudaStream_t stream) {
  constexpr int BM = TM * TY, BN = TN * TX;
  const size_t smem = (size_t)GS_STAGES * (BM + BN) * GS_PITCH * sizeof(float);
  dim3 grid((p.o + BN - 1) / BN, (p.n + BM - 1) / BM, batch);
  if (grid.y > 65535) return FE_ERR_TOO_LARGE;
  return launch_sized(gemm_simt_tile_kernel<TX_, TW_, TM, TN, TY, TX, VEC>, grid, TY * TX, smem, stream, p);
}

template <typename TX, typename TW, int COLS, int LC, int R>
int launch_rows(const Product& p, int batch, cudaStream_t stream) {
  constexpr int ROWS = R * (32 / LC);
  const int groups = (p.n + ROWS - 1) / ROWS, workers = groups * (COLS / LC);
  const size_t stage = COLS * (GSK_KT * sizeof(TW) + 16) + (size_t)groups * ROWS * (GSK_KT * sizeof(TX) + 16);
  const int stages = (int)std::min<size_t>(GSK_MAX_STAGES, std::max<size_t>(2, 110 * 1024 / stage));
  dim3 grid((p.o + COLS - 1) / COLS, 1, batch);
  return launch_sized(gemm_simt_rows_kernel<TX, TW, COLS, LC, R>, grid, 32 * (workers + GSK_LOADERS), stages * stage, stream, p, stages, g_test_fault);
}

template <int NT>
int launch_split(const Product& p, int batch, int cuts, bool ahead, cudaStream_t stream) {
  const dim3 grid((unsigned)((p.o + 127) / 128) * cuts, (p.n + NT - 1) / NT, batch);
  if (grid.y > 65535) return FE_ERR_TOO_LARGE;
  const cudaError_t err = cudaFuncSetAttribute(gemm_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, gst_smem(NT));
  if (err != cudaSuccess) return (int)err;
  return fe_launch_dependent_shaped(gemm_split_kernel<NT>, grid, dim3(gst_workers(NT) + 32), gst_smem(NT), stream, dim3(cuts, 1, 1), p, cuts,
                                    ahead ? 1 : 0, g_test_fault);
}

// Rows of x a block takes, and into how many blocks (a cluster) k is cut: the number for which the time below is least.
// Measured, us, w out of memory: by one block a tile 16 rows x 4,096 x 1,024 29, 1,024 x 2,048 47, 1,024 x 3,072 66 and by eight 18, 16
// and 20; 128 rows of 500 x 4,096 x 1,024 45, 1,024 x 2,048 70, by four 78 and 31, by eight 113 and 51.  So a stretch takes
// 1.15 to 1.6 us, a tile 10 to 19 besides; blocks beyond what the SMs hold start when others have ended (with up to 16 rows two
// share an SM, and the time of a stretch).  Clusters lie in one group of SMs: with a block an SM 15 of eight and 33 of four run at
// once, us, 15 and 16 tiles by eight blocks, 16 by four: 128 rows, depth 1,024 18.5 / 28.7 / 24.5, 3,072 26.6 / 45 / 39, 64 rows, 1,024 16.4 / 24.6 /
// 18.5; 33 and 34 tiles of 32 rows by four, depth 512 14.4 and 24.6, 34 by one 20.5.
int split_cuts(int tile, long long tiles, int k) {
  const int stretches = (k + GST_K - 1) / GST_K;
  const double stretch = tile == 16 ? 1.15 : tile == 32 ? 1.2 : tile == 64 ? 1.3 : 1.6, again = tile == 16 ? 2.5 : tile == 128 ? 11.0 : 8.0;
  const double fixed = tile == 16 ? 10.0 : tile == 32 ? 13.0 : tile == 64 ? 14.0 : 19.0;
  int cuts = 1;
  double least = 0.0;
  for (int c = 1; c <= 8; c = c == 1 ? 4 : 2 * c) {
    const int at_once = tile == 16 ? (c == 8 ? 128 : c == 4 ? 136 : 148) : c == 8 ? 120 : c == 4 ? 132 : 148;
    const double layers = (double)((tiles * c + at_once - 1) / at_once);
    const double time = (c == 1 ? fixed : tile == 16 ? 12.5 : 16.0) + (stretches + c - 1) / c * stretch * layers + again * (layers - 1.0);
    if (c == 1 || time < least) cuts = c, least = time;
  }
  return cuts;
}

int split_tile(int n) { return n <= 16 ? 16 : n <= 32 ? 32 : n <= 64 ? 64 : 128; }

int split_product(const Product& p, int batch, bool ahead, cudaStream_t stream) {
  const int tile = split_tile(p.n);
  const int cuts = split_cuts(tile, (long long)((p.o + 127) / 128) * ((p.n + tile - 1) / tile) * batch, p.k);
  switch (tile) {
    case 16: return launch_split<16>(p, batch, cuts, ahead, stream);
    case 32: return launch_split<32>(p, batch, cuts, ahead, stream);
    case 64: return launch_split<64>(p, batch, cuts, ahead, stream);
    default: return launch_split<128>(p, batch, cuts, ahead, stream);
  }
}

// Which kernel: those below give the same bits.
template <typename TX, typename TW>
int launch_typed(const Product& p, int batch, bool ahead, cudaStream_t stream) {
  if (batch > 65535) return FE_ERR_TOO_LARGE;
  auto whole = [](const void* base, long long ld, long long step, long long k, size_t item) {
    return ((uintptr_t)base & 15) == 0 && (ld * item) % 16 == 0 && (step * item) % 16 == 0 && (k * item) % 16 == 0;
  };
  const bool vec = whole(p.x, p.ldx, batch > 1 ? p.batch_x : 0, p.k, sizeof(TX)) &&
                   whole(p.w, p.k, batch > 1 ? p.batch_w : 0, p.k, sizeof(TW));
  if constexpr (sizeof(TX) == 4 && sizeof(TW) == 4) {
    // Deep rows of 32-bit numbers go to the tensor cores, however many there are, so that a row's bits do not depend on that.  us,
    // the kernels below against those: alone, up to four rows lose, 4 x 4,096 x 1,024 14.6 / 17.3, 4 x 6,144 x 1,024 19.4 / 20.5,
    // 4 x 32,000 x 1,024 46 / 51, 4 x 1,024 x 3,072 19.4 / 19.4 (in a decode step of 4 layers, where a product's weights are asked for
    // ahead, 343 / 326 altogether); 16 x 4,096 x 1,024 20.5 / 17.3, 16 x 32,000 x 1,024 72 / 52, 32 x 32,000 x 1,024 116 / 60, 64 x 4,096 x
    // 1,024 43 / 20, 500 x 4,096 x 1,024 118 / 43, 500 x 1,024 x 3,072 111 / 36, 1,024 x 32,000 x 1,024 1,439 / 540.  Shallower than 256
    // a tile's fixed part is more than the sum; up to about 512 it still is with few outputs, 4 x 512 x 256 8 / 12, 200 x 512 x 256 12 / 17,
    // 64 x 512 x 512 16.4 / 13.3, and is not with many, 2,000 x 2,048 x 256 60 / 39 (the line is where the sums are as exact all the same).
    if (vec && p.k >= GST_MIN_K && p.k < (1 << 22) && p.ldx < (1 << 22)) return split_product(p, batch, ahead, stream);
  }
  const long long big = (long long)((p.o + 63) / 64) * ((p.n + 63) / 64) * batch;
  if (!vec) {
    // Rows that do not start on 16 bytes, 32-bit operands, us (one number a copy, 64 x 64 or 32 x 32 tiles by this
    // rule / 32 x 32 always, filled through registers / 64 x 64 by 256 threads, the kernel before both): 16 x 4,096 x
    // 1,023 27 / 35 / 58, 64 x 4,096 x 1,023 45 / 71 / 60, 500 x 1,024 x 3,071 170 / 318 / 181, 500 x 4,096 x 1,023
    // 130 / 216 / 164, 2,000 x 4,096 x 1,023 434 / 783 / 568.
    if (p.n > 32 && (big >= 296 || (p.n <= 64 && big >= 64))) return launch_tile<TX, TW, 8, 4, 8, 16, false>(p, batch, stream);
    return launch_tile<TX, TW, 4, 4, 8, 8, false>(p, batch, stream);
  }
  // From here on operands of which one or both are bfloat16, and 32-bit ones shallower than 256.  Few rows: as many columns a
  // block as still give every SM one.  Measured, us (8 / 16 / 32 columns), bfloat16 weights, then bfloat16 rows, then both:
  // 4 x 1,024 x 3,072 19.4 / 22.5 / 20.5, 20.5 / 25.5 / 21.3, 22.5 / 26.7 / 22.6; 4 x 4,096 x 1,024 14.3 / 13.3 / 12.4,
  // 15.2 / 15.3 / 13.3, 15.1 / 14.4 / 12.4; 4 x 32,000 x 1,024 42 / 36 / 37, 51 / 49 / 43, 43 / 39 / 40; 16 x 1,024 x 3,072
  // 20.5 / 22.6 / 30.8, 20.5 / 25.6 / 36.9, 22.6 / 28.7 / 39.9; 16 x 4,096 x 1,024 22.6 / 17.4 / 15.4, 27.6 / 18.5 / 18.5,
  // 22.6 / 18.5 / 18.6; 16 x 32,000 x 1,024 107 / 75 / 67, 99 / 81 / 70, 98 / 82 / 74.
  if (p.n <= 4) {
    if (p.o <= 2048) return launch_rows<TX, TW, 8, 8, 1>(p, batch, stream);
    if (p.o <= 8192) return launch_rows<TX, TW, 16, 16, 2>(p, batch, stream);
    return launch_rows<TX, TW, 32, 8, 1>(p, batch, stream);
  }
  if (p.n <= 16) {
    if (p.o <= 2048) return launch_rows<TX, TW, 8, 8, 1>(p, batch, stream);
    if (p.o <= 8192) return launch_rows<TX, TW, 16, 8, 2>(p, batch, stream);
    return launch_rows<TX, TW, 32, 16, 4>(p, batch, stream);
  }
  // Many rows: tiles of 64 x 64 by 128 threads (8 x 4 each) where there are about as many as the chip holds twice, else of
  // 32 x 32 by 64 threads.  Measured, us (32 x 32 / 64 x 64), bfloat16 weights, then bfloat16 rows, then shallow 32-bit products
  // (k 192): 20 x 32,000 x 1,024 74 / 119, 72 / 117, 23 / 29; 64 x 4,096 x 1,024 31 / 45, 33 / 43, 12.3 / 16.4; 48 x 8,192 x 1,024
  // 45.2 / 43.7, 45.1 / 43.0, 14.4 / 16.4; 64 x 32,000 x 1,024 137 / 122, 127 / 119, 35 / 31; 100 x 8,192 x 3,072 199 / 193,
  // 199 / 188, 20.5 / 20.5; 200 x 2,048 x 1,024 45.1 / 45.1, 43.0 / 43.7, 14.3 / 16.4; 200 x 16,384 x 3,072 656 / 580, 655 / 576, 49 / 47.
  // (The line of 64 tiles up to 64 rows that 32-bit products once had cost 20 to 64 rows of these up to 1.7 times the time.)
  constexpr int LINE = sizeof(TX) + sizeof(TW) == 8 ? 296 : 256;       // shallow 32-bit ones: 200 x 4,096 x 192 18.5 / 20.5
  if (p.n > 32 && (big >= LINE || (p.n <= 64 && big >= 128))) return launch_tile<TX, TW, 8, 4, 8, 16, true>(p, batch, stream);
  return launch_tile<TX, TW, 4, 4, 8, 8, true>(p, batch, stream);
}

int launch_coded(int x_dtype, int w_dtype, const Product& p, int batch, bool ahead, cudaStream_t stream) {
  if ((p.y_dtype | x_dtype | w_dtype) & ~1) return FE_ERR_BAD_DTYPE;
  switch (x_dtype * 2 + w_dtype) {
    case 0: return launch_typed<float, float>(p, batch, ahead, stream);
    case 1: return launch_typed<float, bf16>(p, batch, ahead, stream);
    case 2: return launch_typed<bf16, float>(p, batch, ahead, stream);
    default: return launch_typed<bf16, bf16>(p, batch, ahead, stream);
  }
}

}  // namespace

// For tests of the bounded waits only: later launches of the kernel for few rows and of the one on the tensor cores poll at most
// `wait_limit` times per wait (0: the usual bound) and do not report stretch `skip_stretch` of 128 k (-1: none), so that the
// block gives up, sets FE_STATUS_WAIT_TIMEOUT and returns.  Call with (0, -1) to go back to normal.
FE_EXPORT void fe_gemm_simt_set_test_fault(unsigned wait_limit, int skip_stretch) {
  g_test_fault = Fault{wait_limit ? wait_limit : tc5::WAIT_LIMIT, skip_stretch};
}

// Into how many blocks a deep product of 32-bit operands cuts k, for its test.
FE_EXPORT int fe_gemm_split_cuts(int n, int o, int k, int batch) {
  const int tile = split_tile(n);
  return split_cuts(tile, (long long)((o + 127) / 128) * ((n + tile - 1) / tile) * batch, k);
}

// `ahead`: w is complete before the call is made and no kernel that may still run writes it (a layer's weights), so that it may be
// read while the kernels before this one still run.  Without it w may be what the kernel before wrote.
FE_EXPORT int fe_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, const float* bias,
                           void* y, int y_dtype, int n, int o, int k, int accumulate, int ahead,
                           int* status, cudaStream_t stream) {
  if (n <= 0 || o <= 0) return 0;
  if (k <= 0) return FE_ERR_BAD_SHAPE;
  return launch_coded(x_dtype, w_dtype, Product{x, w, bias, y, y_dtype, n, o, k, accumulate, status, k, o, 0, 0, 0}, 1, ahead != 0, stream);
}

// `batch` products at once (one per head): product b reads x + b * batch_x (rows ldx apart),
// the [o, k] matrix w + b * batch_w, and writes y + b * batch_y (rows ldy apart).  All strides
// in elements.
FE_EXPORT int fe_gemm_simt_batched(const void* x, int x_dtype, const void* w, int w_dtype, void* y, int y_dtype,
                                   int n, int o, int k, int batch, long long ldx, long long ldy, long long batch_x,
                                   long long batch_w, long long batch_y, int* status, cudaStream_t stream) {
  if (n <= 0 || o <= 0 || batch <= 0) return 0;
  if (k <= 0 || ldx < k || ldy < o) return FE_ERR_BAD_SHAPE;
  return launch_coded(x_dtype, w_dtype, Product{x, w, nullptr, y, y_dtype, n, o, k, 0, status, ldx, ldy, batch_x, batch_w, batch_y},
                      batch, false, stream);
}

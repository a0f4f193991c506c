// 32-bit matrix products on the tensor cores: every operand is split into two tf32 numbers.
//
// x = hi + lo with hi the nearest tf32 number (11 significant bits) and lo the exact rest, of which the
// tensor core reads 11 more; x y is taken as hi hi + lo hi + hi lo (what is left out is 2^-22 of the
// product and below).  The tensor core's own additions truncate, so the large products of every eight k
// are added to the 32-bit sum outside, rounded to nearest; the two small ones, which are 2^-11 of them, stay
// in its accumulator.  What truncating the large ones drops is 4e-8 of them in the mean, for operands of one
// sign and of both, of one magnitude and of many: SPLIT_MEAN puts it back.  Relative error against 64 bits,
// random normal operands, depth 16, 64 and 128: 0.89e-7, 1.01e-7 and 1.14e-7 (of which along the result:
// 0.05e-7); one chain of 32-bit multiply-adds has 0.74e-7, 1.44e-7 and 2.04e-7; without SPLIT_MEAN 0.95e-7,
// 1.07e-7 and 1.19e-7, of which 0.35e-7 along the result, where products in a row add it up.
//
// An infinite operand gives NaN (its rest is infinity less infinity), in the rows or columns it belongs to.
//
// Fragments of mma.m16n8k8 (lane = 4 g + q): A rows g, g + 8 x columns q, q + 4; B rows q, q + 4 x column g;
// the sum's rows g, g + 8 x columns 2 q, 2 q + 1.
#pragma once
#include "common.cuh"

struct SplitA { unsigned hi[4], lo[4]; };
struct SplitB { unsigned hi[2], lo[2]; };

__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  lo = __float_as_uint(x - __uint_as_float(hi));
}
// A[m][k] at a[m * row + k * col], for this lane's place.
__device__ __forceinline__ void split_load_a(SplitA& f, const float* a, int row, int col) {
  split_tf32(a[0], f.hi[0], f.lo[0]);
  split_tf32(a[8 * row], f.hi[1], f.lo[1]);
  split_tf32(a[4 * col], f.hi[2], f.lo[2]);
  split_tf32(a[8 * row + 4 * col], f.hi[3], f.lo[3]);
}
// B[k][n] at b[k * row], for this lane's place.
__device__ __forceinline__ void split_load_b(SplitB& f, const float* b, int row) {
  split_tf32(b[0], f.hi[0], f.lo[0]);
  split_tf32(b[4 * row], f.hi[1], f.lo[1]);
}
__device__ __forceinline__ void split_mma_raw(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
#define SPLIT_MEAN 4e-8f
// sum += A B over eight k; `small` collects the two small products and joins at the end (split_join).
__device__ __forceinline__ void split_mma(float (&sum)[4], float (&small)[4], const SplitA& a, const SplitB& b) {
  float large[4] = {0.f, 0.f, 0.f, 0.f};
  split_mma_raw(large, a.hi, b.hi);
  split_mma_raw(small, a.lo, b.hi);
  split_mma_raw(small, a.hi, b.lo);
#pragma unroll
  for (int i = 0; i < 4; ++i) sum[i] += large[i];
}
__device__ __forceinline__ float split_join(float sum, float small) { return sum + fmaf(sum, SPLIT_MEAN, small); }

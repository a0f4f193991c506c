// 32-bit matrix products on the tensor cores: every operand is split into three bfloat16 numbers.
//
// x = a + b + c: a is x rounded to 7 significant bits, b the rest rounded to 8, c the rest of that rounded to 8 (what
// is left is 2^-25 of x and below).  x y is taken as aa + (ab + ba + bb + ac + ca); what is left out is 2^-25 of
// the product and below.  The tensor core adds up the products of an instruction exactly but for what falls below the
// 24 bits of the result, which it cuts off.  Products of 7 by 7 bits leave little to cut off; those of every eight k are added
// to the 32-bit sum outside, rounded to nearest.  The others are 2^-7 of them and stay in the tensor core's
// accumulator, sixteen k an instruction where there are as many (the tensor core takes as long for one as for two of eight; it is
// one instruction).  Relative error against 64 bits (of it along the result), 1e-7, random normal operands, depth 8, 16, 64
// and 256: 0.35, 0.37, 0.46 and 0.74 (-0.02); one chain of 32-bit multiply-adds 0.54, 0.73, 1.46 and 2.86.  Two tf32 numbers
// an operand, three products: 0.85, 0.90, 1.02 and 1.35, more than the chain where few products count.
//
// An operand that is infinite, or that rounds to infinity (split_loud), gives NaN in the rows or columns it belongs to, whatever
// it is multiplied with, zeros too.
//
// Fragments of mma.m16n8k8 (lane = 4 g + q): A rows g, g + 8 x columns q, q + 4; B rows q, q + 4 x column g;
// the sum's rows g, g + 8 x columns 2 q, 2 q + 1.  (The instruction calls its eight k 2 q and 2 q + 1 of a lane; which is which
// does not matter as long as A and B agree.)
#pragma once
#include "common.cuh"

struct SplitA { unsigned part[3][2]; };      // of rows g and g + 8: columns q (low half) and q + 4
struct SplitB { unsigned part[3]; };         // of column g: rows q (low half) and q + 4

// Whether x, or x rounded to 7 bits, is not finite.
__device__ __forceinline__ bool split_loud(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x7f7f0000u; }
// Two numbers into the halves of a, b and c.
__device__ __forceinline__ void split_pair(float x, float y, unsigned& a, unsigned& b, unsigned& c) {
  const unsigned u = (__float_as_uint(x) + 0x10000u) & 0xfffe0000u, v = (__float_as_uint(y) + 0x10000u) & 0xfffe0000u;
  a = __byte_perm(u, v, 0x7632);
  x -= __uint_as_float(u), y -= __uint_as_float(v);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b) : "f"(y), "f"(x));
  x -= __uint_as_float(b << 16), y -= __uint_as_float(b & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(c) : "f"(y), "f"(x));
}
// A[m][k] at a[m * row + k * col], for this lane's place.
__device__ __forceinline__ void split_load_a(SplitA& f, const float* a, int row, int col) {
  split_pair(a[0], a[4 * col], f.part[0][0], f.part[1][0], f.part[2][0]);
  split_pair(a[8 * row], a[8 * row + 4 * col], f.part[0][1], f.part[1][1], f.part[2][1]);
}
// B[k][n] at b[k * row], for this lane's place.
__device__ __forceinline__ void split_load_b(SplitB& f, const float* b, int row) {
  split_pair(b[0], b[4 * row], f.part[0], f.part[1], f.part[2]);
}
__device__ __forceinline__ void split_mma_raw(float (&c)[4], const unsigned (&a)[2], unsigned b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(b));
}
// The same of sixteen k: the first eight in a[0..1] and b[0], the others behind them.
__device__ __forceinline__ void split_mma_raw(float (&c)[4], const unsigned (&a)[2], const unsigned (&a2)[2], unsigned b, unsigned b2) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a2[0]), "r"(a2[1]), "r"(b), "r"(b2));
}
// sum += A B over eight k of the leading parts, rounded to nearest.
__device__ __forceinline__ void split_mma_large(float (&sum)[4], const unsigned (&a)[2], unsigned b) {
  float large[4];
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
      : "=f"(large[0]), "=f"(large[1]), "=f"(large[2]), "=f"(large[3])
      : "r"(a[0]), "r"(a[1]), "r"(b), "f"(0.f));
#pragma unroll
  for (int i = 0; i < 4; ++i) sum[i] += large[i];
}
// sum += A B over eight k; `small` collects the small products and joins at the end (split_join).
__device__ __forceinline__ void split_mma(float (&sum)[4], float (&small)[4], const SplitA& a, const SplitB& b) {
  split_mma_large(sum, a.part[0], b.part[0]);
  split_mma_raw(small, a.part[0], b.part[1]);
  split_mma_raw(small, a.part[1], b.part[0]);
  split_mma_raw(small, a.part[1], b.part[1]);
  split_mma_raw(small, a.part[0], b.part[2]);
  split_mma_raw(small, a.part[2], b.part[0]);
}
// The same over sixteen k, eight in a and b and eight in a2 and b2.
__device__ __forceinline__ void split_mma(float (&sum)[4], float (&small)[4], const SplitA& a, const SplitA& a2, const SplitB& b, const SplitB& b2) {
  split_mma_large(sum, a.part[0], b.part[0]);
  split_mma_large(sum, a2.part[0], b2.part[0]);
  split_mma_raw(small, a.part[0], a2.part[0], b.part[1], b2.part[1]);
  split_mma_raw(small, a.part[1], a2.part[1], b.part[0], b2.part[0]);
  split_mma_raw(small, a.part[1], a2.part[1], b.part[1], b2.part[1]);
  split_mma_raw(small, a.part[0], a2.part[0], b.part[2], b2.part[2]);
  split_mma_raw(small, a.part[2], a2.part[2], b.part[0], b2.part[0]);
}
__device__ __forceinline__ float split_join(float sum, float small) { return sum + small; }

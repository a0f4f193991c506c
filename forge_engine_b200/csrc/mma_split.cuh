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

// Tiles that are split once, by whoever writes them: three planes of bfloat16, `plane` numbers apart, rows a multiple of 16
// bytes apart (an odd one: then the eight rows of a matrix fall into different banks).  A fragment of sixteen k, k
// 2 q and 2 q + 1 of a lane in the low and high half of a register.
struct PlanesA { unsigned part[3][4]; };
struct PlanesB { unsigned part[3][2]; };
__device__ __forceinline__ unsigned split_address(const bf16* p) { return (unsigned)__cvta_generic_to_shared(p); }
// A[m][k], 16 x 16, at a[k * pitch + m].
__device__ __forceinline__ void planes_load_a_by_k(PlanesA& f, const bf16* a, int pitch, int plane) {
  const int lane = threadIdx.x & 31;
  const unsigned at = split_address(a + ((lane >> 4) * 8 + (lane & 7)) * pitch + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(f.part[i][0]), "=r"(f.part[i][1]), "=r"(f.part[i][2]), "=r"(f.part[i][3]) : "r"(at + 2 * i * plane) : "memory");
}
// B[k][n], 16 x 8, at b[k * pitch + n].
__device__ __forceinline__ void planes_load_b_by_k(PlanesB& f, const bf16* b, int pitch, int plane) {
  const unsigned at = split_address(b + (threadIdx.x & 15) * pitch);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];"
                 : "=r"(f.part[i][0]), "=r"(f.part[i][1]) : "r"(at + 2 * i * plane) : "memory");
}
// Two neighbouring numbers of a row into the planes.
__device__ __forceinline__ void planes_store2(bf16* to, int plane, float x, float y) {
  unsigned a, b, c;
  split_pair(x, y, a, b, c);
  *reinterpret_cast<unsigned*>(to) = a;
  *reinterpret_cast<unsigned*>(to + plane) = b;
  *reinterpret_cast<unsigned*>(to + 2 * plane) = c;
}
// The small products of each kind in an accumulator of their own: where little else runs, a chain of them is what is waited for.
__device__ __forceinline__ void split_mma(float (&sum)[4], float (&small)[5][4], const PlanesA& a, const PlanesB& b) {
  const unsigned lo[2] = {a.part[0][0], a.part[0][1]}, hi[2] = {a.part[0][2], a.part[0][3]};
  const unsigned lo1[2] = {a.part[1][0], a.part[1][1]}, hi1[2] = {a.part[1][2], a.part[1][3]};
  const unsigned lo2[2] = {a.part[2][0], a.part[2][1]}, hi2[2] = {a.part[2][2], a.part[2][3]};
  split_mma_large(sum, lo, b.part[0][0]);
  split_mma_large(sum, hi, b.part[0][1]);
  split_mma_raw(small[0], lo, hi, b.part[1][0], b.part[1][1]);
  split_mma_raw(small[1], lo1, hi1, b.part[0][0], b.part[0][1]);
  split_mma_raw(small[2], lo1, hi1, b.part[1][0], b.part[1][1]);
  split_mma_raw(small[3], lo, hi, b.part[2][0], b.part[2][1]);
  split_mma_raw(small[4], lo2, hi2, b.part[0][0], b.part[0][1]);
}
__device__ __forceinline__ float split_join(float sum, const float (&small)[5][4], int i) {
  return sum + ((small[0][i] + small[1][i]) + ((small[3][i] + small[4][i]) + small[2][i]));
}

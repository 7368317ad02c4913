// f64_mma.cuh -- complex products on the FP64 tensor cores (mma.sync m8n8k4).
//
// All users contract a complex operand A (rows x k) with a complex operand B
// (k x right-hand sides).  One MMA pair serves 8 rows, 4 right-hand sides and
// 4 complex k:
//
//   A fragment   lane holds the complex A[row = lane / 4][k = lane % 4]
//   B fragment   column n = lane / 4 of the real product is part n % 2 (0 real,
//                1 imaginary) of right-hand side n / 2, so the lane holds the
//                complex B[k = lane % 4][rhs = lane / 8] and hands the MMAs
//                (re, -im) for a real column, (im, re) for an imaginary one
//   accumulator  lane holds the complex C[row = lane / 4][rhs = lane % 4]
//
//   C += Re(A) * first + Im(A) * second
//
// so the complex product costs its four real products and nothing else, the
// results come out interleaved (16-byte stores), and right-hand sides are
// padded to multiples of 4 rather than 8.  Both operands are read straight
// from global memory in fragment order: a load instruction of a warp covers
// 64-byte (A) or 128-byte runs, and the operands' reuse is in the registers of
// the warp that owns the whole tile, so no shared memory and no barrier stands
// between the loads and the MMAs.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gmg {
namespace f64mma {

__device__ __forceinline__ void mma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ double flip(double v, uint32_t sign) {
  return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}

// The B operands of one complex number (see above): part (lane / 4) % 2 of the
// column, s0 / s1 the sign bits (0x80000000 or 0) of the first and second
// operand on top of the plain product's own.  conjugate: the product with
// conj(A) instead, whose second operands are the negatives.
template <class C>
__device__ __forceinline__ void expand(C v, int part, uint32_t s0, uint32_t s1, double& b0, double& b1) {
  b0 = flip((double)(part ? v.y : v.x), s0);
  b1 = flip((double)(part ? v.x : v.y), s1);
}
// sign bit of the second operand: real columns take -im (conj: +im), imaginary
// ones +re (conj: -re)
__device__ __forceinline__ uint32_t second_sign(int part, bool conj) {
  return ((part == 0) != conj) ? 0x80000000u : 0u;
}

}  // namespace f64mma
}  // namespace gmg

// dmma.cuh -- FP64 tensor-core products for the reciprocal sums.
//
// mma.sync m16n8k4 with FP64 operands and accumulators.  On this part it runs at
// the FP64 FMA rate (18.5e12 multiply-adds a second measured, the same pipe as DFMA), but one
// instruction carries 512 of them and its operands are two registers of A and
// one of B per lane: the reciprocal contractions, which are short of issue slots and of
// operand bandwidth on scalar FMAs, come within reach of the pipe's rate, in
// full FP64.
#pragma once
#include <cuda_runtime.h>

namespace mdff {

// D[16][8] += A[16][4] B[4][8]: lane l (g = l / 4, t = l % 4) holds A[g][t] in
// a0, A[g + 8][t] in a1, B[t][g] in b, and D[g][2t], D[g][2t + 1], D[g + 8][2t],
// D[g + 8][2t + 1] in d
__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}

__device__ __forceinline__ double flip_if(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}

}  // namespace mdff

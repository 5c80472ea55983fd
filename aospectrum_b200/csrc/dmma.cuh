// FP64 matrix instruction for complex128 products.
//
// mma.m8n8k4: lane l holds A(l / 4, l % 4), B(l % 4, l / 4) and the pair
// C(l / 4, 2 (l % 4) + {0, 1}).  It runs at the rate of scalar FP64 FMAs (37
// TFLOP/s measured for both), but a lane loads one element of each operand for
// 256 products instead of one per product or two, so kernels built on it are
// not bound by shared memory.
#pragma once

#include "common.cuh"

namespace aosb {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Complex accumulator block and (re, im) += a b.
struct DBlock {
  double re[2], im[2];
};
__device__ __forceinline__ void zmma(DBlock& c, double2 a, double2 b) {
  dmma(c.re, a.x, b.x);
  dmma(c.im, a.x, b.y);
  dmma(c.re, -a.y, b.y);
  dmma(c.im, a.y, b.x);
}

}  // namespace aosb

// A double-precision reciprocal in few FP64 operations.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

namespace rx {

// 1 / x in double precision: for x well within single precision's range the
// single-precision reciprocal and two Newton steps (a double division is three times the
// FP64 operations, and the FP64 pipe is what bounds the records of k_records), else the
// division. Relative error at most 2^-53 (1 + 2^-38): the reciprocal of x rounded to single
// precision is within 2^-23, a Newton step squares that, and the last step's sum is rounded
// once.
__host__ __device__ __forceinline__ double rcp64(double x) {
  if (!(x > 1e-30 && x < 1e30)) return 1.0 / x;
  double y = (double)(1.0f / (float)x);
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

}  // namespace rx

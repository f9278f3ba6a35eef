// From the exact integer sums of the integer GEMMs to the float they stand for.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cb200 {

// y value from the exact integer sums: (256*hi + lo - zero*qsum) as float. Integer zero points in
// [-255, 255] (what the reference packer produces) are handled in integers, anything else in double precision.
// (The double-precision form is rare and kept out of line so that the epilogues stay short.)
static __device__ __noinline__ float recombine_fractional(int32_t hi, int32_t lo, float zero, int qsum) {
  return static_cast<float>(256.0 * hi + static_cast<double>(lo) - static_cast<double>(zero) * qsum);
}
// `zero_int` is the zero point as an integer and `zero_is_int` says whether that is exact; both are
// per-thread constants worked out once, outside the loops over the batch rows.
__device__ __forceinline__ float recombine(int32_t hi, int32_t lo, float zero, int zero_int, bool zero_is_int, int qsum) {
  if (zero_is_int) {
    // 32-bit arithmetic only (64-bit integer math and its conversion cost several times more issue
    // slots): with qsum = 256*qh + ql, v = 256*(hi - z*qh) + (lo - z*ql); both brackets fit in 32 bits
    // for |z| <= 255. The float of v is exact-rounded while the first bracket is below 2^24
    // (|v| < 2^32, far above what cancelled sums reach), and within 1.5 units in the last place beyond.
    const int a = hi - zero_int * (qsum >> 8);
    const int b = lo - zero_int * (qsum & 255);
    return fmaf(static_cast<float>(a), 256.f, static_cast<float>(b));
  }
  return recombine_fractional(hi, lo, zero, qsum);
}

}  // namespace cb200

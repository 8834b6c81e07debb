// widen.cuh -- FP32 to FP64 with integer instructions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rte {

// The conversion instruction runs at the FP64 unit's rate, a sixty-fourth of
// the integer units' on this GPU, and would take as long as the FP64
// operation that follows.  Exact for zeros and normal numbers; `special` is
// set for the rest (denormals, infinities, NaN), whose result is not valid.
__device__ __forceinline__ double widen(float f, bool& special) {
  const uint32_t u = __float_as_uint(f), e = u & 0x7f800000u;
  special |= e == 0x7f800000u || (e == 0u && (u & 0x007fffffu) != 0u);
  const uint32_t hi = e == 0u ? u : (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u);
  return __hiloint2double((int)hi, (int)(u << 29));
}

// Any value.
__device__ __forceinline__ double widen(float f) {
  bool special = false;
  const double d = widen(f, special);
  return special ? (double)f : d;
}

}  // namespace rte

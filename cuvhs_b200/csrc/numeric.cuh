// Conversions that keep off the conversion unit (a quarter of the FP32 rate,
// and what bound the resamplers beside instruction issue).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cuvhs {

// (double)i: the integer, offset to unsigned, as the low word of a double of
// exponent 2^52, less that offset.  Exact for every int.
__device__ __forceinline__ double int_to_double(int i) {
  return __hiloint2double(0x43300000, i ^ (int)0x80000000) - 4503601774854144.0;
}

// Positions ci whose four taps ci - 1 .. ci + 2 lie in a signal of total samples
// (under 2^31): those with (unsigned)ci - 1 below this.
__device__ __forceinline__ unsigned tap_range(long long total) { return total > 3 ? (unsigned)(total - 3) : 0u; }

// (uint16_t)v for 0 <= v < 65536: added to 2^23 rounding down, the integer
// part is the low mantissa bits.
__device__ __forceinline__ uint16_t trunc_u16(float v) {
  return (uint16_t)__float_as_uint(__fadd_rz(v, 8388608.0f));
}

}  // namespace cuvhs

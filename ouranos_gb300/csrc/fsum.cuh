// A warp's sum of FP32 values in 64-bit fixed point, at the accuracy of FP64 or better.
// Every value is placed on the grid of the warp's largest exponent with 34 bits below
// that value's last place, so the integers add exactly and in any order; what is cut
// off is at most 2^-57 of the largest value each, and the total is rounded once, to
// FP64 (an FP64 tree rounds 31 times).  GB300 adds two FP64 lanes a clock but reduces
// 32-bit integers of a whole warp in one instruction.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

namespace ouranos {

constexpr int kFixedBits = 34;  // below the largest value's last place: 32 values of 24 + 34 bits fit 63

// value `bits` (an FP32 number, not infinite or NaN) on the grid of exponent emax >= its own
__host__ __device__ inline int64_t fixed_of(uint32_t bits, int emax) {
  const int f = (int)(bits >> 23) & 255;
  const uint32_t m = (bits & 0x7fffffu) | (f ? 0x800000u : 0u);
  const int sh = emax - (f ? f : 1);
  const int64_t v = sh < 64 ? (int64_t)(((uint64_t)m << kFixedBits) >> sh) : 0;
  return bits >> 31 ? -v : v;
}
// the grid's exponent for a largest magnitude of these bits
__host__ __device__ inline int fixed_exponent(uint32_t bits) {
  const int f = (int)(bits >> 23) & 255;
  return f ? f : 1;
}
// an integer of the grid as FP64 (one rounding)
__host__ __device__ inline double fixed_value(int64_t total, int emax) {
  const uint64_t scale = (uint64_t)(1023 + emax - 150 - kFixedBits) << 52;  // 2^(emax - 184)
  double s;
  memcpy(&s, &scale, 8);
  return (double)total * s;
}

#ifdef __CUDACC__
// lane's share of a warp's sum: the whole warp gets the total and its exponent; 255:
// some value is infinite or NaN, and there is no total
__device__ __forceinline__ int64_t warp_fixed_sum(float t, int& emax) {
  const uint32_t bits = __float_as_uint(t);
  const uint32_t top = __reduce_max_sync(0xffffffffu, bits & 0x7fffffffu);
  emax = fixed_exponent(top);
  if (emax == 255) return 0;  // (the same in all lanes)
  const int64_t v = fixed_of(bits, emax);
  // 26 + 26 bits and the signed rest: 32 of each fit 32 bits
  const uint32_t l0 = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0x3ffffffu);
  const uint32_t l1 = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 26) & 0x3ffffffu);
  const int32_t l2 = __reduce_add_sync(0xffffffffu, (int32_t)(v >> 52));
  return (int64_t)l0 + ((int64_t)l1 << 26) + (int64_t)((uint64_t)(int64_t)l2 << 52);
}
#endif

}  // namespace ouranos

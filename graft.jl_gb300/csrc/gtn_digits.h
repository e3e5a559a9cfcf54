// Device helper of the base-256 digits (digit_word in gtn_layout.cu, gtn_gemm_f64e.cu).
#pragma once
#include <cuda_runtime.h>

// The eighth digit of x under row exponent E: what the seven (rounded half up) leave, in units of 2^-64.
__device__ __forceinline__ int low_digit(double x, int E) {
  const long long bits = __double_as_longlong(x);
  const int e = (int)((bits >> 52) & 0x7ff), r = E - e - 2;
  if (e == 0 || r <= 0 || r >= 62) return 0;
  const long long mant = (bits & 0xFFFFFFFFFFFFFll) | (1ll << 52);
  const long long rest = mant - (r < 60 ? ((mant + (1ll << (r - 1))) >> r) << r : 0);
  const int d = r >= 9 ? (int)((rest + (1ll << (r - 9))) >> (r - 8)) : (int)(rest << (8 - r));
  return bits < 0 ? -d : d;
}

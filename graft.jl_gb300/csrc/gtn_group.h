// Device helper of strided tensor views: the element offset of a multi-index group's index.
#pragma once
#include "gtn_internal.h"

__device__ __forceinline__ int64_t decompose(int64_t i, const GroupSpec& g) {
  int64_t off = 0;
#pragma unroll 1
  for (int j = g.n - 1; j > 0; --j) {
    const int64_t d = g.dim[j];
    const int64_t q = i / d;
    off += (i - q * d) * g.str[j];
    i = q;
  }
  return g.n > 0 ? off + i * g.str[0] : 0;  // what is left is the first leg's index: no division
}

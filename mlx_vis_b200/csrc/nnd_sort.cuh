// Sorted lists of up to 32 (distance, id) keys, one per lane of a warp, for the NNDescent
// row kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace umapb {
namespace nnd {

constexpr float kBig = 1e30f;         // distance of a dropped column (the row itself, a repeated id)
// Behind a list of fewer than 32 keys: (INFINITY, 0x7fffffff), above every key.  Distances can be
// infinite themselves (an FP16 dot product below -65,504, an FP32 overflow), so a mark that
// a kernel compares with them has to be a NaN.
constexpr float kSent = INFINITY;

__device__ __forceinline__ bool key_lt(float a, int ia, float b, int ib) {
  return a < b || (a == b && ia < ib);
}

// ascending bitonic sort of one (distance, id) key per lane across the warp
__device__ __forceinline__ void warp_sort_keys(float& d, int& id, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const float od = __shfl_xor_sync(0xffffffffu, d, stride);
      const int oi = __shfl_xor_sync(0xffffffffu, id, stride);
      const bool lower = (lane & stride) == 0, asc = (lane & size) == 0;
      const bool take = (lower == asc) ? key_lt(od, oi, d, id) : key_lt(d, id, od, oi);
      if (take) {
        d = od;
        id = oi;
      }
    }
  }
}

// ascending order of a bitonic sequence held one key per lane
__device__ __forceinline__ void warp_bitonic_clean(float& d, int& id, int lane) {
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    const float od = __shfl_xor_sync(0xffffffffu, d, stride);
    const int oi = __shfl_xor_sync(0xffffffffu, id, stride);
    const bool take = (lane & stride) == 0 ? key_lt(od, oi, d, id) : key_lt(d, id, od, oi);
    if (take) {
      d = od;
      id = oi;
    }
  }
}

// Inserts (d, id) into the warp-distributed ascending list (lane l holds entry l).
__device__ __forceinline__ void list_insert(float& lv, int& li, float d, int id, int k, int lane) {
  const int pos = __popc(__ballot_sync(0xffffffffu, lane < k && key_lt(lv, li, d, id)));
  const float up_v = __shfl_up_sync(0xffffffffu, lv, 1);
  const int up_i = __shfl_up_sync(0xffffffffu, li, 1);
  if (lane < k) {
    if (lane > pos) {
      lv = up_v;
      li = up_i;
    } else if (lane == pos) {
      lv = d;
      li = id;
    }
  }
}

}  // namespace nnd
}  // namespace umapb

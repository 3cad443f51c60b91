// Pivot search inside a warp, shared by the panel leaf and the batched solver.
#pragma once
#include <cuda_runtime.h>

namespace lub {

// Lane whose (a, pos) is best: largest a among lanes with ok, the lowest
// position on ties; -1 when no lane is ok.  a >= 0 and not NaN where ok, so
// its bit pattern orders as the value does.
__device__ __forceinline__ int lowest_pos(unsigned mask, int pos) {
  if (mask & (mask - 1u)) {
    const int lane = threadIdx.x & 31;
    const bool in = (mask >> lane) & 1u;
    const unsigned best = __reduce_min_sync(0xffffffffu, in ? (unsigned)pos : 0xffffffffu);
    mask = __ballot_sync(0xffffffffu, in && (unsigned)pos == best);
  }
  return __ffs((int)mask) - 1;
}
__device__ __forceinline__ int warp_best(float a, bool ok, int pos) {
  const unsigned k = ok ? __float_as_uint(a) : 0u;
  const unsigned m = __reduce_max_sync(0xffffffffu, k);
  return lowest_pos(__ballot_sync(0xffffffffu, ok && k == m), pos);
}
__device__ __forceinline__ int warp_best(double a, bool ok, int pos) {
  const unsigned hi = ok ? (unsigned)__double2hiint(a) : 0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  bool in = ok && hi == mh;
  unsigned mask = __ballot_sync(0xffffffffu, in);
  if (mask & (mask - 1u)) {
    const unsigned lo = in ? (unsigned)__double2loint(a) : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    in = in && lo == ml;
    mask = __ballot_sync(0xffffffffu, in);
    return lowest_pos(mask, pos);
  }
  return __ffs((int)mask) - 1;
}

}  // namespace lub

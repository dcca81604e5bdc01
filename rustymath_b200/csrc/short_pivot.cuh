// The pivot choice of the one-launch cluster LU: a candidate's key is its magnitude's bits plus an offset
// (so that keys order as magnitudes do and 0 means "no candidate"); of equal keys the lowest
// position wins, as rustymath's `largest` (factor.rs:476).
#pragma once

namespace rm {

// The lane holding the warp's largest key, the lowest position among equal keys; `zero` when
// every key is 0.
__device__ __forceinline__ int short_reduce(unsigned long long key, unsigned pos, bool& zero) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned top = __ballot_sync(0xffffffffu, hi == mhi);
  zero = false;
  if (__popc(top) == 1) return __ffs(top) - 1;  // mhi > 0 here: at most one lane holds a key of 0
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  const bool tie = hi == mhi && lo == mlo;
  const unsigned pmin = __reduce_min_sync(0xffffffffu, tie ? pos : 0xffffffffu);
  zero = mhi == 0u && mlo == 0u;
  return __ffs(__ballot_sync(0xffffffffu, tie && pos == pmin)) - 1;
}

// 1 / pivot, correctly rounded (0 for a subnormal pivot, which is divided by)
__device__ __forceinline__ double short_rcp(double pv) {
  return fabs(pv) < 2.2250738585072014e-308 ? 0.0 : __drcp_rn(pv);
}

}  // namespace rm

#pragma once

namespace bem {

// sum over the warp of eight values per lane: lane 4 q holds value q's sum
// (recursive halving: 9 adds instead of 40)
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int k = 4, o = 16; k >= 1; k >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < k; ++q) {
      const double send = up ? v[q] : v[q + k], keep = up ? v[q + k] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

}  // namespace bem

// deb_warp_sums.cuh -- many sums over a warp at once.  Plain source without
// CUDA headers: the test suite runs it on the host, a thread per lane.
#pragma once

namespace deb {

// Sums of N <= 32 values over the warp, sum i into out[i]: while a lane holds
// more than one value the two halves of them are exchanged, then the one left
// is summed over the remaining lane bits, so N values take about N + 4
// additions instead of 5 N.  Each sum is stored by one lane, the one whose
// remaining bits are clear (several lanes storing to one address would leave
// open which value stays).
template <int N>
__device__ __forceinline__ void warp_sums(double* x, int lane, double* out) {
  int cnt = N, own = 0, left = N;   // left: values of x in this lane that are not padding
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int half = (cnt + 1) >> 1;
    const bool up = (lane & o) != 0;
    if (cnt == 1) {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
      left = up ? 0 : left;
    } else {
#pragma unroll
      for (int i = 0; i < (N + 1) / 2; ++i) {
        if (i < half) {
          const double lo = x[i], hi = (i + half < cnt) ? x[i + half < N ? i + half : 0] : 0.0;
          const double send = up ? lo : hi, keep = up ? hi : lo;
          x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      own += up ? half : 0;
      left = up ? left - half : (left < half ? left : half);
      cnt = half;
    }
  }
  if (left > 0) out[own] = x[0];
  __syncwarp();
}

}  // namespace deb

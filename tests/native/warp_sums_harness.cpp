// Test-only emulation of a warp on the host: 32 threads, one per lane, whose
// shuffles meet at a barrier.  Every lane gets a result array of its own, so
// that what each of them would store is seen.
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

namespace {

struct Warp {
  std::mutex mu;
  std::condition_variable cv;
  int waiting = 0;
  long turn = 0;
  double slot[32];
  void meet() {
    std::unique_lock<std::mutex> lk(mu);
    const long t = turn;
    if (++waiting == 32) {
      waiting = 0;
      ++turn;
      cv.notify_all();
    } else {
      cv.wait(lk, [&] { return turn != t; });
    }
  }
};
Warp* g_warp;
thread_local int t_lane;

double __shfl_xor_sync(unsigned, double x, int o) {
  g_warp->slot[t_lane] = x;
  g_warp->meet();
  const double y = g_warp->slot[t_lane ^ o];
  g_warp->meet();
  return y;
}
void __syncwarp() {}

}  // namespace

#define __device__
#define __forceinline__ inline
#include "../../disco-eb_gb300/csrc/deb_warp_sums.cuh"

namespace {

template <int N>
void run(const double* in, double* out) {
  Warp w;
  g_warp = &w;
  std::vector<std::thread> lanes;
  for (int l = 0; l < 32; ++l)
    lanes.emplace_back([=] {
      t_lane = l;
      double x[N];
      for (int i = 0; i < N; ++i) x[i] = in[l * N + i];
      deb::warp_sums<N>(x, l, out + l * N);
    });
  for (auto& t : lanes) t.join();
}

template <int... Ns>
bool pick(int n, const double* in, double* out, std::integer_sequence<int, Ns...>) {
  return ((n == Ns + 1 ? (run<Ns + 1>(in, out), true) : false) || ...);
}

}  // namespace

// in, out: [32][n], out: what each lane stores (untouched where it stores nothing)
extern "C" int h_warp_sums(int n, const double* in, double* out) {
  return pick(n, in, out, std::make_integer_sequence<int, 20>()) ? 0 : 1;
}

// z2_schedule.h -- how a launch of many chains is laid out on the SMs: a chain's
// relative time, and which build of the chain kernel runs a batch of small
// lattices.  No CUDA types: the host test compiles it as it is.
#pragma once
#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>
#include <vector>

// Relative time of one chain's bin, from the cycles per slice measured at N = 16,
// 36, 64, 100, 144 (65, 134, 183, 466, 688 K) and 256 (5 M: G outside the SM).
inline double z2_chain_cost(int N, int Ltrot, bool g_in_smem) {
  const double n = N;
  return (double)Ltrot * (30.0 + 2.2 * n + 0.016 * n * n) * (g_in_smem ? 1.0 : 3.0);
}

struct Z2ChainLoad {
  int N;
  double cost;     // z2_chain_cost
};

// Length of the work queue's schedule (longest chain first onto the first free of
// `slots` blocks); time(i): chain i in that order.
template <class Time>
inline double z2_makespan(int n, int slots, Time time) {
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (int i = 0; i < slots; ++i) free_at.push(0.0);
  double t = 0.0;
  for (int i = 0; i < n; ++i) {
    const double end = free_at.top() + time(i);
    free_at.pop();
    free_at.push(end);
    t = std::max(t, end);
  }
  return t;
}

// Blocks per SM of the 128-thread kernel, of which occ fit, or 0 for the 256-thread
// kernel (one block per SM): whichever has the shortest schedule.  A chain alone
// on an SM takes 0.98, 1.12 and 1.22 times as long with 128 threads as with 256
// (L = 4, 6, 8), and slow[k] times that as one of k on its SM (in the last round
// of the queue, as many as are left).  Measured on 6 x 6 lattices, 40 slices (ms
// per round of b blocks per SM): 2.4, 3.1, 3.9, 4.9 for b = 1..4; throughput is
// level from b = 2 (2000 chains: 39, 28, 28, 28 ms), so b rises above 2 where it
// saves a round (300 8 x 8 chains, 40 slices: 9.9 ms at 2, 6.4 at 3; 256 threads:
// 10.6) and stays at 2 where a few long chains set the time (512 chains of 4 x 4
// and 6 x 6: 8.2 ms at 2, 10.7 at 4; 256 threads: 10.5).  The 256-thread kernel
// stays where only one block fits beside a large delay rank (300 8 x 8 chains at
// rank 64: 11.6 ms, 13.2 with 128 threads) and where single chains set the time
// (200 4 x 4 chains and one 8 x 8 of 320 slices: 25.4 against 30.9 ms; 128 chains
// each of 4 x 4 and 8 x 8, 80 slices: 10.0 against 11.0).
inline int z2_small_blocks_per_sm(std::vector<Z2ChainLoad> chains, int nsm, int occ) {
  static const double slow[5] = {1.0, 1.0, 1.3, 1.65, 2.05};
  const int n = (int)chains.size();
  std::sort(chains.begin(), chains.end(),
            [](const Z2ChainLoad &a, const Z2ChainLoad &b) { return a.cost > b.cost; });
  int best = 0;
  double tbest = z2_makespan(n, nsm, [&](int i) { return chains[i].cost; });
  for (int b = 1; b <= std::min(occ, 4); ++b) {
    const int slots = b * nsm;
    const double t = z2_makespan(n, slots, [&](int i) {
      const int left = n - i / slots * slots;          // when this chain's round begins
      const int k = std::min(b, (left + nsm - 1) / nsm);
      return chains[i].cost * (0.75 + 0.058 * std::sqrt((double)chains[i].N)) * slow[k];
    });
    if (t < tbest) { best = b; tbest = t; }
  }
  return best;
}

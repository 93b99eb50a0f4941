// Host check of what planning half-range passes costs (plan_half): passes that
// share a set for as long as it looks, against the additions that the search
// cannot do without, timed in the same process.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <vector>

#include "plan.h"

using namespace dmg;

static double now() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

int main() {
  const int m = 4000, reach = 256;
  std::vector<HalfCost> c(m);
  for (int i = 0; i < m; i++) c[i] = {0x3E0u, 2.5, 0.01 + 0.001 * (i % 7), 1000, 1};
  double best = 1e9, floor = 1e9;
  volatile double sink = 0;
  for (int r = 0; r < 5; r++) {
    double t = now();
    double gain = 0;
    const std::vector<uint32_t> S = plan_half(c, 5, 10, &gain);
    best = std::min(best, now() - t);
    if (S[m / 2] == 0 || gain <= 0) return std::printf("no half range planned\n"), 1;
    // one addition after the other per pass, |S| and step: 5 m reach of them
    std::vector<double> us(5 * m, 1.25);
    t = now();
    for (int i = 0; i < m; i++) {
      double sum[5] = {0};
      for (int j = i; j < m && j < i + reach; j++) {
        for (int s = 0; s < 5; s++) sum[s] += us[5 * j + s];
        if (sum[j % 5] < 0) sink = 1;
      }
      sink = sink + sum[i % 5];
    }
    floor = std::min(floor, now() - t);
  }
  std::printf("%s %.3f ms, additions alone %.3f ms\n", best <= 6 * floor ? "ok" : "slow", best * 1e3, floor * 1e3);
  return best <= 6 * floor ? 0 : 1;
}

// Host check of the half-range maps (pass.h): for passes of random circuits
// and every size of the qubit set S, the enumerated tiles (or groups, for the
// register kernel) cover each entry with r & S <= c & S exactly once and no
// other; and the cut into stretches (plan_half) only uses qubits that every
// pass of a stretch allows.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <random>

#include "plan.h"

using namespace dmg;

static bool cover(int n, int L, const int32_t* hipos, int mhi, uint32_t mask) {
  HalfMap hm;
  build_half(n, L, hipos, mhi, mask, &hm);
  const uint64_t dim = 1ull << n;
  std::vector<uint8_t> seen(dim * dim, 0);
  for (uint64_t k = 0; k < hm.count; k++) {
    const uint64_t base = half_base(hm, k, L);
    for (int run = 0; run < (1 << mhi); run++) {
      uint64_t off = 0;
      for (int j = 0; j < mhi; j++) off |= (uint64_t)((run >> j) & 1) << hipos[j];
      for (uint64_t e = 0; e < (1ull << L); e++) {
        const uint64_t i = base + off + e;
        if (i >= dim * dim) return std::printf("entry %llu out of range\n", (unsigned long long)i), false;
        if (seen[i]++) return std::printf("entry %llu twice\n", (unsigned long long)i), false;
      }
    }
  }
  for (uint64_t i = 0; i < dim * dim; i++) {
    const uint32_t r = (uint32_t)(i & (dim - 1)), c = (uint32_t)(i >> n);
    if (seen[i] != ((r & mask) <= (c & mask))) return std::printf("entry (%u, %u) of set %x\n", r, c, mask), false;
  }
  return true;
}

static uint32_t subset(uint32_t allowed, int count, std::mt19937_64& rng) {
  uint32_t m = 0;
  while (count > 0 && allowed) {
    int q = (int)(rng() % 32);
    if (!((allowed >> q) & 1)) continue;
    m |= 1u << q;
    allowed &= ~(1u << q);
    count--;
  }
  return m;
}

int main() {
  std::mt19937_64 rng(11);
  int checked = 0, sizes[kHalfMaxS + 1] = {0};
  for (int s = 1; s <= kHalfMaxS; s++) {  // the pairs of a triangle, in any order
    const uint32_t B = 1u << s, inv = (65536 + B) / (B + 1);
    std::vector<uint8_t> seen(B * B, 0);
    for (uint32_t p = 0; p < B * (B + 1) / 2; p++) {
      uint32_t I, J;
      half_pair(p, s, inv, I, J);
      if (I > J || J >= B || seen[I * B + J]++) return std::printf("pair %u of s = %d\n", p, s), 1;
    }
  }
  for (int trial = 0; trial < 24; trial++) {
    const int n = 6 + trial % 4;  // 6..9 qubits
    std::vector<Basic> basics;
    for (int gi = 0; gi < 24; gi++) {
      GateRec g;
      std::memset(&g, 0, sizeof g);
      static const int ops[] = {0, 1, 2, 3, 8, 13, 16, 18, 20, 23, 26, 28};
      g.op = ops[rng() % (sizeof ops / sizeof ops[0])];
      std::vector<int> qs(n);
      for (int i = 0; i < n; i++) qs[i] = i;
      std::shuffle(qs.begin(), qs.end(), rng);
      for (int i = 0; i < gate_arity(g.op); i++) g.qb[i] = (uint32_t)qs[i];
      g.theta = 0.1 * (double)(rng() % 60);
      g.phi = 0.3;
      g.lambda = 0.1 * (double)(rng() % 60);
      decompose(g, basics);
    }
    for (int k = 1; k <= 4; k++) {
      const std::vector<PassSpec> specs = k == 1 ? plan_plain(basics) : plan_greedy(basics, k);
      std::vector<HalfCost> costs;
      for (size_t i = 0; i < specs.size(); i++) {
        const PassSpec& p = specs[i];
        std::vector<unsigned char> d(std::max(desc_size(p.K), std::max(tc_desc_bytes(4, 0), tc_desc_bytes(4, 2))));
        uint64_t ntiles = 0;
        int tile = 0;
        // tiled, tensor (7 - K free bits) and register geometries
        for (int kind = 0; kind < 3; kind++) {
          if (kind == 1 && !tc_eligible(p, n)) continue;
          if (kind == 2 && p.K != 1) continue;
          if (kind == 1) build_tc_desc(p, n, d.data(), nullptr, &ntiles, &tile, false, 0);
          else build_desc(p, n, d.data(), nullptr, &ntiles, &tile);
          const PassHeader& h = *reinterpret_cast<const PassHeader*>(d.data());
          const uint32_t allowed = half_allowed(h, p, n, kind == 2);
          if (kind == 0) costs.push_back({allowed, 2.0, 1.0 + (double)(rng() % 8), 64.0, 1.0});
          for (int t = 0; t < p.K; t++)
            if ((allowed >> p.q[t]) & 1) return std::printf("a target is allowed\n"), 1;
          if (!allowed || i % 5) continue;
          const uint32_t S = subset(allowed, 1 + (int)(rng() % kHalfMaxS), rng);
          const int32_t reg[2] = {p.q[0], p.q[0] + n};
          const bool ok = kind == 2 ? cover(n, 0, reg, 2, S) : cover(n, h.L, h.hipos, h.mhi, S);
          if (!ok) return std::printf("failed: n=%d K=%d kind %d\n", n, p.K, kind), 1;
          sizes[__builtin_popcount(S)]++;
          checked++;
        }
      }
      double gain = -1;
      const std::vector<uint32_t> S = plan_half(costs, 3.0, 5.0, &gain);
      if (S.size() != costs.size() || gain < 0) return std::printf("plan_half\n"), 1;
      for (size_t i = 0; i < S.size(); i++)
        if ((S[i] & ~costs[i].allowed) || __builtin_popcount(S[i]) > kHalfMaxS) return std::printf("set of pass %zu\n", i), 1;
    }
  }
  for (int s = 1; s <= 4; s++)
    if (!sizes[s]) return std::printf("no set of %d qubits checked\n", s), 1;
  if (checked < 100) return std::printf("too few maps checked: %d\n", checked), 1;
  std::printf("ok %d maps\n", checked);
  return 0;
}

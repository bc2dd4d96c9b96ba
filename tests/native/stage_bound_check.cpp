// Checks that the incidence records which a CTA stages are no more than the
// bound by which launch kinds are chosen (stage_records), so that no batch is
// refused for them after the choice: random networks with even and with very
// uneven degrees (a few hubs, power laws), clusters of 1 to 16 CTAs.
// Prints "bad=0" and exits 0 when the bound holds.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "mfg_mixed_order.h"
#include "mfg_mixed_place.cpp"

using namespace mfg;

int main() {
  std::mt19937 rng(13);
  int bad = 0;
  double closest = 0.0;
  for (int trial = 0; trial < 300; ++trial) {
    const int N = 40 + static_cast<int>(rng() % 2500);
    const int NF = std::max(1, N - static_cast<int>(rng() % (N / 3 + 1)));
    const double skew = trial % 3 == 0 ? 0.0 : (trial % 3 == 1 ? 1.5 : 4.0);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    auto pick = [&] { return std::min(N - 1, static_cast<int>(N * std::pow(u(rng), 1.0 + skew))); };
    std::vector<int2> conn;
    for (int j = 0; j < N; ++j)
      for (int k = 0; k < 2; ++k) {
        const int o = skew == 0.0 ? (j + 1 + static_cast<int>(rng() % 40)) % N : pick();
        if (o != j) conn.push_back(make_int2(j, o));
      }
    // the nodes in random order, so that hubs fall anywhere
    std::vector<int> at(N);
    for (int j = 0; j < N; ++j) at[j] = j;
    if (trial & 1) std::shuffle(at.begin(), at.end(), rng);
    for (int2& c : conn) c = make_int2(at[c.x], at[c.y]);
    const int E = static_cast<int>(conn.size());
    std::vector<int32_t> rowptr(N + 1, 0), inc(2 * E);
    for (const int2& c : conn) rowptr[c.x + 1]++, rowptr[c.y + 1]++;
    for (int j = 0; j < N; ++j) rowptr[j + 1] += rowptr[j];
    std::vector<int> fill(rowptr.begin(), rowptr.end() - 1);
    for (int e = 0; e < E; ++e) {
      inc[fill[conn[e].x]++] = (e << 1) | 0;
      inc[fill[conn[e].y]++] = (e << 1) | 1;
    }
    RveDesc d{};
    d.n_nodes = N;
    d.n_free = NF;
    d.n_fibers = E;
    for (int cl : {1, 2, 4, 8, 16}) {
      std::vector<int2> econn(E);
      std::vector<int32_t> icode(2 * E), mslot(E), gnode(N), mrowptr(N + 1);
      cluster_order(d, cl, true, true, conn, rowptr, inc, econn, icode, mslot, gnode, mrowptr);
      const int64_t n = sell_layout(d, cl, conn, rowptr, inc, gnode, 0, nullptr, nullptr, nullptr);
      std::vector<int2> nsell(N);
      std::vector<int32_t> ncode(n);
      std::vector<int64_t> nfib(n);
      sell_layout(d, cl, conn, rowptr, inc, gnode, 0, nsell.data(), ncode.data(), nfib.data());
      const int fchunk = (NF + cl - 1) / cl;
      std::vector<int64_t> first(cl, -1), count(cl, 0);
      for (int P = 0; P < NF; ++P) {
        const int o = P / fchunk;
        if (first[o] < 0) first[o] = nsell[P].x;
        count[o] = std::max<int64_t>(count[o], nsell[P].x + 32LL * (nsell[P].y - 1) + 1 - first[o]);
      }
      const int64_t most = *std::max_element(count.begin(), count.end());
      const int64_t bound = stage_records(d, cl, rowptr.data());
      closest = std::max(closest, static_cast<double>(most) / static_cast<double>(bound));
      if (most > bound && ++bad <= 10)
        std::printf("N=%d cl=%d: %lld records, bound %lld\n", N, cl, static_cast<long long>(most),
                    static_cast<long long>(bound));
    }
  }
  std::printf("closest %.3f bad=%d\n", closest, bad);
  return bad != 0;
}

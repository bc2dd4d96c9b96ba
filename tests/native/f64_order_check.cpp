// Checks the host-side order of the FP64 cluster solve (mfg_f64_order.h) on
// random networks, for clusters of 2 to 16 CTAs:
//  - the parts' nodes are a permutation of the RVE's, free nodes in falling
//    degree, every local slot below `slots` and named once per part;
//  - every fiber's ends decode to its end nodes, and every part has each
//    fiber of its free nodes among the first n_fib exactly once;
//  - every incidence names the k-th fiber and end of its node's CSR row;
//  - the fibers between two boundary nodes appear once over all parts.
// Prints "bad=0" and exits 0 when every check holds.
#include <algorithm>
#include <cstdio>
#include <random>
#include <set>
#include <vector>

#include "mfg_f64_order.h"

using namespace mfg;

int main() {
  std::mt19937 rng(5);
  int bad = 0;
  auto fail = [&](const char* what) {
    if (++bad <= 10) std::printf("fail: %s\n", what);
  };
  for (int trial = 0; trial < 60; ++trial) {
    const int N = trial < 20 ? 2 + static_cast<int>(rng() % 40) : 50 + static_cast<int>(rng() % 3000);
    const int NB = trial % 7 == 0 ? N : static_cast<int>(rng() % (N / 3 + 1)), NF = N - NB;
    std::vector<int2> conn;
    for (int j = 0; j < N; ++j)
      for (int k = 0; k < 2; ++k) {
        const int o = (j + 1 + static_cast<int>(rng() % std::min(40, N - 1))) % N;
        if (o != j) conn.push_back(make_int2(j, o));
      }
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
    for (int cl : {2, 4, 8, 16}) {
      F64Parts out;
      f64_parts(d, cl, conn.data(), rowptr.data(), inc.data(), out);  // at offset 0
      f64_parts(d, cl, conn.data(), rowptr.data(), inc.data(), out);  // and packed behind it
      if (static_cast<int>(out.part.size()) != 2 * cl) fail("part count");
      for (int copy = 0; copy < 2; ++copy) {
        const F64Part* part = &out.part[copy * cl];
        std::vector<int> seen(N, 0);
        std::multiset<int> between;
        auto decode = [&](int code) {
          const int o = code >> 24, li = code & 0xFFFFFF;
          if (o >= cl || li >= part[o].slots) return -1;
          const F64Part& p = part[o];
          if (li < p.fchunk) return li < p.n_free ? out.gnode[p.node_off + li] : -1;
          return li - p.fchunk < p.n_bnd ? out.gnode[p.node_off + p.n_free + li - p.fchunk] : -1;
        };
        for (int o = 0; o < cl; ++o) {
          const F64Part& p = part[o];
          if (p.slots != part[0].slots || p.fchunk != part[0].fchunk) fail("slots differ");
          std::set<int> need, have;
          for (int t = 0; t < p.n_free + p.n_bnd; ++t) {
            const int j = out.gnode[p.node_off + t];
            seen[j]++;
            if ((j < NF) != (t < p.n_free)) fail("segment");
            if (t >= p.n_free) continue;
            const int deg = rowptr[j + 1] - rowptr[j];
            if (t > 0) {
              const int i = out.gnode[p.node_off + t - 1];
              if (rowptr[i + 1] - rowptr[i] < deg) fail("degree order");
            }
            const int32_t* row = &out.rows[p.row_off + t];
            if (row[1] - row[0] != deg || row[0] < 0 || row[1] > p.n_inc) fail("row");
            for (int k = 0; k < deg; ++k) {
              const int code = out.inc[p.inc_off + row[0] + k], want = inc[rowptr[j] + k];
              need.insert(want >> 1);
              if ((code >> 1) >= p.n_fib || (code & 1) != (want & 1) ||
                  out.slot[p.fib_off + (code >> 1)] != (want >> 1))
                fail("incidence");
            }
          }
          if (o > 0 && p.row_off != part[o - 1].row_off + part[o - 1].n_free + 1) fail("row_off");
          for (int k = 0; k < p.n_len; ++k) {
            const int e = out.slot[p.fib_off + k];
            const int2 c = out.ends[p.fib_off + k];
            if (decode(c.x) != conn[e].x || decode(c.y) != conn[e].y) fail("ends");
            if (k < p.n_fib) {
              if (!have.insert(e).second) fail("fiber twice");
            } else {
              between.insert(e);
            }
          }
          if (need != have) fail("fibers of the free nodes");
        }
        for (int j = 0; j < N; ++j)
          if (seen[j] != 1) fail("nodes are not a permutation");
        for (int e = 0; e < E; ++e)
          if ((conn[e].x >= NF && conn[e].y >= NF) != (between.count(e) == 1) ||
              between.count(e) > 1)
            fail("fibers between boundary nodes");
      }
      if (out.inc.size() > 0 && out.part.back().inc_off + out.part.back().n_inc !=
                                    static_cast<int64_t>(out.inc.size()))
        fail("inc_off");
    }
  }
  std::printf("bad=%d\n", bad);
  return bad != 0;
}

// Orders an RVE in which one node has a fiber to every other (cluster_order,
// clusters of 8 and 16) within 256 MB of address space: the set-up's memory
// goes with the number of incidences, not with the widest row times the nodes.
// Prints "bad=0" and exits 0 when the order is a permutation that keeps each
// CTA's nodes.
#include <cstdio>
#include <vector>

#include <sys/resource.h>

#include "mfg_mixed_order.h"

using namespace mfg;

int main() {
  const int N = 48000, NF = N - 1000, E = N - 1 + N - 2;
  const rlimit limit{256u << 20, 256u << 20};
  if (setrlimit(RLIMIT_AS, &limit) != 0) return 2;
  std::vector<int2> conn;
  for (int j = 1; j < N; ++j) conn.push_back(make_int2(0, j));
  for (int j = 1; j + 1 < N; ++j) conn.push_back(make_int2(j, j + 1));
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
  int bad = 0;
  for (int cl : {8, 16}) {
    std::vector<int2> econn(E);
    std::vector<int32_t> icode(2 * E), mslot(E), gnode(N), mrowptr(N + 1);
    cluster_order(d, cl, true, true, conn, rowptr, inc, econn, icode, mslot, gnode, mrowptr);
    std::vector<char> seen(N, 0);
    const int fchunk = (NF + cl - 1) / cl;
    for (int P = 0; P < N; ++P) {
      const int j = gnode[P];
      bad += seen[j]++ != 0;
      bad += P < NF ? j >= NF || j / fchunk != P / fchunk : j != P;
    }
  }
  std::printf("bad=%d\n", bad);
  return bad != 0;
}

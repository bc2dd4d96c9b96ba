// Prints the placement of a batch (mfg_mixed_place.h, f64_cluster_size) for a
// test to look at. Input, as numbers: SMs, clusters of 1, 2, 4, 8 and 16 CTAs
// the device holds, max_cluster, serving layout, small solve, solves at once,
// number of RVEs; then per RVE its law, nodes, free nodes, fibers, steps and the
// degree of every free node. Output: "f64 <CTAs>", then a line per RVE with its
// launch kind's cluster size, whether fiber-centric, two copies, staged, split.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "mfg_f64_order.h"
#include "mfg_mixed_place.h"

using namespace mfg;

int main() {
  int sms, held[5], max_cluster, serving, small_solve, copies, n;
  if (std::scanf("%d %d %d %d %d %d %d %d %d %d %d", &sms, &held[0], &held[1], &held[2], &held[3],
                 &held[4], &max_cluster, &serving, &small_solve, &copies, &n) != 11)
    return 2;
  std::vector<RveDesc> desc(n);
  std::vector<int32_t> rowptr;
  for (RveDesc& d : desc) {
    d = RveDesc{};
    if (std::scanf("%d %d %d %d %d", &d.law, &d.n_nodes, &d.n_free, &d.n_fibers, &d.max_steps) != 5)
      return 2;
    d.row_off = static_cast<int64_t>(rowptr.size());
    rowptr.push_back(0);
    for (int j = 0; j < d.n_free; ++j) {
      int degree;
      if (std::scanf("%d", &degree) != 1) return 2;
      rowptr.push_back(rowptr.back() + degree);
    }
    rowptr.resize(d.row_off + d.n_nodes + 1, rowptr.back());
  }
  std::printf("f64 %d\n", f64_cluster_size(desc, held, copies));
  constexpr int smem_floats = kSmemBytesMixed / 4;
  std::vector<int> rve_q(n);
  for (int r = 0; r < n; ++r)
    rve_q[r] = bucket_of(desc[r], rowptr.data() + desc[r].row_off, smem_floats,
                         std::min(max_cluster, 8), serving, small_solve, 2);
  if (serving) serve_on_clusters(desc, rowptr, smem_floats, held[2], sms, rve_q);
  std::vector<std::vector<int32_t>> bucket(kBuckets);
  for (int r = 0; r < n; ++r) bucket[rve_q[r]].push_back(r);
  int clusters[kKinds], kind[kBuckets];
  for (int k = 0; k < kKinds; ++k) {
    int log2_cl = 0;
    while (1 << log2_cl < kKind[k].cl) ++log2_cl;
    clusters[k] = held[log2_cl];
  }
  for (int q = 0; q < kBuckets; ++q) {
    kind[q] = q;
    std::stable_sort(bucket[q].begin(), bucket[q].end(), [&](int32_t x, int32_t y) {
      return desc[x].n_fibers > desc[y].n_fibers;
    });
  }
  if (may_widen(bucket, sms, serving, copies))
    choose_kinds(desc, bucket, rowptr, smem_floats, max_cluster, small_solve == 2, clusters, sms,
                 copies, kind);
  for (int r = 0; r < n; ++r) {
    const BucketKind& k = kKind[kind[rve_q[r]]];
    std::printf("%d %d %d %d %d\n", k.cl, k.all, k.db, k.stage, k.split);
  }
  return 0;
}

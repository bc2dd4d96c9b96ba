// Placement of the mixed-precision RVEs (declared, with the rules, in
// mfg_mixed_place.h).
#include "mfg_mixed_place.h"

#include <algorithm>
#include <functional>
#include <queue>

#include "mumfim_gpu.h"

namespace mfg {

namespace {

// Incidence records that a CTA of a cluster of cl stages at most for its free
// nodes: their degrees, and what slices of 32 nodes as wide as their widest
// row add (the nodes are in falling degree within two groups, so a slice is
// no wider than the mean row of the one before it but for each group's first
// two).
int64_t stage_records(const RveDesc& d, int cl, const int32_t* rowptr) {
  const int NF = d.n_free, fchunk = (NF + cl - 1) / cl;
  int64_t most = 0;
  for (int lo = 0; lo < NF; lo += fchunk) {
    const int hi = std::min(NF, lo + fchunk);
    int widest = 0;
    for (int j = lo; j < hi; ++j) widest = std::max(widest, rowptr[j + 1] - rowptr[j]);
    most = std::max<int64_t>(most, rowptr[hi] - rowptr[lo] + 96LL * widest);
  }
  return most;
}

}  // namespace

bool holds(const BucketKind& k, const RveDesc& d, const int32_t* rowptr, int64_t smem_floats) {
  if (cluster_floats(d.n_nodes, d.n_free, d.n_fibers, k.cl, k.all && !k.nodal, k.db) >
      smem_floats / k.ng)
    return false;
  if (!k.stage) return true;
  const int nb = d.n_nodes - d.n_free, fchunk = (d.n_free + k.cl - 1) / k.cl;
  return stage_fits(even_slots(fchunk + (nb + k.cl - 1) / k.cl), fchunk, (nb + k.cl - 1) / k.cl,
                    stage_records(d, k.cl, rowptr), smem_floats);
}

int bucket_of(const RveDesc& d, const int32_t* rowptr, int smem_floats, int max_cluster,
              bool serving_layout, int small_solve, int rves_per_cta) {
  const bool fiber_small =
      small_solve == MFG_SMALL_FIBER_CENTRIC ||
      (small_solve == MFG_SMALL_AUTO && d.law == MFG_LAW_NONLINEAR);
  for (int q : kPref)
    if ((fiber_small || !kKind[q].all) && kKind[q].cl <= max_cluster &&
        !(serving_layout && kKind[q].cl == 2) && kKind[q].ng <= rves_per_cta &&
        holds(kKind[q], d, rowptr, smem_floats))
      return q;
  return kQRuntime;
}

namespace {

// ---- width of the size buckets ------------------------------------------------

// Time of a step of one RVE in launch kind k, in microseconds: fitted to
// batches of 1 to 304 RVEs of one size at every cluster size, as they run side
// by side. Linear law, nodes: us on 1, 2, 4, 8, 16 CTAs -- 1,000: 2.3, 2.3, 2.0,
// 2.0, -; 2,500: 6.3, 3.8, 2.6, 2.4, 2.0; 4,500: 9.9, 5.8, 3.2, 2.6, 2.3; 9,000:
// -, 11.5, 6.3, -, -; 20,000: (100 in global memory), -, 13, 7.0, 4.0.
// Nonlinear -- 1,000: 4.9, 3.8, 2.9, 2.6, -; 4,500: 16, 9.6, 5.7, 4.5, 3.6;
// 20,000: -, -, 21, 12, 7.4.
double step_us(const RveDesc& d, const BucketKind& k) {
  const bool nl = d.law == MFG_LAW_NONLINEAR;
  if (k.all) return k.ng == 2 ? 0.0014 * d.n_fibers + 1.5 : 0.0011 * d.n_fibers + 2.0;
  if (!k.nodal) return 0.002 * d.n_fibers;  // (part of) the state in global memory
  // barriers and the tail of a part, by cluster size (1, 2, 4, 8, 16): one
  // copy of the node records, two, and two with the read-only data staged
  constexpr double fixed[3][5] = {
      {1.2, 2.8, 3.5, 3.5, 4.5}, {1.2, 2.4, 2.3, 2.3, 1.8}, {0.6, 1.4, 1.2, 1.45, 1.6}};
  int log2_cl = 0;
  while (1 << log2_cl < k.cl) ++log2_cl;
  const bool split = k.split == kSplitNonlinear && nl && d.n_free <= k.cl * kSplitNodes;
  if (split) return 0.0019 * d.n_fibers / k.cl + (k.cl == 16 ? 2.0 : 1.9);
  const double per_fiber = nl ? (k.cl == 1 ? 0.0013 : 0.0015) : 0.0008;
  const double t =
      per_fiber * d.n_fibers / k.cl + fixed[k.db + k.stage][log2_cl] + (nl ? 0.9 : 0.0);
  // the nonlinear law along the longest row, however few nodes a part has: 48
  // RVEs of 150, 300, 450 nodes on 2 CTAs 3.8 us a step each; two to a CTA 2.5, 3.4, 4.2
  return nl && k.cl == 2 ? std::max(t, 3.8) : t;
}

// Time of `copies` solves of the batch with the buckets in these kinds: RVE
// after RVE, bucket by bucket with the largest clusters first and the longest
// first in a bucket, each onto the SMs that are free first. No more than
// clusters[k] of a kind run at once, whatever SMs are left beside them: 36 of
// 4 CTAs and 15 of 8 on 152 SMs, which a share of whole SMs a cluster (5 and
// 11) would take for 30 and 13 (36 RVEs of 19,500 nodes, then put on clusters
// of 8 in three waves: 22.0 us a step, on 4 in one wave: 13.0).
double batch_us(const std::vector<RveDesc>& desc, const std::vector<std::vector<int32_t>>& bucket,
                const int* kind, const int* clusters, int sms, int copies) {
  std::vector<int> order;
  for (int q = 0; q < kBuckets; ++q)
    if (!bucket[q].empty()) order.push_back(q);
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return kKind[kind[x]].cl > kKind[kind[y]].cl; });
  std::vector<double> sm(sms, 0.0);  // when each SM is free, ascending
  for (int q : order) {
    const BucketKind& k = kKind[kind[q]];
    const int share = std::min(k.cl, sms);
    const size_t most = static_cast<size_t>(std::max(clusters[kind[q]], 1));
    std::priority_queue<double, std::vector<double>, std::greater<double>> ends;
    const size_t n = bucket[q].size() * copies;
    for (size_t i = 0; i < n; i += k.ng) {
      const RveDesc& d = desc[bucket[q][i / copies]];
      // two RVEs side by side on a CTA take 1.4 times as long as one there
      const double t = step_us(d, k) * d.max_steps * (i + 1 < n && k.ng == 2 ? 1.4 : 1.0);
      double start = sm[share - 1];
      if (ends.size() == most) {  // one of the kind has to end first
        start = std::max(start, ends.top());
        ends.pop();
      }
      ends.push(start + t);
      // the SMs that come free last before then, so that the others stay free
      const auto hi = std::upper_bound(sm.begin(), sm.end(), start);
      sm.erase(hi - share, hi);
      sm.insert(std::upper_bound(sm.begin(), sm.end(), start + t), share, start + t);
    }
  }
  return sm.back();
}

}  // namespace

bool may_widen(const std::vector<std::vector<int32_t>>& bucket, int sms, bool serving_layout,
               int copies) {
  size_t rves = 0, ctas = 0;
  for (int q = 0; q < kBuckets; ++q) {
    rves += bucket[q].size();
    ctas += bucket[q].size() * copies * kKind[q].cl;
  }
  return !serving_layout &&
         (!bucket[kQRuntime].empty() ||
          (copies == 1 ? rves <= 8 * static_cast<size_t>(sms)
                       : 3 * ctas <= 2 * static_cast<size_t>(sms)));
}

void choose_kinds(const std::vector<RveDesc>& desc,
                  const std::vector<std::vector<int32_t>>& bucket,
                  const std::vector<int32_t>& rowptr, int smem_floats, int max_cluster,
                  bool keep_fiber_centric, const int* clusters, int sms,
                  int copies, int* kind) {
  auto fits = [&](int q, int k) {
    for (int32_t r : bucket[q])
      if (!holds(kKind[k], desc[r], rowptr.data() + desc[r].row_off, smem_floats)) return false;
    return true;
  };
  // Four lanes to a node where the bucket has a nonlinear RVE whose parts are
  // small enough (the kernel's linear steps are a tenth slower for it), or
  // where every RVE is linear in such parts (a kernel without the other passes).
  auto splits = [&](int q, int cl, int split) {
    bool some = false, all = true;
    for (int32_t r : bucket[q]) {
      const bool small = desc[r].n_free <= cl * kSplitNodes;
      some = some || (small && desc[r].law == MFG_LAW_NONLINEAR);
      all = all && small && desc[r].law != MFG_LAW_NONLINEAR;
    }
    return split == kSplitNonlinear ? some : all;
  };
  // the kind of cl CTAs for bucket q: staged, else two record copies, else one
  auto wider = [&](int q, int cl) {
    for (int level = 3; level >= 0; --level)
      for (int k = 0; k < kKinds; ++k)
        if (kKind[k].nodal && kKind[k].cl == cl &&
            (kKind[k].split != kSplitNone) + kKind[k].stage + kKind[k].db == level &&
            clusters[k] > 0 && fits(q, k) &&
            (kKind[k].split == kSplitNone || splits(q, cl, kKind[k].split)))
          return k;
    return -1;
  };
  // widen the bucket whose RVE takes longest, again and again; keep the best
  // state met (a state no better than the one before it may lead to one)
  int best[kBuckets], now[kBuckets];
  std::copy(kind, kind + kBuckets, best);
  std::copy(kind, kind + kBuckets, now);
  double t_best = batch_us(desc, bucket, kind, clusters, sms, copies);
  for (;;) {
    int q_long = -1;
    double longest = 0.0;
    for (int q = 0; q < kBuckets; ++q)
      for (int32_t r : bucket[q]) {
        const double t = step_us(desc[r], kKind[now[q]]) * desc[r].max_steps;
        if (t > longest) {
          longest = t;
          q_long = q;
        }
      }
    if (q_long < 0 || (kKind[now[q_long]].all && keep_fiber_centric)) break;
    int k = -1;
    for (int cl = 2 * kKind[now[q_long]].cl; k < 0 && cl <= max_cluster; cl *= 2)
      k = wider(q_long, cl);
    if (k < 0) break;
    now[q_long] = k;
    const double t = batch_us(desc, bucket, now, clusters, sms, copies);
    if (t < 0.97 * t_best) {  // a wider bucket has to pay
      t_best = t;
      std::copy(now, now + kBuckets, best);
    } else if (t > (kKind[kind[q_long]].all ? 1.6 : 1.15) * t_best) {
      break;  // (from fiber-centric the way to four lanes a node leads through 2 CTAs)
    }
  }
  std::copy(best, best + kBuckets, kind);
}

void serve_on_clusters(const std::vector<RveDesc>& desc, const std::vector<int32_t>& rowptr,
                       int smem_floats, int clusters, int sms, std::vector<int>& rve_q) {
  constexpr int kQCluster = 2, kQClusterDB = 1;
  static_assert(kKind[kQCluster].cl == kClusterServe && kKind[kQClusterDB].cl == kClusterServe,
                "bucket table");
  const size_t n = rve_q.size();
  // a wave that fills the CTAs several times over is better off on single ones
  if (clusters < 1 || n > 4 * static_cast<size_t>(clusters) * kClusterServe) return;
  std::vector<double> one(n), four(n);  // a request's time on one CTA and on a cluster
  std::vector<int> movable;
  std::vector<char> big(n, 0);  // solved on a cluster
  for (size_t r = 0; r < n; ++r) {
    // the serving kernels stage nothing and have no clusters of 8
    const int q = rve_q[r] == kQNodalStage ? kQNodalDB
                                           : (kKind[rve_q[r]].cl > kClusterServe ? kQRuntime : rve_q[r]);
    one[r] = step_us(desc[r], kKind[q]) * desc[r].max_steps * (kKind[q].ng == 2 ? 1.3 : 1.0);
    four[r] = step_us(desc[r], kKind[kQCluster]) * desc[r].max_steps;
    big[r] = kKind[q].cl == kClusterServe;
    if (kKind[q].cl == 1 && q != kQRuntime && four[r] < 0.8 * one[r] &&
        holds(kKind[kQCluster], desc[r], rowptr.data() + desc[r].row_off, smem_floats))
      movable.push_back(static_cast<int>(r));
  }
  std::stable_sort(movable.begin(), movable.end(), [&](int x, int y) { return one[x] > one[y]; });
  using Heap = std::priority_queue<double, std::vector<double>, std::greater<double>>;
  auto any_big = [&] { return std::find(big.begin(), big.end(), 1) != big.end(); };
  // end of a wave when `share` CTAs of a cluster take small requests at a time
  auto wave = [&](int share) {
    Heap by_cluster, by_cta;
    double end = 0.0;
    auto next = [&](Heap& heap, double time) {
      const double t = heap.top() + time;
      heap.pop();
      heap.push(t);
      end = std::max(end, t);
    };
    if (any_big()) {
      for (int c = 0; c < clusters; ++c) by_cluster.push(0.0);
      for (size_t r = 0; r < n; ++r)
        if (big[r]) next(by_cluster, four[r]);
      for (; !by_cluster.empty(); by_cluster.pop())
        for (int k = 0; k < share; ++k) by_cta.push(by_cluster.top());
    } else {
      for (int c = 0; c < sms; ++c) by_cta.push(0.0);
    }
    for (size_t r = 0; r < n; ++r)
      if (!big[r]) next(by_cta, one[r]);
    return end;
  };
  // time of a request of every RVE when requests never run out: the SMs' or,
  // since an RVE solves one request at a time, the RVEs' own
  auto saturated = [&] {
    double sm = 0.0, chain = 0.0;
    for (size_t r = 0; r < n; ++r) {
      sm += big[r] ? kClusterServe * four[r] : one[r];
      chain += big[r] ? four[r] : one[r];
    }
    return std::max(sm / (any_big() ? kClusterServe * clusters : sms), chain / n);
  };
  double best = 0.9 * wave(kClusterServe);
  const double spread = wave(1), busy = saturated();
  size_t take = 0, m = 0;
  while (m < movable.size()) {
    const size_t next = std::min(movable.size(), m + 1 + m / 3);
    for (; m < next; ++m) big[movable[m]] = 1;
    const double t = wave(kClusterServe);
    if (t < best && wave(1) <= spread && saturated() <= 1.05 * busy) {
      best = t;
      take = m;
    }
  }
  for (size_t k = 0; k < take; ++k) {
    const int r = movable[k];
    rve_q[r] = holds(kKind[kQClusterDB], desc[r], rowptr.data() + desc[r].row_off, smem_floats)
                   ? kQClusterDB
                   : kQCluster;
  }
}

}  // namespace mfg

// Host-side order of the FP64 cluster solve (declared, with what it writes,
// in mfg_f64_order.h).
#include "mfg_f64_order.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <queue>

namespace mfg {

void f64_parts(const RveDesc& d, int cl, const int2* conn, const int32_t* rowptr,
               const int32_t* inc, F64Parts& out) {
  const int N = d.n_nodes, NF = d.n_free, NB = N - NF, E = d.n_fibers;
  const int fchunk = std::max(1, (NF + cl - 1) / cl), bchunk = std::max(1, (NB + cl - 1) / cl);
  std::vector<uint8_t> owner(N);
  for (int j = 0; j < N; ++j)
    owner[j] = static_cast<uint8_t>(j < NF ? j / fchunk : (j - NF) / bchunk);
  // each part's nodes (free ones by falling degree) and every node's code
  std::vector<int32_t> code(N), count;
  const size_t node0 = out.gnode.size();
  out.gnode.resize(node0 + N);
  std::vector<size_t> first(cl + 1, node0);
  for (int o = 0; o < cl; ++o) {
    const int lo = std::min(NF, o * fchunk), hi = std::min(NF, lo + fchunk);
    const int b0 = std::min(NB, o * bchunk), b1 = std::min(NB, b0 + bchunk);
    int32_t* v = out.gnode.data() + first[o];
    int max_deg = 0;
    for (int j = lo; j < hi; ++j) max_deg = std::max(max_deg, rowptr[j + 1] - rowptr[j]);
    count.assign(max_deg + 2, 0);  // counting sort, falling degree
    for (int j = lo; j < hi; ++j) ++count[max_deg - (rowptr[j + 1] - rowptr[j]) + 1];
    for (int k = 0; k <= max_deg; ++k) count[k + 1] += count[k];
    for (int j = lo; j < hi; ++j) {
      const int t = count[max_deg - (rowptr[j + 1] - rowptr[j])]++;
      v[t] = j;
      code[j] = (o << 24) | t;
    }
    for (int q = b0; q < b1; ++q) {
      v[hi - lo + q - b0] = NF + q;
      code[NF + q] = (o << 24) | (fchunk + q - b0);
    }
    first[o + 1] = first[o] + (hi - lo) + (b1 - b0);
  }
  // each part's fibers: those that reach into another CTA, those inside,
  // those between two boundary nodes
  std::vector<std::vector<int32_t>> reach(cl), inside(cl), between(cl);
  for (int e = 0; e < E; ++e) {
    const int x = conn[e].x, y = conn[e].y, ox = owner[x], oy = owner[y];
    if (x >= NF && y >= NF) {
      between[owner[std::min(x, y)]].push_back(e);
    } else if (ox == oy) {
      inside[ox].push_back(e);
    } else {
      if (x < NF) reach[ox].push_back(e);
      if (y < NF) reach[oy].push_back(e);
    }
  }
  std::vector<int32_t> at(E);  // position of a fiber slot in the current part
  for (int o = 0; o < cl; ++o) {
    F64Part p{};
    p.n_free = std::min(NF, (o + 1) * fchunk) - std::min(NF, o * fchunk);
    p.n_bnd = static_cast<int32_t>(first[o + 1] - first[o]) - p.n_free;
    p.fchunk = fchunk;
    p.slots = fchunk + bchunk;
    p.node_off = static_cast<int64_t>(first[o]);
    p.row_off = static_cast<int64_t>(out.rows.size());
    p.inc_off = static_cast<int64_t>(out.inc.size());
    p.fib_off = static_cast<int64_t>(out.ends.size());
    int32_t k = 0;
    for (const auto* list : {&reach[o], &inside[o], &between[o]}) {
      if (list == &between[o]) p.n_fib = k;
      for (int e : *list) {
        at[e] = k++;
        out.ends.push_back(make_int2(code[conn[e].x], code[conn[e].y]));
        out.slot.push_back(e);
      }
    }
    p.n_len = k;
    for (int t = 0; t < p.n_free; ++t) {
      const int j = out.gnode[first[o] + t];
      out.rows.push_back(static_cast<int32_t>(static_cast<int64_t>(out.inc.size()) - p.inc_off));
      for (int q = rowptr[j]; q < rowptr[j + 1]; ++q)
        out.inc.push_back((at[inc[q] >> 1] << 1) | (inc[q] & 1));
    }
    p.n_inc = static_cast<int32_t>(static_cast<int64_t>(out.inc.size()) - p.inc_off);
    out.rows.push_back(p.n_inc);
    out.part.push_back(p);
  }
}

namespace {

// Time of a step of one RVE over CL = 2^k CTAs, in microseconds: the fibers'
// share (8 ns a fiber on one SM; a part also evaluates the fibers it shares, a
// surface term), and what does not shrink with CL. Measured, one RVE on 16
// CTAs: 3.7 us at 1,000 nodes, 9.7 at 4,500, 30 at 20,000; 36 RVEs of 4,500
// nodes on 4 CTAs each 28 us; on single CTAs 120 us alone on an SM, 178 us for
// two.
double f64_step_us(const RveDesc& d, int k) {
  const double cl = 1 << k, fibers = d.n_fibers / cl;
  if (k == 0) return 0.0080 * fibers + 2.0;  // as one of two RVEs on an SM
  const double shared = std::pow(std::max(1.0, d.n_nodes / cl), -1.0 / 3.0);
  return 0.0082 * fibers * (1.0 + shared) + 3.0;
}

}  // namespace

double f64_batch_us(const std::vector<RveDesc>& desc, int k, int clusters, int copies) {
  // longest first onto the cluster that is free first, as the kernel's queue does
  std::vector<double> t;
  t.reserve(desc.size() * copies);
  for (const RveDesc& d : desc) t.insert(t.end(), copies, f64_step_us(d, k) * d.max_steps);
  std::sort(t.begin(), t.end(), std::greater<double>());
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (int c = 0; c < std::max(1, clusters); ++c) free_at.push(0.0);
  // a single CTA alone on its SM does not fill it
  double end = k == 0 && !t.empty() ? 1.3 * t.front() : 0.0;
  for (double x : t) {
    const double at = free_at.top() + x;
    free_at.pop();
    free_at.push(at);
    end = std::max(end, at);
  }
  return end;
}

int f64_cluster_size(const std::vector<RveDesc>& desc, const int clusters[5], int copies) {
  int best = 0;
  double t_best = 0.0;
  for (int k = 0; k < 5; ++k) {
    if (clusters[k] < 1) continue;
    const double t = f64_batch_us(desc, k, clusters[k], copies);
    // a larger cluster has to be clearly faster
    if (k == 0 || t < 0.95 * t_best) {
      best = k;
      t_best = t;
    }
  }
  return 1 << best;
}

}  // namespace mfg

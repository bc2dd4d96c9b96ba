// Host-side order of the FP64 cluster solve (mfg_relax_f64.cu): an RVE split
// over the CTAs of a thread-block cluster. Built once per batch at set-up.
#ifndef MFG_F64_ORDER_H
#define MFG_F64_ORDER_H

#include <cstdint>
#include <vector>

#include "mfg_internal.h"

namespace mfg {

// One RVE's parts for clusters of cl CTAs, appended to the packed arrays.
//
// CTA o owns the free nodes [o fchunk, (o+1) fchunk) and the boundary nodes
// [o bchunk, (o+1) bchunk) of the RVE's storage order (both segments follow a
// Morton curve). Its nodes are listed by falling degree, so that the lanes of
// a warp gather rows of nearly the same length, then its boundary nodes. It
// evaluates every fiber that touches one of its free nodes -- a fiber between
// two CTAs is evaluated by both, so force vectors never leave a CTA -- the
// ones that reach into another CTA first; after them come the fibers between
// two boundary nodes it was given for the shortest length. A fiber's ends
// are (owner CTA << 24 | local node slot), local slots counting the owner's
// free nodes, then (from fchunk) its boundary nodes.
struct F64Parts {
  std::vector<F64Part> part;
  std::vector<int32_t> gnode;  // by node: id in the RVE's storage order
  std::vector<int32_t> rows;   // by free node (+1 per part): first incidence
  std::vector<int32_t> inc;    // (fiber of the part << 1) | end, ascending original fiber id
  std::vector<int2> ends;      // by fiber of the part
  std::vector<int32_t> slot;   // by fiber of the part: fiber slot in the RVE's storage order
};
void f64_parts(const RveDesc& d, int cl, const int2* conn, const int32_t* rowptr,
               const int32_t* inc, F64Parts& out);

// Shared-memory bytes a part cannot do without: two copies of its node
// positions and its force vectors.
inline int64_t f64_part_bytes(const F64Part& p) {
  return 48LL * p.slots + 24LL * p.n_fib;
}

// Cluster size for the FP64 solve of `copies` solves each of these RVEs at
// once, by the estimate below; `clusters[k]` is the number of clusters of 2^k
// CTAs the device holds at once (0: not available).
int f64_cluster_size(const std::vector<RveDesc>& desc, const int clusters[5], int copies);
// The estimate: time of the solves of the whole batch, all their steps, in
// clusters of 2^k CTAs, `clusters` at once.
double f64_batch_us(const std::vector<RveDesc>& desc, int k, int clusters, int copies);

}  // namespace mfg

#endif

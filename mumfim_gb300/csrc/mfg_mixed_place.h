// Placement of the mixed-precision RVEs (mfg_relax_mixed.cu): the launch kinds
// of the relaxation kernel, which of them hold an RVE, and the choice among
// those. Host code without a device call: the device's cluster counts come
// as arguments.
#ifndef MFG_MIXED_PLACE_H
#define MFG_MIXED_PLACE_H

#include <cstdint>
#include <vector>

#include "mfg_internal.h"

namespace mfg {

constexpr int kBuckets = 11;
constexpr int kMaxCluster = 16;
constexpr int kThreadsMixed = 1024;
constexpr int kSmemBytesMixed = 220 * 1024;
// Four lanes to a node: of the nonlinear RVEs of a bucket, or of every RVE of
// a bucket that is all linear and all in small parts.
enum { kSplitNone, kSplitNonlinear, kSplitLinear };
// How the RVEs of a size bucket are solved.
struct BucketKind {
  int cl;      // CTAs per cluster
  bool all;    // fiber-centric: force vectors in shared memory too
  bool nodal;  // node-centric solve (node state in shared memory)
  int ng;      // RVEs solved side by side by one CTA (fiber-centric, all on chip)
  bool db;     // node-centric with two copies of the node records
  bool stage;  // and the read-only data of the step in shared memory too
  int split = kSplitNone;  // and four lanes to a node (nodal_kick_split)
};
// Launch kinds: each bucket's own (the same index), then the wider clusters a
// bucket may take when the batch leaves SMs idle (choose_kinds).
constexpr int kKinds = 24;
constexpr BucketKind kKind[kKinds] = {
    {8, false, true, 1, false, false}, {4, false, true, 1, true, false},
    {4, false, true, 1, false, false}, {2, false, true, 1, true, false},
    {2, false, true, 1, false, false}, {1, false, true, 1, false, false},
    {1, false, true, 1, true, false},  {1, true, false, 1, false, false},
    {1, true, false, 2, false, false}, {1, false, false, 1, false, false},
    {1, false, true, 1, true, true},
    // wider
    {8, false, true, 1, true, false},  {16, false, true, 1, true, false},
    {16, false, true, 1, false, false}, {2, false, true, 1, true, true},
    {4, false, true, 1, true, true},   {8, false, true, 1, true, true},
    {16, false, true, 1, true, true},
    {4, false, true, 1, true, true, kSplitNonlinear},
    {8, false, true, 1, true, true, kSplitNonlinear},
    {16, false, true, 1, true, true, kSplitNonlinear},
    {4, false, true, 1, true, true, kSplitLinear},
    {8, false, true, 1, true, true, kSplitLinear},
    {16, false, true, 1, true, true, kSplitLinear}};
// Placement preference (bucket_of): the first bucket whose shared memory
// holds the RVE, else the run-time placement. At each cluster size two
// copies of the node records come first where they fit, on one CTA with the
// step's read-only data before without.
constexpr int kPref[] = {8, 7, 10, 6, 5, 3, 4, 1, 2, 0};
// The single-CTA buckets with an RVE order of their own, by kind.
constexpr int kQNodal1 = 5, kQNodalDB = 6, kQFiberAll = 7, kQFiberPair = 8, kQRuntime = 9,
              kQNodalStage = 10;
static_assert(kKind[kQNodal1].cl == 1 && kKind[kQNodal1].nodal, "bucket table");
static_assert(kKind[kQNodalDB].cl == 1 && kKind[kQNodalDB].db, "bucket table");
static_assert(kKind[kQNodalStage].cl == 1 && kKind[kQNodalStage].stage, "bucket table");
static_assert(!kKind[kQRuntime].all && !kKind[kQRuntime].nodal, "bucket table");
static_assert(kKind[kQFiberAll].cl == 1 && kKind[kQFiberAll].all, "bucket table");
static_assert(kKind[kQFiberPair].all && kKind[kQFiberPair].ng == 2, "bucket table");

// Clusters of the serving kernel.
constexpr int kClusterServe = 4;
// Lanes to a node in the split kinds, and the free nodes a CTA may have there.
constexpr int kLanes = 4;
constexpr int kSplitNodes = kThreadsMixed / kLanes;

// Node slots rounded up to an even count, so that an array of records after
// another starts on a 16-byte boundary.
__host__ __device__ inline int64_t even_slots(int64_t n) { return (n + 1) & ~static_cast<int64_t>(1); }

// Shared-memory floats per CTA of an RVE solved by CL CTAs: 9 per node slot
// (displacement hi, lo and velocity; ceil(NF/CL) free plus ceil(NB/CL)
// boundary slots), 15 with two copies of the node records, plus 4 per fiber
// slot (ceil(E/CL)) when the force vectors are kept in shared memory too
// (all: the fiber-centric single CTA).
__host__ __device__ inline int64_t cluster_floats(int n_nodes, int n_free, int n_fibers, int cl,
                                                  bool all, bool two_copies = false) {
  const int64_t nb = n_nodes - n_free;
  const int64_t cap = even_slots((static_cast<int64_t>(n_free) + cl - 1) / cl + (nb + cl - 1) / cl);
  const int64_t echunk = (static_cast<int64_t>(n_fibers) + cl - 1) / cl;
  return (two_copies ? 15 : 9) * cap + (all ? 4 * echunk : 0);
}

// First float of the staged read-only data behind two record copies and the
// velocities (16-byte aligned), and whether it fits: 16 bytes per incidence
// record, 16 per free node (row and mass), 24 per boundary node (RAMP).
__host__ __device__ inline int64_t stage_offset(int64_t slots) {
  return (15 * slots + 3) & ~static_cast<int64_t>(3);
}
__host__ __device__ inline bool stage_fits(int64_t slots, int64_t n_free, int64_t n_bnd,
                                           int64_t n_rec, int64_t smem_floats) {
  return stage_offset(slots) + 4 * n_rec + 4 * n_free + 6 * n_bnd <= smem_floats;
}

// Whether launch kind k holds an RVE in its CTAs' shared memory.
bool holds(const BucketKind& k, const RveDesc& d, const int32_t* rowptr, int64_t smem_floats);

// Bucket of an RVE: the smallest of one CTA or a cluster of 2, 4 or 8 CTAs
// whose shared memory holds its node state (node-centric solve; at that
// size with two copies of the node records where they fit), else one
// CTA that keeps what fits in shared memory and streams the rest from global
// memory (fiber-centric solve). Clusters of 8 are the last resort: with
// 220 KB per CTA only 15 of them (120 SMs) are resident at once, against 36
// clusters of 4 (144 SMs). Clusters above max_cluster CTAs are not used,
// nor clusters of 2 in the serving layout (the serving kernel solves in
// clusters of 4 only).
// With the fiber-centric small solve, RVEs whose whole state fits half a
// CTA's shared memory come first (two of them share a CTA, at most
// rves_per_cta), then those whose whole state fits one CTA; otherwise those
// buckets are skipped and every RVE whose node state fits takes the
// node-centric solve. small_solve (mfg_small_rve_solve) picks the solve;
// AUTO takes the fiber-centric one for RVEs on the nonlinear law, whose
// exponential the node-centric solve would evaluate at both ends of every
// fiber, and the node-centric one for the linear law, where it runs 2 %
// (500 - 1,300 nodes) to 37 % (1,300 - 3,300 nodes) faster.
int bucket_of(const RveDesc& d, const int32_t* rowptr, int smem_floats, int max_cluster,
              bool serving_layout, int small_solve, int rves_per_cta);

// Whether choose_kinds() is asked: not in the serving layout (its kernels solve
// in clusters of 4), and not for a batch that fills the GPU many times (not
// worth estimating). For several solves at once only where they leave a third of
// the SMs idle: their clusters wait for neighbouring SMs to fall free (six
// solves of 32 RVEs of 1,000 - 10,000 nodes, 200 steps: 4.2 ms widened, 3.7 not;
// of 8 RVEs of 500 - 20,000, 84 SMs of 152: 1.7 ms, 2.8 not).
bool may_widen(const std::vector<std::vector<int32_t>>& bucket, int sms, bool serving_layout,
               int copies);

// Widens buckets while the batch's estimated time falls: a batch that leaves
// SMs idle solves its RVEs on larger clusters than they need. Starts from
// each bucket's own kind in `kind`; RVEs in global memory (the run-time placement)
// go to clusters of 16 where those hold them. Bucket by bucket, so that a
// batch keeps one launch per size bucket.
void choose_kinds(const std::vector<RveDesc>& desc,
                  const std::vector<std::vector<int32_t>>& bucket,
                  const std::vector<int32_t>& rowptr, int smem_floats, int max_cluster,
                  bool keep_fiber_centric, const int* clusters, int sms,
                  int copies, int* kind);

// Serving layout: which of the RVEs that one CTA holds go to clusters of 4 all
// the same. A wave of requests, one per RVE, ends with its longest chain, and
// a single CTA takes two to three times as long for its RVE as a cluster, which
// takes up to 3.2 times the SM time for it. Three estimates, for the longest 0,
// 1, 2, 3, 4, 6, ... single-CTA RVEs moved:
//  - the wave with large requests taken first and each CTA free for small ones
//    has to be a tenth shorter;
//  - the wave with one CTA of a cluster at work on small requests must not be
//    longer: a cluster's CTAs that find no small request when they look wait
//    for the one that did, so requests that come one by one occupy a cluster
//    each (without clusters, all `sms` CTAs serve on their own);
//  - the time of a request of every RVE in a stream that never runs dry must not
//    grow by more than a twentieth.
// The best by the first is taken. Requests/s of a stream with three waves queued,
// and ms of two waves (200 steps), with every RVE on the smallest placement / by
// the first estimate alone / so:
//   150 RVEs of 3,000 - 6,000, linear  80,400, 7.3 / 42,200, 10.8 / 80,400, 7.3
//   36 of these                        18,500, 5.8 / 27,000, 4.0 / 27,000, 4.0
//   110 of 300 - 6,200, both laws      83,100, 9.5 / 58,800, 7.0 / 82,700, 9.5
//   96 of 500 - 20,000, both laws      31,900, 12.6 / 31,600, 11.3 / 31,300, 11.2
// Returns the bucket per RVE in rve_q.
void serve_on_clusters(const std::vector<RveDesc>& desc, const std::vector<int32_t>& rowptr,
                       int smem_floats, int clusters, int sms, std::vector<int>& rve_q);

}  // namespace mfg

#endif

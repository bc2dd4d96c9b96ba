// Plain FP64 relaxation kernel: one persistent CTA solves one RVE at a time.
//
// Restates, in one launch, the reference's affine predictor
// (src/mumfim/microscale/batched_analysis/BatchedFiberRVEAnalysisExplicitBase.h:16-57),
// volume update (same file :127-154), the three TeamOuterLoop kernels
// (src/mumfim/microscale/batched_analysis/BatchedFiberRVEAnalysisExplicitTeamOuterLoop.h:215-434)
// and the Cauchy stress (BatchedFiberRVEAnalysisExplicitBase.h:58-126).
//
// Bit-exactness with a serial run of the same algorithm:
//  - this file is compiled with --fmad=false and every expression keeps the
//    reference's operation order; quotients and square roots are correctly
//    rounded (mfg_exact.cuh, or the IEEE operations where it does not apply);
//  - nodal forces are gathered node by node over a CSR list of incident
//    fibers in ascending fiber id, which adds the per-fiber force vectors in
//    exactly the order the serial scatter f_int[n1] -= t; f_int[n2] += t
//    does, instead of the reference's nondeterministic global atomics;
//  - the stress is summed by six threads, one per Voigt component, in
//    boundary-list order.
// Only the residual norm uses a tree reduction; it decides when to stop and
// is compared against the tolerance, never written into the state.
//
// Step structure. The reference's step s is
//   kick(h_s) + drift | lengths | forces | kick(h_s)
// with a barrier between each. The trailing kick of step s and the leading
// kick + drift of step s+1 touch only node-local data, so they are fused into
// one node pass that starts by gathering the forces of step s:
//   node pass  : f = gather(nrm); v += h_s f/m; v += h_{s+1} f/m; x += 2h_{s+1} v
//   fiber pass : l = |x2 - x1|; T = law(l0, l); nrm = (x2 - x1) * (T / l)
// giving two block barriers per step.
//
// What bounds it: the FP64 pipe, one warp instruction in 19 cycles and SM, at
// 84 FP64 instructions a fiber and step with the general divisions and square
// root, a second quotient h f / m for the trailing kick and a minimum no step
// needed. Quotients, square roots and half of a fiber's products run on the
// integer units instead (mfg_exact.cuh), which idle otherwise: 24 FP64
// instructions a fiber, the same bits; 512 threads at 64 registers, two CTAs
// an SM, so that 32 warps keep both busy. 256 RVEs of 4,500 nodes: 4.4e9 ->
// 1.6e10 fiber-steps/s.
//
// A batch that leaves SMs idle runs with every RVE split over a cluster of
// 2 to 16 CTAs instead (relax_f64_cluster_kernel below).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

#include <cooperative_groups.h>

#include "mumfim_gpu.h"

#include "mfg_common.cuh"
#include "mfg_exact.cuh"
#include "mfg_internal.h"

namespace cg = cooperative_groups;

namespace mfg {
namespace {

constexpr int kThreadsF64 = 512;
constexpr int kSumThreads = 256;  // partial sums of the residual
// Whether the products of the length's squares and of the force vector run in
// integers. An FP64 product costs 19 cycles of the SM's pipe, an integer one 30
// issue slots, so it pays where warps are many. Fiber-steps/s without, with
// these, with the linear law's too, and with the nodes' too: 304 RVEs of 4,500
// nodes on single CTAs 1.20, 1.51, 1.54, 1.50e10, but 1.08, 1.26, 1.20, 1.18e10
// for 152 (one CTA an SM); 36 on clusters of 512 threads -, 28, 30, 31 us a step
// (34 with the force vector's alone). A small part's warps are few, and a step is
// a chain: 4.0 us with them at 512 threads for one RVE of 1,000 nodes, 3.7
// without at 256.
constexpr bool kIntF64 = true, kIntCluster = true, kIntSmall = false;

// Reaction law of one RVE with everything that does not depend on the fiber
// formed once, by the expressions the reference forms per fiber.
//
// Linear (BatchedFiberRVEAnalysisExplicitBase.h:155-172):
//   T = lr E A g,  g = 1/2 (lr^2 - 1),  lr = l / l0
// Nonlinear (NonlinearReaction::forceReaction().first, src/mumfim/microscale/
// FiberReactions.cc:16-71; compressive transition ratio 1.0,
// FiberNetworkIO_impl.h:35), with alpha = E A / B:
//   toe        alpha lr (e^(B g) - 1)
//   beyond it  m (lr - r) l0 + b at a transition ratio r (lt above, 1 below),
//              m = alpha / l0 ((1 + r^2 B) e^(B g_r) - 1), b the toe's force at r
struct LawF64 {
  bool nonlinear;
  bool exact;  // E A (half_E, below) and alpha (div_known) are far from underflow
  double E, A;
  double half_E;  // E / 2: the linear law's factor 1/2, moved to where it is exact (with `exact`)
  double alpha, B, lt, kt, bt, kc, bc;
};

__device__ __forceinline__ LawF64 make_law_f64(const RveDesc& d) {
  LawF64 L;
  L.nonlinear = d.law == 1;
  L.E = d.E;
  L.half_E = 0.5 * d.E;
  L.A = d.A;
  L.alpha = L.B = L.lt = L.kt = L.bt = L.kc = L.bc = 0.0;
  if (L.nonlinear) {
    const double cmp = 1.0;
    L.alpha = d.E * d.A / d.B;
    L.B = d.B;
    L.lt = d.lt;
    const double gt = 1.0 / 2.0 * (d.lt * d.lt - 1);
    const double gc = 1.0 / 2.0 * (cmp * cmp - 1);
    L.kt = (1 + d.lt * d.lt * d.B) * exp(d.B * gt) - 1;
    L.bt = L.alpha * d.lt * (exp(d.B * gt) - 1);
    L.kc = (1 + cmp * cmp * d.B) * exp(d.B * gc) - 1;
    L.bc = L.alpha * cmp * (exp(d.B * gc) - 1);
  }
  L.exact = in_range(d.E) && in_range(d.E * d.A) && (!L.nonlinear || in_range(L.alpha));
  return L;
}

// a b, in integers (mul_exact) when kInt.
template <bool kInt>
__device__ __forceinline__ double product(double a, double b) {
  if constexpr (kInt)
    return mul_exact(a, b);
  else
    return a * b;
}

// Force at length ratio lr of a fiber of reference length l0; alpha_l0 =
// alpha / l0 (nonlinear law only).
__device__ __forceinline__ double reaction_force(const LawF64& L, double lr, double l0,
                                                 double alpha_l0) {
  if (!L.nonlinear)
    return lr * L.half_E * L.A * (lr * lr - 1);
  if (lr > L.lt) return alpha_l0 * L.kt * (lr - L.lt) * l0 + L.bt;
  if (lr < 1.0) return alpha_l0 * L.kc * (lr - 1.0) * l0 + L.bc;
  const double gs = 1.0 / 2.0 * (lr * lr - 1);
  return L.alpha * lr * (exp(L.B * gs) - 1);
}

// Force vector d T / l of one fiber with end-to-end vector d, by the general
// operations: the numbers fiber_vector() does not take. Returns l.
__device__ __noinline__ double fiber_vector_general(const LawF64& L, const double d[3], double l0,
                                                    double n[3]) {
  const double l = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  const double lr = l / l0;
  const double T = L.nonlinear ? reaction_force(L, lr, l0, L.alpha / l0)
                               : lr * L.E * L.A * (0.5 * (lr * lr - 1));
  const double q = T / l;
  for (int k = 0; k < 3; ++k) n[k] = d[k] * q;
  return l;
}

// The same, with the square root and the quotients of mfg_exact.cuh (R0 =
// exact_reciprocal(l0), 0 to ask for the general operations): 16 FP64
// instructions on the linear law instead of 45 (10 with kInt), the same
// bits.
template <bool kInt>
__device__ __forceinline__ double fiber_vector(const LawF64& L, const double d[3], double l0,
                                               uint64_t R0, double n[3]) {
  const double s =
      product<kInt>(d[0], d[0]) + product<kInt>(d[1], d[1]) + product<kInt>(d[2], d[2]);
  if (L.exact && in_range(s) && R0 != 0) {
    double l;
    uint64_t R;
    if (sqrt_recip(s, rsqrt_start(root_operand(s)), l, R)) {
      const double T = reaction_force(L, div_known(l, l0, R0), l0,
                                      L.nonlinear ? div_known(L.alpha, l0, R0) : 0.0);
      const bool zero = is_zero(T);
      if (zero || in_range(T)) {
        const double q = zero ? T : div_root(T, l, R);
#pragma unroll
        for (int k = 0; k < 3; ++k) n[k] = product<kInt>(d[k], q);
        return l;
      }
    }
  }
  return fiber_vector_general(L, d, l0, n);
}

// x / m for a node's mass (R = exact_reciprocal(m), or 0): div_known() where
// it applies. The general division is a call: inlined, the compiler runs it
// ahead of the test on every node.
__device__ __noinline__ double general_quotient(double x, double m) { return x / m; }

__device__ __forceinline__ double over_mass(double x, double m, uint64_t R) {
  if (is_zero(x)) {
    if (R != 0) return x;  // else the mass may be zero: 0 / 0
  } else if (in_range(x) && R != 0) {
    return div_known(x, m, R);
  }
  return general_quotient(x, m);
}

// x with its sign flipped where `flip`; no FP64 instruction.
__device__ __forceinline__ double flip_sign(double x, bool flip) {
  return __hiloint2double(__double2hiint(x) ^ (flip ? 0x80000000 : 0), __double2loint(x));
}

struct RveView {
  const double *X0, *X1, *X2;
  double *x0, *x1, *x2, *u0, *u1, *u2, *v0, *v1, *v2;
  const double *m, *mc;
  const uint64_t* rm;
  const int2* conn;
  const double* l0;
  const uint64_t* rl0;
  double *n0, *n1, *n2;
  double *fi0, *fi1, *fi2;
  const int32_t* rowptr;
  const int32_t* inc;
  double* ramp;
};

__device__ __forceinline__ RveView make_view(const DevBatch& b, const RveDesc& d) {
  RveView r;
  const int64_t nt = b.nt, et = b.et, no = d.node_off, fo = d.fiber_off;
  r.X0 = b.X + no; r.X1 = b.X + nt + no; r.X2 = b.X + 2 * nt + no;
  r.x0 = b.x + no; r.x1 = b.x + nt + no; r.x2 = b.x + 2 * nt + no;
  r.u0 = b.u + no; r.u1 = b.u + nt + no; r.u2 = b.u + 2 * nt + no;
  r.v0 = b.v + no; r.v1 = b.v + nt + no; r.v2 = b.v + 2 * nt + no;
  r.fi0 = b.fint + no; r.fi1 = b.fint + nt + no; r.fi2 = b.fint + 2 * nt + no;
  r.m = b.m + no; r.rm = b.rm + no; r.mc = b.mc + no;
  r.conn = b.conn + fo;
  r.l0 = b.l0 + fo; r.rl0 = b.rl0 + fo;
  r.n0 = b.nrm + fo; r.n1 = b.nrm + et + fo; r.n2 = b.nrm + 2 * et + fo;
  r.rowptr = b.rowptr + d.row_off;
  r.inc = b.inc + d.inc_off;
  r.ramp = b.ramp + 6 * d.bnd_off;
  return r;
}

// f_int of node i: incident fiber vectors in ascending fiber id, subtracted at
// the fiber's first node and added at its second
// (BatchedFiberRVEAnalysisExplicitBase.h:246-251 in serial order). The first
// one is taken as it is: adding it to zero changes no bit but a zero's sign.
__device__ __forceinline__ void gather_fint(const RveView& r, int i, double& a0, double& a1,
                                            double& a2) {
  a0 = 0.0; a1 = 0.0; a2 = 0.0;
  const int pb = __ldg(r.rowptr + i), pe = __ldg(r.rowptr + i + 1);
  if (pb == pe) return;
  {
    const int code = __ldg(r.inc + pb);
    const int e = code >> 1;
    const bool neg = !(code & 1);
    a0 = flip_sign(r.n0[e], neg); a1 = flip_sign(r.n1[e], neg); a2 = flip_sign(r.n2[e], neg);
  }
  for (int p = pb + 1; p < pe; ++p) {
    const int code = __ldg(r.inc + p);
    const int e = code >> 1;
    const bool neg = !(code & 1);
    a0 = a0 + flip_sign(r.n0[e], neg);
    a1 = a1 + flip_sign(r.n1[e], neg);
    a2 = a2 + flip_sign(r.n2[e], neg);
  }
}

// Fiber pass: lengths, reaction force and per-fiber force vector
// (TeamOuterLoop.h:53-82 and BatchedFiberRVEAnalysisExplicitBase.h:203-252).
// Returns this thread's minimum length when kLen (every 100th step; an FP64
// minimum is an instruction of the pipe that bounds the kernel).
template <bool kLen>
__device__ __forceinline__ double fiber_pass(const RveView& r, const RveDesc& d, const LawF64& L) {
  double lmin = DBL_MAX;
  for (int e = threadIdx.x; e < d.n_fibers; e += kThreadsF64) {
    const int2 c = __ldg(r.conn + e);
    const double dv[3] = {r.x0[c.y] - r.x0[c.x], r.x1[c.y] - r.x1[c.x], r.x2[c.y] - r.x2[c.x]};
    double n[3];
    const double l = fiber_vector<kIntF64>(L, dv, __ldg(r.l0 + e), __ldg(r.rl0 + e), n);
    if (kLen) lmin = fmin(lmin, l);
    r.n0[e] = n[0];
    r.n1[e] = n[1];
    r.n2[e] = n[2];
  }
  return lmin;
}

// One node's trailing kick of the last step and leading kick of this one from
// its internal force a, in place on the velocity w
// (BatchedFiberRVEAnalysisExplicitBase.h:253-287, TeamOuterLoop.h:157-175).
// Between refreshes of the time step both half kicks add the same quotient
// h f / m, formed once
// (`same`).
__device__ __forceinline__ void kick(double a, double m, uint64_t rm, double mc, double h_prev,
                                     double h, bool first, bool same, double& w) {
  const double f = -(a + mc * w);  // f = -f_int - c m v
  const double q = over_mass(h * f, m, rm);
  if (!first) w += same ? q : over_mass(h_prev * f, m, rm);
  w += q;
}

// computeCauchyStress (BatchedFiberRVEAnalysisExplicitBase.h:58-126) and the
// status record, by one CTA. The sum over the boundary follows the
// reference's order, one thread per Voigt component; its terms are formed by
// the whole CTA, kTerms nodes at a time, in shared memory (6 kTerms doubles):
// six threads that load them one by one take about 0.3 us a boundary node.
// Reads x and f_int past the L1 cache: other CTAs of a cluster wrote them.
constexpr int kTerms = 128;

template <int NT>
__device__ void cauchy_stress(const DevBatch& b, const RunArgs& a, const RveDesc& d, int rve,
                              int status, int step, double residual, double* terms) {
  const int tid = threadIdx.x;
  const int64_t no = d.node_off, nt = b.nt;
  const int32_t* bo = b.bnd + d.bnd_off;
  const int nb = d.n_nodes - d.n_free;
  double s = 0.0;
  for (int q0 = 0; q0 < nb; q0 += kTerms) {
    const int n = min(kTerms, nb - q0);
    for (int t = tid; t < 6 * n; t += NT) {
      const int k = t / n, q = t - k * n;
      const int64_t i = no + bo[q0 + q];
      // component k: (i, j) index pair of the symmetric part x_i f_j
      const int ci = k < 3 ? k : (k == 3 ? 1 : 0);
      const int cj = k < 3 ? k : (k == 5 ? 1 : 2);
      const double xi = __ldcg(b.x + ci * nt + i), fj = __ldcg(b.fint + cj * nt + i);
      double v = xi * fj;
      if (k >= 3) v = 0.5 * (v + __ldcg(b.x + cj * nt + i) * __ldcg(b.fint + ci * nt + i));
      terms[k * kTerms + q] = v;
    }
    __syncthreads();
    if (tid < 6)
      for (int q = 0; q < n; ++q) s += terms[tid * kTerms + q];
    __syncthreads();
  }
  if (tid < 6) {
    s *= d.scale / b.vol[rve];
    a.sigma[6 * rve + tid] = s;
    if (a.update_coords) b.cur_stress[6 * rve + tid] = s;
    if (!isfinite(s)) status = 4;
  }
  // status word: any thread of the first warp that saw a non-finite stress
  const unsigned bad = __ballot_sync(0xffffffffu, tid < 32 && status == 4);
  if (tid == 0) {
    a.st_status[rve] = bad ? 4 : status;
    a.st_steps[rve] = step;
    a.st_residual[rve] = residual;
  }
  __syncthreads();
}

__device__ void solve_rve(const DevBatch& b, const RunArgs& a, int rve, double* red,
                          double* terms) {
  const RveDesc d = b.desc[rve];
  const RveView r = make_view(b, d);
  const LawF64 L = make_law_f64(d);
  const int N = d.n_nodes, NF = d.n_free;
  const int tid = threadIdx.x;
  const double* F = a.F + 9 * (a.n_F > 1 ? rve : 0);
  const bool ramp = d.mode == 1;
  double Fm[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Fm[k] = F[k];
  // updateVolume (BatchedFiberRVEAnalysisExplicit.h:271)
  if (a.update_coords && tid == 0) b.vol[rve] = jacobian(Fm) * b.vol[rve];

  // ---- prologue: predictor (RELAX), x = X + u, v = 0, RAMP increments ----
  for (int i = tid; i < N; i += kThreadsF64) {
    const double xo0 = r.x0[i], xo1 = r.x1[i], xo2 = r.x2[i];
    double up0 = r.u0[i], up1 = r.u1[i], up2 = r.u2[i];
    if (!ramp) {
      up0 = (Fm[0] - 1) * xo0 + (Fm[1] - 0) * xo1 + (Fm[2] - 0) * xo2 + up0;
      up1 = (Fm[3] - 0) * xo0 + (Fm[4] - 1) * xo1 + (Fm[5] - 0) * xo2 + up1;
      up2 = (Fm[6] - 0) * xo0 + (Fm[7] - 0) * xo1 + (Fm[8] - 1) * xo2 + up2;
    }
    const double xn0 = r.X0[i] + up0, xn1 = r.X1[i] + up1, xn2 = r.X2[i] + up2;
    r.x0[i] = xn0; r.x1[i] = xn1; r.x2[i] = xn2;
    r.v0[i] = 0.0; r.v1[i] = 0.0; r.v2[i] = 0.0;
    if (ramp && i >= NF) {
      double* rb = r.ramp + 6 * (i - NF);
      rb[0] = xn0; rb[1] = xn1; rb[2] = xn2;
      rb[3] = (Fm[0] - 1) * xn0 + (Fm[1] - 0) * xn1 + (Fm[2] - 0) * xn2;
      rb[4] = (Fm[3] - 0) * xn0 + (Fm[4] - 1) * xn1 + (Fm[5] - 0) * xn2;
      rb[5] = (Fm[6] - 0) * xn0 + (Fm[7] - 0) * xn1 + (Fm[8] - 1) * xn2;
    }
  }
  __syncthreads();

  // ---- RunInitialization: lengths, dt_crit, first forces -----------------
  double dt_crit = block_min<kThreadsF64>(fiber_pass<true>(r, d, L), red) / d.sound_speed;

  // ---- main loop ---------------------------------------------------------
  const int cap = d.max_steps;  // host resolves the default cap for RELAX
  int step = 0;
  double residual = 10.0;
  double h = d.crit * dt_crit * 0.5;  // TeamOuterLoop.h:345
  double h2 = 2 * h, h_prev = 0.0;
  double done = 0.0;  // (double)step, and the RAMP fraction's divisor
  const double cap_d = static_cast<double>(cap);
  int status = 0;
  for (;;) {
    // `step` steps are complete. Every UPDATE_FREQ steps the residual of the
    // last step's forces is refreshed (TeamOuterLoop.h:119-133); the loop
    // condition is the reference's (TeamOuterLoop.h:371) plus the step cap.
    const bool res_step = step > 0 && ((step - 1) % kUpdateFreq) == 0;
    if (res_step) {
      // shares through global memory (f_int's first component, unused at free
      // nodes), summed in the order of kSumThreads strided partial sums
      for (int i = tid; i < NF; i += kThreadsF64) {
        double a0, a1, a2;
        gather_fint(r, i, a0, a1, a2);
        r.fi0[i] = a0 * a0 + a1 * a1 + a2 * a2;
      }
      __syncthreads();
      double part = 0.0;
      if (tid < kSumThreads)
        for (int i = tid; i < NF; i += kSumThreads) part += r.fi0[i];
      residual = sqrt(block_sum<kThreadsF64>(part, red));
      if (!isfinite(residual)) {
        status = 4;  // MFG_E_NONFINITE
        break;
      }
    }
    if (!ramp && res_step && !(residual > d.tol)) break;
    if (step >= cap) break;  // RAMP: exactly max_steps steps; RELAX: cap reached
    const bool same = h == h_prev;
    // node pass: trailing kick of step-1, leading kick + drift of step
    for (int i = tid; i < NF; i += kThreadsF64) {
      double a0, a1, a2;
      gather_fint(r, i, a0, a1, a2);
      const double mass = __ldg(r.m + i), mc = __ldg(r.mc + i);
      const uint64_t rm = __ldg(r.rm + i);
      double w0 = r.v0[i], w1 = r.v1[i], w2 = r.v2[i];
      kick(a0, mass, rm, mc, h_prev, h, step == 0, same, w0);
      kick(a1, mass, rm, mc, h_prev, h, step == 0, same, w1);
      kick(a2, mass, rm, mc, h_prev, h, step == 0, same, w2);
      r.v0[i] = w0; r.v1[i] = w1; r.v2[i] = w2;
      r.x0[i] = r.x0[i] + h2 * w0;
      r.x1[i] = r.x1[i] + h2 * w1;
      r.x2[i] = r.x2[i] + h2 * w2;
    }
    if (ramp) {
      const double alpha = div_known(done + 1.0, cap_d, d.r_steps);
      for (int i = NF + tid; i < N; i += kThreadsF64) {
        const double* rb = r.ramp + 6 * (i - NF);
        r.x0[i] = rb[0] + alpha * rb[3];
        r.x1[i] = rb[1] + alpha * rb[4];
        r.x2[i] = rb[2] + alpha * rb[5];
      }
    }
    __syncthreads();
    h_prev = h;
    if (step % kUpdateFreq == 0) {
      dt_crit = block_min<kThreadsF64>(fiber_pass<true>(r, d, L), red) / d.sound_speed;
      h = d.crit * dt_crit * 0.5;
      h2 = 2 * h;
    } else {
      fiber_pass<false>(r, d, L);
      __syncthreads();
    }
    done += 1.0;
    ++step;
  }
  if (status == 0 && !ramp && residual > d.tol) status = 3;  // MFG_E_NOT_CONVERGED

  // ---- FinalizeData: boundary f_int, u = x - X -----------------------------
  for (int i = NF + tid; i < N; i += kThreadsF64) {
    double a0, a1, a2;
    gather_fint(r, i, a0, a1, a2);
    r.fi0[i] = a0; r.fi1[i] = a1; r.fi2[i] = a2;
  }
  if (a.update_coords) {
    for (int i = tid; i < N; i += kThreadsF64) {
      r.u0[i] = r.x0[i] - r.X0[i];
      r.u1[i] = r.x1[i] - r.X1[i];
      r.u2[i] = r.x2[i] - r.X2[i];
    }
  }
  __syncthreads();
  cauchy_stress<kThreadsF64>(b, a, d, rve, status, step, residual, terms);
}

__global__ void __launch_bounds__(kThreadsF64, 2) relax_f64_kernel(const DevBatch b, const RunArgs a) {
  __shared__ double red[kThreadsF64 / 32 + 1];
  __shared__ double terms[6 * kTerms];
  __shared__ int s_rve;
  for (;;) {
    if (threadIdx.x == 0) {
      const int w = atomicAdd(b.queue, 1);
      s_rve = w < b.n_rve ? b.order[w] : -1;
    }
    __syncthreads();
    const int rve = s_rve;
    __syncthreads();
    if (rve < 0) break;
    solve_rve(b, a, rve, red, terms);
  }
}

__global__ void __launch_bounds__(kThreadsF64, 2) server_f64_kernel(const DevBatch b,
                                                                 const ServerArgs sa) {
  __shared__ double red[kThreadsF64 / 32 + 1];
  __shared__ double terms[6 * kTerms];
  server_loop(sa, [&](const RunArgs& a, int rve) { solve_rve(b, a, rve, red, terms); });
}


// ---- one RVE over a cluster of CTAs ------------------------------------------
//
// For batches that leave SMs idle. One CTA solves an RVE at the FP64 rate of
// one SM: 64 us a step at 1,000 nodes, as the kernel was, with 151 SMs doing
// nothing; 3.7 us on 16. Here CL CTAs
// on CL SMs share it (f64_parts): each keeps two copies of its nodes'
// positions, their velocities and the force vectors of the fibers it
// evaluates in shared memory and reads other CTAs' positions through
// distributed shared memory. A fiber between two CTAs is evaluated by both,
// so force vectors stay local and a step has one cluster barrier (positions
// moved) and one block barrier (forces formed); the two position copies swap
// roles every step, so that no CTA writes what a slower one still reads.
// Every number is formed by the expressions and in the order of the single
// CTA: the same bits.
//
// The read-only data of the step (fiber ends and lengths, masses, rows) is
// copied into shared memory as far as it fits: the barrier's acquire drops
// the L1 cache, and a step of a small part is a chain of loads.

struct ClusterX {
  uint32_t base;     // shared address of the copy being read, in this CTA
  uint32_t stride;   // bytes from one component to the next
  __device__ __forceinline__ void load(int code, double x[3]) const {
    uint32_t p;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(p)
                 : "r"(base + 8u * (static_cast<uint32_t>(code) & 0xFFFFFFu)),
                   "r"(static_cast<uint32_t>(code) >> 24));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x[0]) : "r"(p));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x[1]) : "r"(p + stride));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x[2]) : "r"(p + 2 * stride));
  }
};

// Minimum over the cluster of a block-reduced value.
template <int CL>
__device__ double cluster_min(double part, double* slot) {
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x == 0) *slot = part;
  cl.sync();
  double t = DBL_MAX;
#pragma unroll
  for (int o = 0; o < CL; ++o) t = fmin(t, *cl.map_shared_rank(slot, o));
  cl.sync();
  return t;
}

// Copies n items to the shared memory at `at` when they fit below `end`, and
// returns where to read them.
template <int NT, typename T>
__device__ __forceinline__ const T* stage(const T* src, int n, unsigned char*& at,
                                          const unsigned char* end) {
  const size_t bytes = (static_cast<size_t>(n) * sizeof(T) + 15) & ~static_cast<size_t>(15);
  if (at + bytes > end) return src;
  T* dst = reinterpret_cast<T*>(at);
  for (int k = threadIdx.x; k < n; k += NT) dst[k] = src[k];
  at += bytes;
  return dst;
}

template <int CL, int NT, bool kInt>
__device__ void solve_rve_cluster(const DevBatch& b, const RunArgs& a, const F64Plan& plan,
                                  int rve, double* red, double* cred, double* alpha_s,
                                  double* terms,
                                  unsigned char* smem, int smem_bytes) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x;
  const RveDesc d = b.desc[rve];
  const F64Part part = plan.part[static_cast<int64_t>(rve) * CL + rank];
  const LawF64 L = make_law_f64(d);
  const int64_t no = d.node_off, nt = b.nt;
  const int NF = d.n_free, nfo = part.n_free, nbo = part.n_bnd, S = part.slots;
  const int n_own = nfo + nbo;
  const bool ramp = d.mode == 1;
  // shared memory: two copies of the positions, force vectors, velocities,
  // then the read-only data
  const unsigned char* end = smem + smem_bytes;
  double* xs = reinterpret_cast<double*>(smem);
  double* nrm = xs + 6 * S;
  unsigned char* at = reinterpret_cast<unsigned char*>(nrm + 3 * part.n_fib);
  at = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(at) + 15) & ~uintptr_t(15));
  double* vel = b.v + 3 * (no + rank * part.fchunk);  // 3 per own free node
  if (at + 24 * nfo + 16 <= end) {
    vel = reinterpret_cast<double*>(at);
    at += (24 * nfo + 15) & ~15;
  }
  double* rbs = b.ramp + 6 * (d.bnd_off + rank * (part.slots - part.fchunk));
  if (ramp && at + 48 * nbo <= end) {
    rbs = reinterpret_cast<double*>(at);
    at += 48 * nbo;
  }
  const int2* ends = stage<NT>(plan.ends + part.fib_off, part.n_len, at, end);
  const F64Len* len = stage<NT>(plan.len + part.fib_off, part.n_len, at, end);
  const int32_t* rows = stage<NT>(plan.rows + part.row_off, nfo + 1, at, end);
  const int32_t* inc = stage<NT>(plan.inc + part.inc_off, part.n_inc, at, end);
  const F64Mass* mass = stage<NT>(plan.mass + part.node_off, nfo, at, end);
  const int32_t* gnode = plan.gnode + part.node_off;

  const double* F = a.F + 9 * (a.n_F > 1 ? rve : 0);
  double Fm[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Fm[k] = F[k];
  if (a.update_coords && rank == 0 && tid == 0) b.vol[rve] = jacobian(Fm) * b.vol[rve];

  // ---- prologue, as solve_rve -------------------------------------------------
  for (int t = tid; t < n_own; t += NT) {
    const int64_t gi = no + gnode[t];
    const int li = t < nfo ? t : part.fchunk + (t - nfo);
    const double xo0 = b.x[gi], xo1 = b.x[nt + gi], xo2 = b.x[2 * nt + gi];
    double up0 = b.u[gi], up1 = b.u[nt + gi], up2 = b.u[2 * nt + gi];
    if (!ramp) {
      up0 = (Fm[0] - 1) * xo0 + (Fm[1] - 0) * xo1 + (Fm[2] - 0) * xo2 + up0;
      up1 = (Fm[3] - 0) * xo0 + (Fm[4] - 1) * xo1 + (Fm[5] - 0) * xo2 + up1;
      up2 = (Fm[6] - 0) * xo0 + (Fm[7] - 0) * xo1 + (Fm[8] - 1) * xo2 + up2;
    }
    const double xn0 = b.X[gi] + up0, xn1 = b.X[nt + gi] + up1, xn2 = b.X[2 * nt + gi] + up2;
    xs[li] = xn0; xs[S + li] = xn1; xs[2 * S + li] = xn2;
    if (t < nfo) {
      vel[t] = 0.0; vel[nfo + t] = 0.0; vel[2 * nfo + t] = 0.0;
    } else {
      // the boundary does not move in RELAX mode: both copies hold it
      xs[3 * S + li] = xn0; xs[4 * S + li] = xn1; xs[5 * S + li] = xn2;
      if (ramp) {
        double* rb = rbs + 6 * (t - nfo);
        rb[0] = xn0; rb[1] = xn1; rb[2] = xn2;
        rb[3] = (Fm[0] - 1) * xn0 + (Fm[1] - 0) * xn1 + (Fm[2] - 0) * xn2;
        rb[4] = (Fm[3] - 0) * xn0 + (Fm[4] - 1) * xn1 + (Fm[5] - 0) * xn2;
        rb[5] = (Fm[6] - 0) * xn0 + (Fm[7] - 0) * xn1 + (Fm[8] - 1) * xn2;
      }
    }
  }
  const uint32_t xs_addr = static_cast<uint32_t>(__cvta_generic_to_shared(xs));
  int cur = 0;  // the copy that holds the current positions
  ClusterX x{xs_addr, 8u * static_cast<uint32_t>(S)};

  // fiber pass over the part's fibers; with kLen also the shortest length,
  // for which the fibers between boundary nodes count too
  auto fiber_pass = [&](auto want_len) {
    constexpr bool kLen = decltype(want_len)::value;
    double lmin = DBL_MAX;
    const int n = kLen ? part.n_len : part.n_fib;
    for (int e = tid; e < n; e += NT) {
      const int2 c = ends[e];
      const F64Len q = len[e];
      double xa[3], xb[3], nv[3];
      x.load(c.x, xa);
      x.load(c.y, xb);
      const double dv[3] = {xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]};
      const double l = fiber_vector<kInt>(L, dv, q.l0, q.r, nv);
      if (kLen) {
        lmin = fmin(lmin, l);
        if (e >= part.n_fib) continue;
      }
      nrm[e] = nv[0];
      nrm[part.n_fib + e] = nv[1];
      nrm[2 * part.n_fib + e] = nv[2];
    }
    return lmin;
  };
  // component k of f_int of the own free node t: its fibers in ascending
  // original id
  auto gather = [&](int t, int k) {
    const int pb = rows[t], pe = rows[t + 1];
    const double* nk = nrm + k * part.n_fib;
    double f = 0.0;
    for (int p = pb; p < pe; ++p) {
      const int code = inc[p];
      const double v = flip_sign(nk[code >> 1], !(code & 1));
      f = p == pb ? v : f + v;
    }
    return f;
  };
  cluster.sync();
  double dt_crit = cluster_min<CL>(
                       block_min<NT>(fiber_pass(std::true_type{}), red), cred) /
                   d.sound_speed;

  // ---- main loop, as solve_rve --------------------------------------------------
  // Node pass: one thread per node and component, each component padded to
  // whole warps, then the boundary's. A warp's FP64 instruction occupies its
  // SM sub-partition's unit for 64 cycles, whatever it depends on, so a part
  // of 60 nodes (2 warps of whole nodes) would leave half of the SM idle.
  const int W = (nfo + 31) & ~31;
  const int cap = d.max_steps;
  int step = 0;
  double residual = 10.0;
  double h = d.crit * dt_crit * 0.5;  // TeamOuterLoop.h:345
  double h2 = 2 * h, h_prev = 0.0;
  int status = 0;
  // RAMP fraction of the next step, kept by the last warp
  const double cap_d = static_cast<double>(cap);
  double done = 1.0;
  if (tid == NT - 1) *alpha_s = div_known(done, cap_d, d.r_steps);
  __syncthreads();
  for (;;) {
    const bool res_step = step > 0 && ((step - 1) % kUpdateFreq) == 0;
    if (res_step) {
      // the nodes' shares go through global memory (f_int's first component,
      // unused at free nodes) and every CTA sums all of them in the order of
      // solve_rve
      for (int t = tid; t < nfo; t += NT) {
        const double f0 = gather(t, 0), f1 = gather(t, 1), f2 = gather(t, 2);
        b.fint[no + gnode[t]] = f0 * f0 + f1 * f1 + f2 * f2;
      }
      cluster.sync();
      double sum = 0.0;
      if (tid < kSumThreads)
        for (int i = tid; i < NF; i += kSumThreads) sum += __ldcg(b.fint + no + i);
      residual = sqrt(block_sum<NT>(sum, red));
      if (!isfinite(residual)) {
        status = 4;  // MFG_E_NONFINITE
        break;
      }
    }
    if (!ramp && res_step && !(residual > d.tol)) break;
    if (step >= cap) break;
    const bool same = h == h_prev;
    const double* xc = xs + 3 * S * cur;
    double* xn = xs + 3 * S * (1 - cur);
    const int n_items = 3 * W + (ramp ? 3 * nbo : 0);
    for (int item = tid; item < n_items; item += NT) {
      if (item < 3 * W) {
        const int k = item < W ? 0 : (item < 2 * W ? 1 : 2);
        const int t = item - k * W;
        if (t < nfo) {
          const F64Mass mm = mass[t];
          double w = vel[k * nfo + t];
          kick(gather(t, k), mm.m, mm.rm, mm.mc, h_prev, h, step == 0, same, w);
          vel[k * nfo + t] = w;
          xn[k * S + t] = xc[k * S + t] + h2 * w;
        }
      } else {
        const int q = item - 3 * W;
        const int k = q < nbo ? 0 : (q < 2 * nbo ? 1 : 2);
        const double* rb = rbs + 6 * (q - k * nbo) + k;
        xn[k * S + part.fchunk + (q - k * nbo)] = rb[0] + *alpha_s * rb[3];
      }
    }
    cur = 1 - cur;
    x.base = xs_addr + 24u * static_cast<uint32_t>(S) * static_cast<uint32_t>(cur);
    cluster.sync();
    if (ramp && tid == NT - 1) {
      done += 1.0;
      *alpha_s = div_known(done, cap_d, d.r_steps);
    }
    h_prev = h;
    if (step % kUpdateFreq == 0) {
      dt_crit = cluster_min<CL>(block_min<NT>(fiber_pass(std::true_type{}), red), cred) /
                d.sound_speed;
      h = d.crit * dt_crit * 0.5;
      h2 = 2 * h;
    } else {
      fiber_pass(std::false_type{});
      __syncthreads();
    }
    ++step;
  }
  if (status == 0 && !ramp && residual > d.tol) status = 3;  // MFG_E_NOT_CONVERGED

  // ---- FinalizeData: positions, u = x - X, boundary f_int, stress ------------------
  const double* xc = xs + 3 * S * cur;
  for (int t = tid; t < n_own; t += NT) {
    const int64_t gi = no + gnode[t];
    const int li = t < nfo ? t : part.fchunk + (t - nfo);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double xk = xc[k * S + li];
      b.x[k * nt + gi] = xk;
      if (a.update_coords) b.u[k * nt + gi] = xk - b.X[k * nt + gi];
    }
  }
  cluster.sync();
  // boundary rows from the positions just written (past the L1 cache): the
  // vectors of their fibers may be another CTA's
  for (int q = tid; q < nbo; q += NT) {
    const int i = gnode[nfo + q];
    const int32_t* row = b.rowptr + d.row_off + i;
    double f[3] = {0.0, 0.0, 0.0};
    for (int p = row[0]; p < row[1]; ++p) {
      const int code = b.inc[d.inc_off + p];
      const int64_t e = d.fiber_off + (code >> 1);
      const int2 c = b.conn[e];
      double dv[3], nv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
        dv[k] = __ldcg(b.x + k * nt + no + c.y) - __ldcg(b.x + k * nt + no + c.x);
      fiber_vector<false>(L, dv, b.l0[e], b.rl0[e], nv);
#pragma unroll
      for (int k = 0; k < 3; ++k) f[k] = f[k] + flip_sign(nv[k], !(code & 1));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) b.fint[k * nt + no + i] = f[k];
  }
  cluster.sync();
  if (rank == 0) cauchy_stress<NT>(b, a, d, rve, status, step, residual, terms);
}

template <int CL, int NT, bool kInt>
__global__ void __launch_bounds__(NT, 1)
relax_f64_cluster_kernel(const DevBatch b, const RunArgs a, const F64Plan plan) {
  extern __shared__ double4 smem_f64[];
  __shared__ double red[NT / 32 + 1];
  __shared__ double terms[6 * kTerms];
  __shared__ double cred, alpha;
  __shared__ int s_rve;
  cg::cluster_group cluster = cg::this_cluster();
  for (;;) {
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
      const int w = atomicAdd(b.queue, 1);
      s_rve = w < b.n_rve ? b.order[w] : -1;
    }
    cluster.sync();
    const int rve = *cluster.map_shared_rank(&s_rve, 0);
    cluster.sync();  // also: no CTA overwrites what a slower one still reads
    if (rve < 0) break;
    solve_rve_cluster<CL, NT, kInt>(b, a, plan, rve, red, &cred, &alpha, terms,
                          reinterpret_cast<unsigned char*>(smem_f64), plan.smem_bytes);
  }
}

// ---- set-up -------------------------------------------------------------------
//
// On the device, as the host would form them: the reciprocals on the host cores
// and their upload made a batch's creation a third longer (256 RVEs of 4,500
// nodes 44.8 ms, 32.8 with these; 64 of 500 - 20,000 on clusters 26.2, 21.0).

constexpr int kThreadsSetup = 256;

__global__ void f64_divisors_kernel(const DevBatch b, double* m, double* l0) {
  uint64_t* rm = reinterpret_cast<uint64_t*>(m + b.nt);
  uint64_t* rl0 = reinterpret_cast<uint64_t*>(l0 + b.et);
  for (int rve = blockIdx.y; rve < b.n_rve; rve += gridDim.y) {
    const RveDesc& d = b.desc[rve];
    const int first = blockIdx.x * kThreadsSetup + threadIdx.x, stride = gridDim.x * kThreadsSetup;
    for (int j = first; j < d.n_nodes; j += stride) {
      const int64_t i = d.node_off + j;
      rm[i] = exact_reciprocal(m[i]);
      m[2 * b.nt + i] = m[i] * d.c;
    }
    for (int e = first; e < d.n_fibers; e += stride) {
      const int64_t i = d.fiber_off + e;
      rl0[i] = exact_reciprocal(l0[i]);
    }
  }
}

__global__ void f64_plan_kernel(const DevBatch b, const F64Plan plan, F64Mass* mass, F64Len* len,
                                const int32_t* slot) {
  for (int q = blockIdx.y; q < b.n_rve * plan.cl; q += gridDim.y) {
    const F64Part& p = plan.part[q];
    const RveDesc& d = b.desc[q / plan.cl];
    const int first = blockIdx.x * kThreadsSetup + threadIdx.x, stride = gridDim.x * kThreadsSetup;
    for (int t = first; t < p.n_free + p.n_bnd; t += stride) {
      const int64_t i = d.node_off + plan.gnode[p.node_off + t];
      mass[p.node_off + t] = {b.m[i], b.rm[i], b.mc[i]};
    }
    for (int e = first; e < p.n_len; e += stride) {
      const int64_t i = d.fiber_off + slot[p.fib_off + e];
      len[p.fib_off + e] = {b.l0[i], b.rl0[i]};
    }
  }
}

using ClusterKernel = void (*)(DevBatch, RunArgs, F64Plan);

template <int NT, bool kInt>
ClusterKernel cluster_kernel_of(int cl) {
  switch (cl) {
    case 2: return relax_f64_cluster_kernel<2, NT, kInt>;
    case 4: return relax_f64_cluster_kernel<4, NT, kInt>;
    case 8: return relax_f64_cluster_kernel<8, NT, kInt>;
    case 16: return relax_f64_cluster_kernel<16, NT, kInt>;
    default: return nullptr;
  }
}

cudaError_t cluster_config(int cl, int threads, int grid, int smem_bytes, cudaStream_t s,
                           ClusterKernel* kernel, cudaLaunchConfig_t* cfg,
                           cudaLaunchAttribute* attr) {
  *kernel = threads == kF64ClusterThreads ? cluster_kernel_of<kF64ClusterThreads, kIntCluster>(cl)
                                          : cluster_kernel_of<kF64SmallThreads, kIntSmall>(cl);
  if (!*kernel) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(*kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kF64ClusterSmem);
  if (e == cudaSuccess && cl > 8)
    e = cudaFuncSetAttribute(*kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  *cfg = {};
  cfg->gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg->blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg->dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  cfg->stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cl);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return e;
}

}  // namespace

cudaError_t launch_f64_divisors(const DevBatch& b, double* m, double* l0, cudaStream_t s) {
  const dim3 grid(8, static_cast<unsigned>(std::min(b.n_rve, 65535)));
  f64_divisors_kernel<<<grid, kThreadsSetup, 0, s>>>(b, m, l0);
  return cudaGetLastError();
}

cudaError_t launch_f64_plan(const DevBatch& b, const F64Plan& plan, F64Mass* mass, F64Len* len,
                            const int32_t* slot, cudaStream_t s) {
  const dim3 grid(2, static_cast<unsigned>(
                         std::min<int64_t>(static_cast<int64_t>(b.n_rve) * plan.cl, 65535)));
  f64_plan_kernel<<<grid, kThreadsSetup, 0, s>>>(b, plan, mass, len, slot);
  return cudaGetLastError();
}

int relax_f64_max_clusters(int cl, int smem_bytes, int sms) {
  int n = 0;
  ClusterKernel kernel = nullptr;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg;
  cudaError_t e =
      cluster_config(cl, kF64ClusterThreads, cl * sms, smem_bytes, nullptr, &kernel, &cfg, attr);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();  // an unsupported size is no failure of the caller's
    return 0;
  }
  return n;
}

cudaError_t launch_relax_f64_cluster(const DevBatch& b, const RunArgs& a, const F64Plan& plan,
                                     int grid, cudaStream_t s) {
  ClusterKernel kernel = nullptr;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg;
  const cudaError_t e =
      cluster_config(plan.cl, plan.threads, grid, plan.smem_bytes, s, &kernel, &cfg, attr);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&cfg, kernel, b, a, plan);
}

cudaError_t launch_server_f64(const DevBatch& b, const ServerArgs& sa, int grid, cudaStream_t s) {
  server_f64_kernel<<<grid, kThreadsF64, 0, s>>>(b, sa);
  return cudaGetLastError();
}

cudaError_t launch_relax_f64(const DevBatch& b, const RunArgs& a, int threads, int grid,
                             cudaStream_t s) {
  (void)threads;
  relax_f64_kernel<<<grid, kThreadsF64, 0, s>>>(b, a);
  return cudaGetLastError();
}

int relax_f64_max_blocks_per_sm(int threads) {
  (void)threads;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, relax_f64_kernel, kThreadsF64, 0) !=
      cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

// ---- fixed-scratch variant ---------------------------------------------------
// The same relaxation kernel, with every scratch buffer it writes (per-fiber
// force vectors, internal forces, RAMP boundary data, the work counter and the
// per-RVE status words) carved out of one file-scope device array instead of
// buffers allocated with the batch. Every GPU that loads this library holds
// the array until the process exits; all calls on a device share it.
static __device__ __align__(256) unsigned char g_relax_scratch[MFG_NOALLOC_SCRATCH_BYTES];

namespace {

inline size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

}  // namespace

// Device address of the scratch array on the current device. The host-side
// symbol is only a stand-in for it. Looking the address up also loads this
// file's device code on the device if it is not loaded yet (CUDA loads
// modules lazily), and loading it is what reserves the array, so batch
// creation calls this once ahead of any solve. The lookup is repeated on
// every solve rather than cached, so an address never outlives the context
// it belongs to; once the module is loaded the lookup allocates nothing.
cudaError_t relax_f64_static_scratch_address(void** addr) {
  *addr = nullptr;
  return cudaGetSymbolAddress(addr, g_relax_scratch);
}

size_t relax_f64_static_scratch_bytes(const DevBatch& b, int64_t n_boundary_total) {
  const size_t R = static_cast<size_t>(b.n_rve);
  return align256(sizeof(int32_t)) + align256(R * sizeof(int32_t)) * 2 +
         align256(R * sizeof(double)) + align256(3 * static_cast<size_t>(b.et) * sizeof(double)) +
         align256(3 * static_cast<size_t>(b.nt) * sizeof(double)) +
         align256(6 * static_cast<size_t>(n_boundary_total > 0 ? n_boundary_total : 1) *
                  sizeof(double));
}

cudaError_t launch_relax_f64_static(const DevBatch& batch, const RunArgs& args, int grid,
                                    int64_t n_boundary_total, cudaStream_t s,
                                    StaticStatus* status) {
  if (relax_f64_static_scratch_bytes(batch, n_boundary_total) > MFG_NOALLOC_SCRATCH_BYTES)
    return cudaErrorInvalidValue;
  void* addr = nullptr;
  cudaError_t e = relax_f64_static_scratch_address(&addr);
  if (e != cudaSuccess) return e;
  unsigned char* base = static_cast<unsigned char*>(addr);
  const size_t R = static_cast<size_t>(batch.n_rve);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = base + off;
    off += align256(bytes);
    return p;
  };
  DevBatch b = batch;
  RunArgs a = args;
  b.queue = reinterpret_cast<int32_t*>(take(sizeof(int32_t)));
  a.st_status = reinterpret_cast<int32_t*>(take(R * sizeof(int32_t)));
  a.st_steps = reinterpret_cast<int32_t*>(take(R * sizeof(int32_t)));
  a.st_residual = reinterpret_cast<double*>(take(R * sizeof(double)));
  b.nrm = reinterpret_cast<double*>(take(3 * static_cast<size_t>(b.et) * sizeof(double)));
  b.fint = reinterpret_cast<double*>(take(3 * static_cast<size_t>(b.nt) * sizeof(double)));
  b.ramp = reinterpret_cast<double*>(
      take(6 * static_cast<size_t>(n_boundary_total > 0 ? n_boundary_total : 1) * sizeof(double)));
  // The work counter is the only scratch read before it is written.
  e = cudaMemsetAsync(b.queue, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return e;
  relax_f64_kernel<<<grid, kThreadsF64, 0, s>>>(b, a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  status->status = a.st_status;
  status->steps = a.st_steps;
  status->residual = a.st_residual;
  return cudaSuccess;
}

}  // namespace mfg

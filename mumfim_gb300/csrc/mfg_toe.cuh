// End of the nonlinear law's toe as a limit on lambda^2 (mfg_mixed_law.cuh).
// Compiles for the host too, where a test compares it with the square root.
#ifndef MFG_TOE_CUH
#define MFG_TOE_CUH

#include <cfloat>
#include <cmath>

namespace mfg {

// The largest number whose rounded square root is at most lt, for lt >= 1 (a
// transition ratio of any size: infinite past the largest float, and then so
// is the limit). A root rounds to lt or less exactly when it lies below the
// midpoint m of lt and the next float; a root is never on m (its square would
// have 50 bits). m has 25 bits, so m^2 is exact in FP64, and the limit is m^2
// rounded down. A closed form: a search in steps of one unit has no end where
// lt^2 or lt is infinite.
#ifdef __CUDACC__
__host__ __device__ __forceinline__
#else
inline
#endif
float toe_limit(float lt) {
  if (!(lt <= FLT_MAX)) return lt;
  const double m = 0.5 * (static_cast<double>(lt) + static_cast<double>(nextafterf(lt, INFINITY)));
  const double m2 = m * m;
  if (!(m2 < static_cast<double>(FLT_MAX))) return FLT_MAX;
  const float x = static_cast<float>(m2);
  return static_cast<double>(x) > m2 ? nextafterf(x, 0.f) : x;
}

}  // namespace mfg

#endif

// Compares mfg_mixed_law.cuh on the GPU with the IEEE operations, bit for bit:
//  - the square root and the reciprocals of tension_over_length(): every
//    lambda^2 of the two binades [1/4, 1) and [1, 4), all that occur up to a
//    power of four, through the branch below the toe (and the one above it);
//  - every Green strain of a sweep of representable numbers over all branches,
//    from subnormal to infinite, NaN included, for several laws.
// Prints "bad=0" and exits 0 when every result is the same.
#include <cstdint>
#include <cstdio>

#include "mfg_mixed_law.cuh"

using namespace mfg;

// the law as it is defined, by the general operations
__device__ float reference(const Law& L, float g, float rl0) {
  const float lam2 = fmaf(2.f, g, 1.f);
  if (g < 0.f) {
    const float lam = sqrtf(fmaxf(lam2, 0.f));
    const float lm1 = 2.f * g / (lam + 1.f);
    return L.ea * lm1 * rl0 / lam;
  }
  const float lam = sqrtf(lam2);
  if (lam > L.lt) {
    const float T = fmaf(L.Mt, lam - L.lt, L.bt);
    return T * rl0 / lam;
  }
  return L.ea_b * expm1f(L.B * g) * rl0;
}

__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}

__global__ void check(RveDesc d, unsigned long long* bad, float* first) {
  const Law L = make_law(d);
  const uint64_t n = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  // every 2^k-th bit pattern of g, and every one near 0 and the transition
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < (1ull << 28);
       i += n) {
    uint32_t bits = static_cast<uint32_t>(i << 4) + static_cast<uint32_t>(i % 13);
    if (i < (1u << 25))  // every g whose lambda^2 = 1 + 2 g lies in [1/4, 1)
      bits = __float_as_uint(-0.5f * (1.f - __uint_as_float(0x3E800000u + (bits >> 5))));
    else if (i < (1u << 26))  // every lambda^2 in [1, 4)
      bits = __float_as_uint(0.5f * (__uint_as_float(0x3F800000u + (bits >> 5) % 0x1000000u) - 1.f));
    const float g = __uint_as_float(bits);
    const float rl0 = 17.0f + static_cast<float>(i % 977);
    const float a = tension_over_length(L, g, rl0), b = reference(L, g, rl0);
    if (!same(a, b) && atomicAdd(bad, 1ull) == 0) {
      first[0] = g;
      first[1] = a;
      first[2] = b;
    }
  }
}

int main() {
  unsigned long long* bad;
  float* first;
  if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMalloc(&first, 12) != cudaSuccess) return 2;
  unsigned long long total = 0;
  const double laws[][4] = {{1.0, 3.14e-6, 4.0, 1.05}, {2.3, 2.2e-6, 1.0, 1.15},
                            {0.6, 5.0e-6, 9.7, 1.02},  {1.0e8, 7.9e-9, 2.0, 1.0},
                            {1.0, 1.0e-28, 3.0, 1.3}};
  for (const double* p : laws) {
    RveDesc d{};
    d.law = 1;
    d.E = p[0];
    d.A = p[1];
    d.B = p[2];
    d.lt = p[3];
    cudaMemset(bad, 0, 8);
    check<<<152 * 4, 256>>>(d, bad, first);
    unsigned long long h = 0;
    float f[3] = {0, 0, 0};
    if (cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(f, first, 12, cudaMemcpyDeviceToHost) != cudaSuccess)
      return 2;
    if (h) std::printf("law E=%g lt=%g: %llu differ, g=%a: %a, not %a\n", p[0], p[3], h, f[0], f[1], f[2]);
    total += h;
  }
  std::printf("bad=%llu\n", total);
  return total != 0;
}

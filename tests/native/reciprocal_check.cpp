// Compares exact_reciprocal() (mfg_exact.cuh) with a 128-bit division, on the
// host (g++) or, compiled as CUDA, on the device: significands at random, next to
// powers of two and with few bits set, over the divisors' exponents; and 0 for
// everything outside 2^-100 .. 2^100. Prints "bad=0" and exits 0 when all agree.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "mfg_exact.cuh"

using namespace mfg;

namespace {

uint64_t state = 29;
uint64_t next() {  // xorshift64*
  state ^= state >> 12;
  state ^= state << 25;
  state ^= state >> 27;
  return state * 2685821657736338717ull;
}

double make(uint64_t significand, int exponent) {
  return std::ldexp(static_cast<double>(significand & 0xFFFFFFFFFFFFFull | 1ull << 52), exponent - 52);
}

std::vector<double> divisors() {
  std::vector<double> d = {1.0, 2.0, 0x1p-100, 0x1p100, 3.0, 1.0 / 3.0};
  for (int k = 0; k < 4000; ++k)
    for (int e : {-100, -1, 0, 99}) {
      d.push_back(make(k, e));                  // just above a power of two
      d.push_back(make(0xFFFFFFFFFFFFFull - k, e));
    }
  for (int i = 0; i < 52; ++i)
    for (int j = 0; j < 52; ++j) d.push_back(make(1ull << i | 1ull << j, 7));
  for (int k = 0; k < 3000000; ++k) d.push_back(make(next(), static_cast<int>(next() % 200) - 100));
  return d;
}

#ifdef __CUDACC__
__global__ void reciprocals(const double* d, uint64_t* r, int n) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    r[k] = exact_reciprocal(d[k]);
}

bool run(const std::vector<double>& d, std::vector<uint64_t>& r) {
  double* dd = nullptr;
  uint64_t* dr = nullptr;
  const size_t n = d.size();
  bool ok = cudaMalloc(&dd, 8 * n) == cudaSuccess && cudaMalloc(&dr, 8 * n) == cudaSuccess &&
            cudaMemcpy(dd, d.data(), 8 * n, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    reciprocals<<<512, 256>>>(dd, dr, static_cast<int>(n));
    ok = cudaMemcpy(r.data(), dr, 8 * n, cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(dd);
  cudaFree(dr);
  return ok;
}
#else
bool run(const std::vector<double>& d, std::vector<uint64_t>& r) {
  for (size_t k = 0; k < d.size(); ++k) r[k] = exact_reciprocal(d[k]);
  return true;
}
#endif

}  // namespace

int main() {
  std::vector<double> d = divisors();
  const size_t inside = d.size();
  for (double x : {0.0, -0.0, -1.0, 0x1p-101, 0x1.8p100, 1e300, 5e-324, 1e-310, HUGE_VAL, -HUGE_VAL,
                   static_cast<double>(NAN)})
    d.push_back(x);
  std::vector<uint64_t> r(d.size());
  if (!run(d, r)) return 2;
  long bad = 0;
  for (size_t k = 0; k < d.size(); ++k) {
    uint64_t want = 0;
    if (k < inside) {
      const uint64_t D = significand(bits_of(d[k])) << 11;
      const unsigned __int128 q = (static_cast<unsigned __int128>(1) << 127) / D;
      want = q >> 64 ? ~0ull : static_cast<uint64_t>(q);
    }
    if (r[k] != want && ++bad <= 10)
      std::printf("%a: %llx, not %llx\n", d[k], static_cast<unsigned long long>(r[k]),
                  static_cast<unsigned long long>(want));
  }
  std::printf("bad=%ld\n", bad);
  return bad != 0;
}

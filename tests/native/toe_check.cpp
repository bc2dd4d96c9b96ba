// Checks toe_limit() (mfg_toe.cuh) on the host: the limit's rounded square
// root is at most the transition ratio and the next number's is not, for
// ratios over the whole range that a batch accepts (a double of at least 1,
// cast to float), those whose square or whose cast is infinite among them.
// Prints "bad=0" and exits 0 when every limit is right.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "mfg_toe.cuh"

int main() {
  long bad = 0;
  auto check = [&](double ratio) {
    const float lt = static_cast<float>(ratio), x = mfg::toe_limit(lt);
    const float next = std::nextafterf(x, INFINITY);
    const bool ok = std::isinf(lt) ? std::isinf(x)
                                   : std::isfinite(x) && std::sqrt(x) <= lt && std::sqrt(next) > lt;
    if (!ok && ++bad <= 10) std::printf("ratio %a: limit %a\n", ratio, x);
  };
  for (double r : {1.0, 1.0000001, 1.02, 1.05, 1.3, 2.0, 1e19, 1.8446742e19, 1.8446744e19, 2e19,
                   1e38, 3.4e38, static_cast<double>(FLT_MAX), 3.4028236e38, 1e39, 1e300, DBL_MAX})
    check(r);
  std::mt19937_64 rng(3);
  for (int k = 0; k < 4000000; ++k) {  // every binade from 1 to FLT_MAX
    const uint32_t bits = 0x3F800000u + static_cast<uint32_t>(rng() % (0x7F800000u - 0x3F800000u));
    float lt;
    std::memcpy(&lt, &bits, 4);
    check(lt);
  }
  for (uint32_t k = 0; k < 4096; ++k) {  // next to 1, to sqrt(FLT_MAX) and to FLT_MAX
    for (uint32_t b : {0x3F800000u + k, 0x5F7FFFFFu - 2048u + k, 0x7F7FFFFFu - k}) {
      float lt;
      std::memcpy(&lt, &b, 4);
      check(lt);
    }
  }
  std::printf("bad=%ld\n", bad);
  return bad != 0;
}

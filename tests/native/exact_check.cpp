// Checks mfg_exact.cuh on the host: div_known(), sqrt_recip() and div_root()
// against the general operations, on random operands and on operands next to a rounding
// boundary (where an approximate correction would round the wrong way).
//  - quotients x / d that lie k / (2^54 d) of an ulp from a midpoint, k odd and
//    small: Q d + k = 2^54 x is solved for the 54-bit midpoint Q (d odd);
//  - square roots next to a midpoint M + 1/2: M^2 + M + j = 0 mod 2^52 is
//    solved for M by Newton's iteration in 2-adic integers, so that
//    s = M^2 + M + j has 53 significant bits.
// The start of sqrt_recip() is perturbed by up to 2^-22, the error it allows.
// Prints "bad=0" and exits 0 when every result is the general operation's.
#include <cstdint>
#include <cstdio>
#include <random>

#include "mfg_exact.cuh"

using namespace mfg;

namespace {

std::mt19937_64 rng(11);
long bad = 0;

uint64_t inverse(uint64_t a) {  // of an odd a, mod 2^64
  uint64_t x = a;
  for (int i = 0; i < 6; ++i) x *= 2 - a * x;
  return x;
}

double random_significand() { return std::ldexp(static_cast<double>((rng() >> 11) | (1ull << 52)), -52); }

void check_div(double x, double d) {
  const uint64_t R = exact_reciprocal(d);
  if (R == 0 || !in_range(x) || div_known(x, d, R) != x / d || div_known(-x, d, R) != -(x / d)) {
    if (++bad <= 10) std::printf("div %a / %a\n", x, d);
  }
}

void check_mul(double a, double b) {
  const double want = a * b, got = mul_exact(a, b);
  if (bits_of(got) != bits_of(want) && !(want != want && got != got)) {
    if (++bad <= 10) std::printf("mul %a * %a = %a, not %a\n", a, b, want, got);
  }
}

// sqrt(s), and quotients by it: of f, and of an operand next to a midpoint
void check_sqrt(double s, double f) {
  const float off = (static_cast<float>(rng() % 2001) - 1000.f) / 1000.f;
  const float y0 = rsqrt_start(root_operand(s)) * (1.f + std::ldexp(off, -22));
  double l = 0.0;
  uint64_t R = 0;
  const bool ok = sqrt_recip(s, y0, l, R);
  int e;
  if (!in_range(s) || l != std::sqrt(s) || (!ok && std::frexp(l, &e) != 0.5)) {
    if (++bad <= 10) std::printf("sqrt %a: %a\n", s, l);
  }
  if (!ok) return;
  const uint64_t M = significand(bits_of(l));
  const int64_t k = 2 * static_cast<int64_t>(rng() % 16) - 15;
  double hard = f;
  if (M & 1) {
    const uint64_t Q = (0 - static_cast<uint64_t>(k)) * inverse(M) & ((1ull << 54) - 1);
    const unsigned __int128 P = static_cast<unsigned __int128>(Q) * M + static_cast<__int128>(k);
    const uint64_t X = static_cast<uint64_t>(P >> 54);
    if (X >> 52 == 1) hard = static_cast<double>(X);
  }
  for (double x : {f, -f, hard, l, 2.0 * l})
    if (div_root(x, l, R) != x / l) {
      if (++bad <= 10) std::printf("div_root %a / %a\n", x, l);
    }
}

}  // namespace

int main() {
  long n = 0;
  for (long t = 0; t < 4000000; ++t) {  // hard quotients
    const uint64_t M = (rng() >> 11) | (1ull << 52) | 1;
    const int64_t k = 2 * static_cast<int64_t>(rng() % 16) - 15;
    const uint64_t Q = (0 - static_cast<uint64_t>(k)) * inverse(M) & ((1ull << 54) - 1);
    if (!(Q >> 53)) continue;
    const unsigned __int128 P = static_cast<unsigned __int128>(Q) * M + static_cast<__int128>(k);
    const uint64_t X = static_cast<uint64_t>(P >> 54);
    if (X == 0 || X >> 53) continue;
    const int e = static_cast<int>(rng() % 140) - 70;
    check_div(std::ldexp(static_cast<double>(X), e), static_cast<double>(M));
    ++n;
  }
  for (int t = 0; t < 2000000; ++t) {
    check_div(std::ldexp(random_significand(), static_cast<int>(rng() % 1500) - 750),
              std::ldexp(random_significand(), static_cast<int>(rng() % 190) - 95));
    check_sqrt(std::ldexp(random_significand(), static_cast<int>(rng() % 1500) - 750), random_significand());
  }
  for (int t = 0; t < 4000000; ++t) {
    const double a = std::ldexp(random_significand(), static_cast<int>(rng() % 1200) - 600);
    const double b = std::ldexp(random_significand(), static_cast<int>(rng() % 1200) - 600);
    check_mul(a, t & 1 ? b : -b);
    // 27-bit operands: products halfway between two numbers among them
    check_mul(static_cast<double>(rng() >> 37), static_cast<double>(rng() >> 37));
    check_mul(static_cast<double>(rng() >> 11), static_cast<double>(rng() % 8));
  }
  const double odd_ones[] = {0.0, -0.0, 1.0, 1e-310, 1e-300, 1e300, HUGE_VAL, -HUGE_VAL, NAN};
  for (double a : odd_ones)
    for (double b : odd_ones) check_mul(a, b), check_mul(a, 1.5 * b), check_mul(3e8 * a, b);
  for (uint64_t k = 0; k < 2000; ++k) {  // next to powers of two
    check_sqrt(1.0 + static_cast<double>(k) * 0x1p-52, random_significand());
    check_sqrt(2.0 - static_cast<double>(k + 1) * 0x1p-52, random_significand());
    check_sqrt(4.0 - static_cast<double>(k + 1) * 0x1p-51, random_significand());
    check_div(2.0 - static_cast<double>(k + 1) * 0x1p-52, 2.0 - 0x1p-52);
    check_div(1.0 + static_cast<double>(k) * 0x1p-52, 2.0 - 0x1p-52);
    check_div(static_cast<double>(k + 1), 0x1p20);
    check_div(static_cast<double>(k + 1), 3.0 * static_cast<double>(k + 1));
  }
  for (int64_t j = -4000; j <= 4000; j += 2)  // hard square roots
    for (uint64_t root = 0; root < 2; ++root) {
      uint64_t M = root;
      for (int i = 0; i < 8; ++i)
        M -= (M * M + M + static_cast<uint64_t>(j)) * inverse(2 * M + 1);
      for (int bits = 52; bits <= 53; ++bits) {
        const uint64_t m = (M & ((1ull << bits) - 1)) | (bits == 52 ? 1ull << 52 : 0);
        if (m < (1ull << 52) || m >= (1ull << 53)) continue;
        unsigned __int128 S = static_cast<unsigned __int128>(m) * m + m + static_cast<__int128>(j);
        int shift = 0;
        while (!(S & 1)) S >>= 1, ++shift;
        if (S >> 53) continue;
        check_sqrt(std::ldexp(static_cast<double>(static_cast<uint64_t>(S)), shift), random_significand());
        check_sqrt(std::ldexp(static_cast<double>(static_cast<uint64_t>(S)), shift - 130), 1.0);
        ++n;
      }
    }
  std::printf("hard cases %ld bad=%ld\n", n, bad);
  return bad != 0 || n < 100000;
}

// Runs the core routines of fv2d_gb300/csrc/softfp.cuh, compiled for the
// host, against the host's binary64 division, square root and product:
//   softfp_harness N SEED ULPS
// N operand sets from SEED with the FP32 seeds moved by ULPS units in the
// last place; prints the number of mismatches and the first one of each.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../fv2d_gb300/csrc/softfp.cuh"

namespace sf = fv2d::softfp;

static uint64_t mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

// significand classes: random; few set bits; next to a power of two; runs of
// ones and zeros at the digit boundaries
static double operand(uint64_t r, uint64_t r2) {
  uint64_t f = r & 0xFFFFFFFFFFFFFull;
  switch (r2 & 7) {
    case 0: f &= 0xFF00000000000ull; break;
    case 1: f &= 0xFFFull; break;
    case 2: f = 0xFFFFFFFFFFFFFull - (f & 0xFFFull); break;
    case 3: f |= (1ull << 30) - 1; break;
    case 4: f &= ~((1ull << 29) - 1); break;
    default: break;
  }
  const int e = (r2 & 0x700) ? 1023 - 30 + (int)((r2 >> 16) % 61) : (int)((r2 >> 16) % 2047);
  return sf::from_bits((r & 0x8000000000000000ull) | ((uint64_t)e << 52) | f);
}

static bool same(double a, double b) { return sf::bits(a) == sf::bits(b) || (a != a && b != b); }

int main(int argc, char **argv) {
  if (argc != 4) return 2;
  const long long n = std::atoll(argv[1]);
  const uint64_t seed = std::strtoull(argv[2], nullptr, 10);
  sf::seed_ulps = std::atoi(argv[3]);
  long long bad[4] = {0, 0, 0, 0};
  for (long long i = 0; i < n; ++i) {
    const uint64_t r0 = mix(seed ^ (4 * i)), r1 = mix(seed ^ (4 * i + 1)), r2 = mix(seed ^ (4 * i + 2)),
                   r3 = mix(seed ^ (4 * i + 3));
    double a = operand(r0, r2);
    const double b = operand(r1, r3);
    const int near = (int)(r3 >> 60) & 3;  // dividends and radicands next to exact results
    const double nudge[4] = {0, 1, -1, 0};
    auto ulp = [&](double x) { return sf::from_bits(sf::bits(x) + (int64_t)nudge[near]); };
    if (near) a = ulp(a * b);
    if (!std::isfinite(a)) a = b;
    const double d[4] = {a / b, std::sqrt(std::fabs(a)), a * b, std::sqrt(ulp(b * b))};
    const double s[4] = {sf::div_rn(a, b), sf::sqrt_rn(std::fabs(a)), sf::mul_rn(a, b), sf::sqrt_rn(ulp(b * b))};
    for (int k = 0; k < 4; ++k)
      if (!same(d[k], s[k]) && ++bad[k] == 1) std::printf("op %d: %a %a -> %a, not %a\n", k, a, b, s[k], d[k]);
    // a reciprocal word formed on the host serves the device's quotients
    if (!same(a / b, sf::div_by(a, b, sf::recip_of_host(b))) && ++bad[0] == 1) std::printf("host word: %a %a\n", a, b);
  }
  std::printf("%lld\n", bad[0] + bad[1] + bad[2] + bad[3]);
  return 0;
}

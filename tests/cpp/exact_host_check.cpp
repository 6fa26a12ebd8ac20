// Host check of pieces of the exact FP64 physics (csrc/fvs_physics_exact.cuh,
// its device functions compiled as plain C++ without contraction) against the
// reference's expressions in IEEE arithmetic, bit for bit (any NaN equals any
// other): the half slopes of every limiter and the Roe mean's squared sound
// speed, over zeros of both signs, ties,
// subnormals, infinities, NaN, neighbours and random numbers of every exponent.
// Prints "bad 0" and exits 0 when all agree.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __dsub_rn(double a, double b) { return a - b; }

#include "fvs_physics_exact.cuh"

using namespace fvs;

namespace {

double Min(double a, double b) { return a < b ? a : b; }
double Max(double a, double b) { return a > b ? a : b; }

double Slope(int limiter, double sL, double sR) {
  if (limiter == exact::kVanLeer) {
    const double c = 2.0 * sL * sR;
    return c > 0.0 ? c / (sL + sR) : 0.0;
  }
  if (limiter == exact::kMinMod)
    return sR > 0 ? Max(0.0, Min(sL, sR)) : Min(0.0, Max(sL, sR));
  if (limiter == exact::kNoLimiter) return 0.5 * (sL + sR);
  return 0.0;
}

int Differ(double a, double b) {
  return !(ieee64::Bits(a) == ieee64::Bits(b) || (a != a && b != b));
}

int SlopesDiffer(double sL, double sR) {
  int bad = 0;
  for (int limiter = 0; limiter < 4; ++limiter)
    bad += Differ(exact::HalfSlopeOf(limiter, sL, sR), 0.5 * Slope(limiter, sL, sR));
  return bad;
}

int RoeDiffers(double u, double h) {
  const exact::Gas eq{1.4, 1.0 / (1.4 - 1.0)};
  return Differ(exact::RoeA2(eq, u, h), (eq.gamma - 1.0) * (h - 0.5 * u * u));
}

}  // namespace

int main() {
  const double inf = INFINITY, nan = NAN;
  const std::vector<double> special = {
      0.0, -0.0, 1.0, -1.0, 2.0, -2.0, 0.5, 1.0 + 0x1p-52, -1.0 - 0x1p-52, 3.0, -3.0, inf, -inf, nan,
      5e-324, -5e-324, 1e-310, -1e-310, 2.2250738585072014e-308, 1.7976931348623157e308,
      -1.7976931348623157e308, 0x1p511, 0x1p512, -0x1p512, 0x1p-510, 0x1p-511, -0x1p-537, 1e154};
  long bad = 0;
  for (double a : special)
    for (double b : special) bad += SlopesDiffer(a, b) + RoeDiffers(a, b);
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> u(-2.0, 2.0);
  for (int i = 0; i < 2000000; ++i) {
    const int span = i % 3 == 0 ? 1 : i % 3 == 1 ? 250 : 500;
    auto draw = [&] { return std::ldexp(u(rng), int(rng() % (2 * span + 1)) - span); };
    const double a = draw(), b = i % 8 ? draw() : a;
    bad += SlopesDiffer(a, b) + RoeDiffers(a, b);
  }
  std::printf("bad %ld\n", bad);
  return bad ? 1 : 0;
}

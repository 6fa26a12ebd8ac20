// fvs_physics_exact.cuh -- perfect-gas Euler physics in FP64 with the
// reference's exact operation order.
//
// Translation units that include this header are compiled with -fmad=false:
// every a*b+c stays a rounded multiply followed by a rounded add, division and
// sqrt are the IEEE correctly rounded ones, so the results are bit-identical
// to the reference's x86-64 SSE2 build (no FMA contraction).
//
// The kernels of this flavour are bound by the FP64 pipe, so whatever has the
// same bits elsewhere is taken off it: quotients and square roots run on the
// integer pipes (fvs_ieee64.cuh: 137 and 143 clocks of the FP64 pipe per warp
// become about 25 of the integer pipes), comparisons of signs and magnitudes
// are integer ones, and products with 0.5 and 2 are left out or done on the
// exponent.
//
// Reference functions restated here (maikel/FiniteVolumeSolver):
//   PerfectGas<D>::CompleteFromCons, Flux   src/equations/PerfectGas.cpp:25-124
//   EinfeldtSignalVelocities<PerfectGas<D>> src/equations/perfect_gas/EinfeldtSignalVelocities.hpp:64-97
//   Hll<...>::ComputeNumericFlux (array)    include/fub/flux_method/HllMethod.hpp:260-293
//   VanLeer / MinMod slopes                 include/fub/flux_method/MusclHancockMethod.hpp:92-187
//   MusclHancock::ComputeNumericFlux        include/fub/flux_method/MusclHancockMethod.hpp:419-485
#pragma once

#include <cstdint>

#include "fvs_ieee64.cuh"

namespace fvs {
namespace exact {

using ieee64::Div;
using ieee64::MakeDivisor;
using ieee64::Sqrt;

struct Gas {
  double gamma;
  double gamma_minus_1_inv;
};

template <int D> struct Complete {
  double rho;
  double m[D];
  double E;
  double p;
  double c;
};

// |m|^2 in the order of the reference's array path (Eigen default traversal
// splits the 3-term sum as m0^2 + (m1^2 + m2^2)).
template <int D> __device__ __forceinline__ double SquaredNorm(const double* m) {
  if constexpr (D == 1) {
    return m[0] * m[0];
  } else if constexpr (D == 2) {
    return m[0] * m[0] + m[1] * m[1];
  } else {
    return m[0] * m[0] + (m[1] * m[1] + m[2] * m[2]);
  }
}

__device__ __forceinline__ double PMin(double a, double b) { return ieee64::Less(a, b) ? a : b; }
__device__ __forceinline__ double PMax(double a, double b) { return ieee64::Less(b, a) ? a : b; }
// PMin(a, 0) and PMax(a, 0)
__device__ __forceinline__ double PMin0(double a) { return ieee64::Negative(a) ? a : 0.0; }
__device__ __forceinline__ double PMax0(double a) { return ieee64::Positive(a) ? a : 0.0; }

// CompleteFromCons: e_kin = 0.5*|m|^2/rho, p = (E - e_kin) / gamma_minus_1_inv,
// c = sqrt(gamma*p/rho).
template <int D>
__device__ __forceinline__ void CompleteFromCons(const Gas& eq, Complete<D>& q,
                                                 const double* u) {
  q.rho = u[0];
#pragma unroll
  for (int d = 0; d < D; ++d) q.m[d] = u[1 + d];
  q.E = u[1 + D];
  const ieee64::Divisor rho = MakeDivisor(q.rho);
  const double e_kin = Div<true>(SquaredNorm<D>(q.m), rho);
  const double e_int = q.E - e_kin;
  q.p = Div(e_int, eq.gamma_minus_1_inv);
  q.c = Sqrt(Div(eq.gamma * q.p, rho));
}

template <int D>
__device__ __forceinline__ void Flux(double* f, const Complete<D>& q, int dir) {
  const double velocity = Div(q.m[dir], q.rho);
  f[0] = q.m[dir];
#pragma unroll
  for (int d = 0; d < D; ++d) f[1 + d] = velocity * q.m[d];
  f[1 + dir] += q.p;
  f[1 + D] = velocity * (q.E + q.p);
}

template <int D>
__device__ __forceinline__ void AsCons(double* u, const Complete<D>& q) {
  u[0] = q.rho;
#pragma unroll
  for (int d = 0; d < D; ++d) u[1 + d] = q.m[d];
  u[1 + D] = q.E;
}

// (gamma - 1) (roeH - 0.5 roeU roeU), rounded as written in every translation
// unit, the half off the FP64 pipe
__device__ __forceinline__ double RoeA2(const Gas& eq, double roeU, double roeH) {
  return (eq.gamma - 1.0) * __dsub_rn(roeH, __dmul_rn(ieee64::HalfFactor(roeU), roeU));
}

template <int D>
__device__ __forceinline__ void Einfeldt(const Gas& eq, const Complete<D>& L,
                                         const Complete<D>& R, int dir,
                                         double& sL, double& sR) {
  const double rhoL = L.rho;
  const double rhoR = R.rho;
  const double sqRhoL = Sqrt(rhoL);
  const double sqRhoR = Sqrt(rhoR);
  const double oosqRhoSum = Div(1.0, sqRhoL + sqRhoR);
  const double uL = Div(L.m[dir], rhoL);
  const double uR = Div(R.m[dir], rhoR);
  const double roeU = (uL * sqRhoL + uR * sqRhoR) * oosqRhoSum;
  const double hL = Div(L.E + L.p, rhoL);
  const double hR = Div(R.E + R.p, rhoR);
  const double roeH = (hL * sqRhoL + hR * sqRhoR) * oosqRhoSum;
  const double roeA = Sqrt(RoeA2(eq, roeU, roeH));
  sL = PMin(uL - L.c, roeU - roeA);
  sR = PMax(roeU + roeA, uR + R.c);
}

template <int D>
__device__ __forceinline__ void HllFlux(const Gas& eq, double* nf,
                                        const Complete<D>& L,
                                        const Complete<D>& R, int dir) {
  constexpr int K = D + 2;
  double s0, s1;
  Einfeldt<D>(eq, L, R, dir, s0, s1);
  double fL[K], fR[K], qL[K], qR[K];
  Flux<D>(fL, L, dir);
  Flux<D>(fR, R, dir);
  AsCons<D>(qL, L);
  AsCons<D>(qR, R);
  const double sL = PMin0(s0);
  const double sR = PMax0(s1);
  const double sLsR = sL * sR;
  double ds = sR - sL;
  ds = ieee64::Positive(ds) ? ds : 1.0;
  const ieee64::Divisor dds = MakeDivisor(ds);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    nf[k] = Div(sR * fL[k] - sL * fR[k] + sLsR * (qR[k] - qL[k]), dds);
  }
}

// Per-cell quantities of the HLLE stable-dt estimate (Einfeldt speeds of the
// two cells of a face): sqrt(rho), normal velocity, enthalpy, sound speed.
struct CellWave {
  double sq;
  double u;
  double h;
  double a;
};

template <int D>
__device__ __forceinline__ CellWave MakeCellWave(const Gas& eq, const double* u,
                                                 int dir) {
  Complete<D> q;
  CompleteFromCons<D>(eq, q, u);
  CellWave w;
  const ieee64::Divisor rho = MakeDivisor(q.rho);
  w.sq = Sqrt(q.rho);
  w.u = Div(q.m[dir], rho);
  w.h = Div(q.E + q.p, rho);
  w.a = q.c;
  return w;
}

// max(0, |sL|, |sR|) of the face between two cells; the stable dt of the face
// is dx divided by it (Hll::ComputeStableDt, HllMethod.hpp:337-347).
__device__ __forceinline__ double FaceMaxSpeed(const Gas& eq, const CellWave& L,
                                               const CellWave& R) {
  const double oosqRhoSum = Div(1.0, L.sq + R.sq);
  const double roeU = (L.u * L.sq + R.u * R.sq) * oosqRhoSum;
  const double roeH = (L.h * L.sq + R.h * R.sq) * oosqRhoSum;
  const double roeA = Sqrt(RoeA2(eq, roeU, roeH));
  const double sL = PMin(L.u - L.a, roeU - roeA);
  const double sR = PMax(roeU + roeA, R.u + R.a);
  return PMax(PMax(0.0, fabs(sL)), fabs(sR));
}

// VanLeer, MinMod, NoLimiter (the central slope, unlimited) and NoGradient
// (slope 0) -- include/fub/flux_method/MusclHancockMethod.hpp:31-187.
enum Limiter : int { kVanLeer = 0, kMinMod = 1, kNoLimiter = 2, kNoGradient = 3 };

// Half the limited slope, what the predictor adds and subtracts.  Van Leer:
// 0.5 ((2 sL sR) / (sL + sR)) has the bits of (sL sR) / (sL + sR) unless the
// product or the sum leaves the range of ieee64's quotients.
__device__ __forceinline__ double HalfSlopeOf(int limiter, double sL, double sR) {
  if (limiter == kVanLeer) {
    const double c = sL * sR;
    const bool pos = ieee64::Positive(c);
    const ieee64::Divisor sum = MakeDivisor(pos ? sL + sR : 1.0);
    double hs = Div(c, sum);
    hs = pos ? hs : 0.0;
    const uint32_t span = ieee64::Span(ieee64::Hi(c));
    if ((span > sum.span ? span : sum.span) >= ieee64::kSpan && !ieee64::IsZero(sL) &&
        !ieee64::IsZero(sR)) {
      const double c2 = 2.0 * sL * sR;
      hs = 0.5 * ((c2 > 0.0) ? ieee64::IeeeDiv(c2, sL + sR) : 0.0);
    }
    return hs;
  }
  if (limiter == kMinMod) return 0.5 * ieee64::MinMod(sL, sR);
  if (limiter == kNoLimiter) return 0.5 * (0.5 * (sL + sR));
  return 0.0;
}

__device__ __forceinline__ double HalfSlope(int limiter, double qL, double qM, double qR) {
  return HalfSlopeOf(limiter, qM - qL, qR - qM);
}

// MUSCL-Hancock predictor of one cell: the Hancock-evolved states at its left
// face (recL, the reference's rec_[1] when the cell is stencil[2]) and at its
// right face (recR, rec_[0] when the cell is stencil[1]).  Computing both once
// per cell gives bit-identical face states to the reference, which computes
// each cell's predictor twice (once for each of its faces).
// From the cell's state and its differences to the two neighbours.
template <int D>
__device__ __forceinline__ void MusclPredictDiff(const Gas& eq, Complete<D>& recL,
                                                 Complete<D>& recR, const double* q1,
                                                 const double* sL, const double* sR, int limiter,
                                                 double lambda_half, int dir) {
  constexpr int K = D + 2;
  double uL[K], uR[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double hs = HalfSlopeOf(limiter, sL[k], sR[k]);
    uL[k] = q1[k] - hs;
    uR[k] = q1[k] + hs;
  }
  Complete<D> qL, qR;
  CompleteFromCons<D>(eq, qL, uL);
  CompleteFromCons<D>(eq, qR, uR);
  double fL[K], fR[K];
  Flux<D>(fL, qL, dir);
  Flux<D>(fR, qR, dir);
  double a[K], b[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double df = fL[k] - fR[k];
    b[k] = uR[k] + lambda_half * df;
    a[k] = uL[k] + lambda_half * df;
  }
  CompleteFromCons<D>(eq, recR, b);
  CompleteFromCons<D>(eq, recL, a);
}

template <int D>
__device__ __forceinline__ void MusclPredictBoth(const Gas& eq, Complete<D>& recL,
                                                 Complete<D>& recR, const double* q0,
                                                 const double* q1, const double* q2, int limiter,
                                                 double lambda_half, int dir) {
  constexpr int K = D + 2;
  double sL[K], sR[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    sL[k] = q1[k] - q0[k];
    sR[k] = q2[k] - q1[k];
  }
  MusclPredictDiff<D>(eq, recL, recR, q1, sL, sR, limiter, lambda_half, dir);
}

}  // namespace exact
}  // namespace fvs

// fvs_kernels_hllem.cu -- the HLLEM family's sweeps and stable dt with the
// reference's exact FP64 arithmetic (compiled with -fmad=false, like
// fvs_kernels_exact.cu).
#include "fvs_hllem.cuh"
#include "fvs_internal.h"
#include "fvs_physics_exact.cuh"
#include "fvs_policy_exact.cuh"
#include "fvs_recon_hllem.cuh"
#include "fvs_stable.cuh"
#include "fvs_sweep.cuh"

namespace fvs {

// HLLEM sweeps: the marching sweep with Hllem<PerfectGas, Larrouturou> as
// the face flux and its stable-dt speed as the CFL check (fvs_hllem.cuh),
// after one of four reconstructions: none (first order), MUSCL-Hancock of
// the conservative variables, the characteristic or the primitive
// reconstruction of the perfect gas (fvs_recon_hllem.cuh).
template <int D> struct HllemWave {
  exact::Complete<D> q;
  int dir;
};

enum HllemRecon : int { kReconNone = 0, kReconCons = 1, kReconChar = 2, kReconPrim = 3 };

template <int D, int kRecon> struct HllemPolicyT {
  using Real = double;
  static constexpr bool kWarpX = false;
  static constexpr int kMinBlocks = 1;
  static constexpr int kLaneBlocks = 3;
  static constexpr bool kHllemCfl = true;  // CFL speeds screened in FP32 (HllemScreen)
  using Gas = exact::Gas;
  using Rec = exact::Complete<D>;
  using Wave = HllemWave<D>;
  using Stats = NoStats;
  static __device__ __forceinline__ Gas MakeGas(double gamma) {
    return ExactPolicy<D>::MakeGas(gamma);
  }
  static __device__ __forceinline__ Gas MakeGasFor(const SweepArgs& a) { return MakeGas(a.gamma); }
  static __device__ __forceinline__ void ToCell(double* c, const double* u) {
#pragma unroll
    for (int k = 0; k < D + 2; ++k) c[k] = u[k];
  }
  static __device__ __forceinline__ void Predict(const Gas& eq, Rec& recL, Rec& recR,
                                                 const double* q0, const double* q1,
                                                 const double* q2, int limiter,
                                                 double lambda_half, int dir) {
    if constexpr (kRecon == kReconCons) {
      exact::MusclPredictBoth<D>(eq, recL, recR, q0, q1, q2, limiter, lambda_half, dir);
    } else if constexpr (kRecon == kReconChar || kRecon == kReconPrim) {
      // dt/dx: lambda_half is (0.5 dt)/dx, so doubling it is exact
      const double lambda = 2.0 * lambda_half;
      exact::Complete<D> s0, s1, s2;
      exact::CompleteFromCons<D>(eq, s0, q0);
      exact::CompleteFromCons<D>(eq, s1, q1);
      exact::CompleteFromCons<D>(eq, s2, q2);
      if constexpr (kRecon == kReconChar)
        exact::CharPredictBoth<D>(eq, recL, recR, s0, s1, s2, lambda, dir);
      else
        exact::PrimPredictBoth<D>(eq, recL, recR, s0, s1, s2, lambda, dir);
    } else {
      exact::CompleteFromCons<D>(eq, recL, q1);
      recR = recL;
    }
  }
  static __device__ __forceinline__ Wave MakeWave(const Gas& eq, const double* u, int dir) {
    Wave w;
    exact::CompleteFromCons<D>(eq, w.q, u);
    w.dir = dir;
    return w;
  }
  static __device__ __forceinline__ double FaceMaxSpeed(const Gas& eq, const Wave& wL,
                                                        const Wave& wR) {
    return exact::HllemMaxSpeed<D>(eq, wL.q, wR.q, wL.dir);
  }
  static __device__ __forceinline__ void FluxOnly(const Gas& eq, double* F, const Rec& L,
                                                  const Rec& R, int dir) {
    exact::HllemFlux<D>(eq, F, L, R, dir);
  }
  static __device__ __forceinline__ double Face(const Gas& eq, double* F, const Rec& L,
                                                const Rec& R, const Wave& wL, const Wave& wR,
                                                int dir, Stats&) {
    exact::HllemFlux<D>(eq, F, L, R, dir);
    return exact::HllemMaxSpeed<D>(eq, wL.q, wR.q, dir);
  }
};

template <int D> struct HllemPolicy : HllemPolicyT<D, kReconNone> {};
template <int D> struct MusclHllemPolicy : HllemPolicyT<D, kReconCons> {};
template <int D> struct CharHllemPolicy : HllemPolicyT<D, kReconChar> {};
template <int D> struct PrimHllemPolicy : HllemPolicyT<D, kReconPrim> {};

template <template <int> class PT>
cudaError_t LaunchSweepRanks(const SweepArgs& a, cudaStream_t s) {
  switch (a.rank) {
  case 1:
    return LaunchSweepT<1, PT>(a, s);
  case 2:
    return LaunchSweepT<2, PT>(a, s);
  default:
    return LaunchSweepT<3, PT>(a, s);
  }
}

cudaError_t LaunchSweepHllem(const SweepArgs& a, int recon, cudaStream_t s) {
  switch (recon) {
  case kReconCons:
    return LaunchSweepRanks<MusclHllemPolicy>(a, s);
  case kReconChar:
    return LaunchSweepRanks<CharHllemPolicy>(a, s);
  case kReconPrim:
    return LaunchSweepRanks<PrimHllemPolicy>(a, s);
  default:
    return LaunchSweepRanks<HllemPolicy>(a, s);
  }
}

cudaError_t LaunchStableDtHllem(const StableDtArgs& a, cudaStream_t s) {
  return LaunchStableDtT<HllemPolicy>(a, s);
}

}  // namespace fvs

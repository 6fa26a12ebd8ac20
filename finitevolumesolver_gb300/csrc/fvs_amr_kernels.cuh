// fvs_amr_kernels.cuh -- kernels of the batched AMR patch update (2-D).
//
// PatchSweepKernel: one persistent launch per level and sweep.  Each thread
// takes segments of the level's rows (grid-stride) and marches along them
// with the same three-cell window, policy arithmetic and update as the
// uniform grid's SweepMarchKernel (fvs_sweep.cuh): for a segment [j0, j1) of
// a row it reads the ghosted cells j0-2..j1+1 of the input buffer, computes
// the faces j0..j1, writes the updated cells j0..j1-1 to the output buffer,
// accumulates dt_split * F into the flux-register entries of the row's
// captured faces (each entry belongs to exactly one face, so no atomics and
// a deterministic sum) and reduces the row's max signal speed for the
// per-sweep CFL check.  The halo cells at the ends of a row are read where
// they live (Seg::halo): the same level's current buffer or the coarser
// level, which is the ghost fill of those strips at sweep time.
//
// PatchRowWarpKernel and PatchMaxSpeedKernel put a cell on each lane, the rows
// laid end to end: the FP64 sweeps' default and every max-speed pass.
//
// For EinfeldtCfl policies (exact and fast FP64) the kernels screen the CFL
// speeds in FP32 as the uniform sweeps do (fvs_sweep.cuh): a face's exact
// speed is evaluated only when its FP32 speed plus error bound reaches the
// thread's threshold.  The rows of a warp can differ in length, so the
// decisions are per thread (no warp votes); the threshold is the thread's own
// maximum and the launch's max slot, read at every segment start, and a
// thread publishes its maximum at a segment end when it exceeds the slot
// value it read.  The maxima are the same numbers, bit for bit; the max slots
// must start at zero (or at an exact speed of the same sweep).
#pragma once

#include <climits>

#include "fvs_amr.h"
#include "fvs_sweep.cuh"

namespace fvs {
namespace amr {

template <int DIR, template <int> class PT>
__global__ void __launch_bounds__(128, PT<2>::kMinBlocks) PatchSweepKernel(PatchSweepArgs a) {
  using P = PT<2>;
  using R = typename P::Real;
  constexpr int K = kComp;
  const double split_dt = a.dt_scale * (*a.dt_ptr);
  const typename P::Gas eq = P::MakeGas(a.gamma);
  const double lambda_half = ieee64::Div(0.5 * split_dt, a.dx);
  const double dt_dx = ieee64::Div(split_dt, a.dx);
  const int64_t N = a.ncells;
  const double* __restrict__ in = a.in;
  double* __restrict__ out = a.out;
  R smax = R(0);
  int status = 0;
  typename P::Stats stats;
  constexpr bool kFilter = EinfeldtCfl<P>::value && HasFluxOnly<P>::value;
  const bool screen = kFilter && a.gamma > 1.0 && a.gamma <= 2.0;
  fast::Gas<float> g32;
  g32.gamma = static_cast<float>(a.gamma);
  g32.gm1 = static_cast<float>(a.gamma - 1.0);
  float thr = 0.0f;
  unsigned long long known = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < a.nsegs;
       r += gridDim.x * blockDim.x) {
    const Seg w = a.segs[r];
    if constexpr (kFilter) {
      known = *reinterpret_cast<volatile unsigned long long*>(a.smax_out);
      thr = fmaxf(thr, CflFloatBelow(__longlong_as_double(static_cast<long long>(known))));
    }
    int cap = w.cap_begin;
    int next_face = cap < w.cap_end ? a.caps[cap].face : INT_MAX;
    const int j0 = w.j0, j1 = w.j1;
    // returns whether the cell is a reflective boundary's image, whose
    // momentum along the row the caller negates after the conversion (so the
    // prefetched load is not waited for early)
    auto load = [&](double* u, int j) -> bool {
      const double* src = in;
      int64_t off, cs = N;
      bool flip = false;
      if (j >= 0 && j < w.n) {
        off = int64_t(w.base) + int64_t(j + kGhost) * w.stride;
      } else {  // halo cell: its source in this level or the coarser one
        const int h = j < 0 ? j + 2 : j - w.n + 2;
        const int32_t g = w.halo[h];
        if (g >= 0) {
          off = g;
        } else {
          off = -int64_t(g) - 1;
          src = a.coarse;
          cs = a.coarse_ncells;
        }
        flip = (w.flip >> h) & 1;
      }
#pragma unroll
      for (int c = 0; c < K; ++c) u[c] = __ldg(src + c * cs + off);
      return flip;
    };
    // the update re-reads the FP64 state of cell j-1 (an L1 hit) instead of
    // carrying a window of FP64 states in registers
    double dn[K];
    R cm[K], cc[K], cp[K];
    const bool flip_cm = load(dn, j0 - 2);
    P::ToCell(cm, dn);
    if (flip_cm) cm[1 + DIR] = -cm[1 + DIR];
    const bool flip_cc = load(dn, j0 - 1);
    P::ToCell(cc, dn);
    if (flip_cc) cc[1 + DIR] = -cc[1 + DIR];
    bool flip_dn = load(dn, j0);
    using FluxT = typename FluxOf<P>::type;
    typename P::Rec recR_prev;
    typename P::Wave w_prev;
    FluxT F_prev[K];
    fast::Wave<float> v_prev{};
    bool ok_prev = false;
    bool have_prev = false;  // w_prev holds the exact wave of cell j-1
    for (int j = j0 - 1; j <= j1; ++j) {
      if constexpr (kFilter) {
        float c32[K];
#pragma unroll
        for (int c = 0; c < K; ++c) c32[c] = CflToF32(cc[c]);
        const fast::Wave<float> v = fast::MakeWave<2, float>(g32, c32, DIR);
        const bool ok = screen && CflInRange<2>(c32) && v.a > 0.0f;
        if (j >= j0) {
          const float s32 = fast::FaceMaxSpeed<float>(g32, v_prev, v);
          const float sh = fast::Math<float>::Sqrt(fmaxf(v_prev.h, v.h));
          const float bound = fmaf(s32, kCflRel, fmaf(kCflScale, sh, kCflAbs));
          if (!(ok && ok_prev && bound < thr)) {
            const typename P::Wave wl = have_prev ? w_prev : P::MakeWave(eq, cm, DIR);
            w_prev = P::MakeWave(eq, cc, DIR);
            const R s = P::FaceMaxSpeed(eq, wl, w_prev);
            smax = s > smax ? s : smax;
            thr = fmaxf(thr, CflFloatBelow(static_cast<double>(smax)));
            have_prev = true;
          } else {
            have_prev = false;
          }
        }
        ok_prev = ok;
        v_prev = v;
      }
      P::ToCell(cp, dn);
      if (flip_dn) cp[1 + DIR] = -cp[1 + DIR];  // a reflective boundary's image
      if (j + 2 <= j1 + 1) flip_dn = load(dn, j + 2);
      typename P::Rec recL, recR;
      P::Predict(eq, recL, recR, cm, cc, cp, a.limiter, lambda_half, DIR);
      typename P::Wave wv{};
      if constexpr (!kFilter) wv = P::MakeWave(eq, cc, DIR);
      if (j >= j0) {
        FluxT F[K];
        if constexpr (kFilter) {
          SweepFluxOnly<P>(eq, F, recR_prev, recL, DIR);
        } else {
          const R s = SweepFace<P>(eq, F, recR_prev, recL, w_prev, wv, DIR, stats);
          smax = s > smax ? s : smax;
        }
        if (j == next_face) {
          double* dst = a.reg + int64_t(a.caps[cap].dst) * K;
#pragma unroll
          for (int c = 0; c < K; ++c) dst[c] = dst[c] + split_dt * FluxWiden(F[c]);
          ++cap;
          next_face = cap < w.cap_end ? a.caps[cap].face : INT_MAX;
        }
        if (j > j0) {
          const int64_t off = int64_t(w.base) + int64_t(j - 1 + kGhost) * w.stride;
#pragma unroll
          for (int c = 0; c < K; ++c) {
            const double v = __ldg(in + c * N + off) + dt_dx * FluxDiff(F_prev[c], F[c]);
            out[c * N + off] = v;
            if (c == 0 && __double_as_longlong(v) <= 0) status |= kStatusNonPositiveDensity;
          }
        }
#pragma unroll
        for (int c = 0; c < K; ++c) F_prev[c] = F[c];
      }
      recR_prev = recR;
      if constexpr (!kFilter) w_prev = wv;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        cm[c] = cc[c];
        cc[c] = cp[c];
      }
    }
    if constexpr (kFilter) {
      const unsigned long long b =
          static_cast<unsigned long long>(__double_as_longlong(static_cast<double>(smax)));
      if (b > known) atomicMax(a.smax_out, b);
    }
  }
  const double smax_d = static_cast<double>(smax);
  BlockMaxAtomic<1>(a.smax_out, &smax_d);
  if (status) atomicOr(&a.ctrl->step_status, status);
}

// The cell at position x (-2..n+1) of a row: interior, or a halo cell where
// it lives (this level or the coarser one; a reflective image's momentum
// along the row negated).
template <int DIR>
__device__ __forceinline__ void LoadRowCell(double* u, const Seg* seg, int n, int x,
                                            const double* __restrict__ in, int64_t N,
                                            const double* __restrict__ coarse, int64_t NC) {
  const double* src = in;
  int64_t off, cs = N;
  bool flip = false;
  if (x >= 0 && x < n) {
    off = int64_t(seg->base) + int64_t(x + kGhost) * (DIR == 0 ? 1 : seg->stride);
  } else {
    const int h = x < 0 ? x + 2 : x - n + 2;
    const int32_t g = seg->halo[h];
    if (g >= 0) {
      off = g;
    } else {
      off = -int64_t(g) - 1;
      src = coarse;
      cs = NC;
    }
    flip = (seg->flip >> h) & 1;
  }
#pragma unroll
  for (int k = 0; k < kComp; ++k) u[k] = __ldg(src + k * cs + off);
  if (flip) u[1 + DIR] = -u[1 + DIR];
}

// The CFL speed of the face between a lane's cell and its left neighbour's
// (by shuffles), folded into smax for `own` lanes.  Screened policies evaluate
// it only in warps one of whose faces can hold the launch's maximum (the FP32
// bound of the marching sweep against the published maximum).
template <int DIR, class P, class Real>
__device__ __forceinline__ void LaneFaceSpeed(const typename P::Gas& eq, const Real* c,
                                              double gamma, unsigned long long* slot, bool own,
                                              Real& smax) {
  if constexpr (EinfeldtCfl<P>::value) {
    fast::Gas<float> g32;
    g32.gamma = static_cast<float>(gamma);
    g32.gm1 = static_cast<float>(gamma - 1.0);
    const float thr =
        CflFloatBelow(BitsToDouble(*reinterpret_cast<volatile unsigned long long*>(slot)));
    float c32[kComp];
#pragma unroll
    for (int k = 0; k < kComp; ++k) c32[k] = CflToF32(c[k]);
    const fast::Wave<float> v = fast::MakeWave<2, float>(g32, c32, DIR);
    const bool ok = gamma > 1.0 && gamma <= 2.0 && CflInRange<2>(c32) && v.a > 0.0f;
    const fast::Wave<float> vm = ShflUp(v, 1);
    const bool okm = __shfl_up_sync(0xffffffffu, ok ? 1 : 0, 1) != 0;
    const float s32 = fast::FaceMaxSpeed<float>(g32, vm, v);
    const float sh = fast::Math<float>::Sqrt(fmaxf(vm.h, v.h));
    const float bound = fmaf(s32, kCflRel, fmaf(kCflScale, sh, kCflAbs));
    if (!__any_sync(0xffffffffu, own && !(ok && okm && bound < thr))) return;
  }
  const typename P::Wave w = P::MakeWave(eq, c, DIR);
  const typename P::Wave wm = ShflUp(w, 1);
  const Real s = P::FaceMaxSpeed(eq, wm, w);
  if (own) smax = s > smax ? s : smax;
}

// PatchRowWarpKernel: the sweep with the lanes of a warp along the rows.  The
// level's rows are laid end to end as slots, n + 2 per row (cells -1..n);
// warp w takes slots 30w .. 30w + 31 (grid-stride).  Lane l holds the cell of
// slot 30w + l in the compute precision and gets its neighbours by shuffles,
// or loads them where the neighbour lies in another row (the halo cells -2
// and n + 1) or outside the warp; it evaluates that cell's MUSCL predictor
// once, and the flux of the face on the cell's left.  Lanes 1..30 own their
// slots: they update interior cells (0 <= c < n) with the faces on both sides
// (the right one from the next lane), accumulate captured faces into the flux
// registers and fold their faces' signal speeds into the sweep's maximum.
// Every predictor is evaluated once per row (plus those of cells -1 and n,
// which faces 0 and n need), where PatchSweepKernel's segments repeat two per
// segment and load four halo cells each, and a warp's loads of an x row are
// consecutive.  The arithmetic per cell and face is PatchSweepKernel's: the
// results are the same, bit for bit, in the exact and mixed flavours; in fast
// FP64 the compiler may contract other products.
//
// FP64 flavours take it in both directions: a marching thread's row is a
// serial chain of FP64 instructions (64 clocks each in the FP64 unit that one
// warp saturates), and a level of 65 k cells has only ~2000 rows, 60 warps on
// the chip; as slots it has 2300 warps.  Mixed: x only (y columns would load a
// sector per value).
template <int DIR, template <int> class PT>
__global__ void __launch_bounds__(128, PT<2>::kMinBlocks) PatchRowWarpKernel(PatchSweepArgs a) {
  using P = PT<2>;
  using R = typename P::Real;
  constexpr int K = kComp;
  constexpr bool kFilter = EinfeldtCfl<P>::value && HasFluxOnly<P>::value;
  using Cell = CellArr<R, K>;
  using FluxT = typename FluxOf<P>::type;
  using Flx = CellArr<FluxT, K>;
  const double split_dt = a.dt_scale * (*a.dt_ptr);
  const typename P::Gas eq = P::MakeGas(a.gamma);
  const double lambda_half = ieee64::Div(0.5 * split_dt, a.dx);
  const double dt_dx = ieee64::Div(split_dt, a.dx);
  const int64_t N = a.ncells;
  const double* __restrict__ in = a.in;
  double* __restrict__ out = a.out;
  const int lane = threadIdx.x & 31;
  R smax = R(0);
  int status = 0;
  typename P::Stats stats;
  const int64_t nwarps = a.nslots > 1 ? (a.nslots - 1 + kRowWarpStep - 1) / kRowWarpStep : 0;
  const int64_t wstride = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < nwarps;
       w += wstride) {
    // slots past the end take the last one again and own nothing
    const int64_t s = w * kRowWarpStep + lane;
    const bool valid = s < a.nslots;
    const int64_t sc = valid ? s : a.nslots - 1;
    const int32_t r = a.slot_row[sc];
    const Seg* row = a.segs + r;
    const int n = row->n;
    const int c = static_cast<int>(sc - a.row_slot0[r]) - 1;
    auto load = [&](double* u, int x) {
      LoadRowCell<DIR>(u, row, n, x, in, N, a.coarse, a.coarse_ncells);
    };
    Cell C, Cm, Cp;
    double u[K];
    load(u, c);
    P::ToCell(C.v, u);
    Cm = ShflUp(C, 1);
    Cp = ShflDown(C, 1);
    if (c == -1 || lane == 0) {
      load(u, c - 1);
      P::ToCell(Cm.v, u);
    }
    if (c == n || lane == 31) {
      load(u, c + 1);
      P::ToCell(Cp.v, u);
    }
    const bool own = valid && lane >= 1 && lane <= kRowWarpStep && c >= 0;
    if constexpr (kFilter) LaneFaceSpeed<DIR, P, R>(eq, C.v, a.gamma, a.smax_out, own, smax);
    typename P::Rec recL, recR;
    P::Predict(eq, recL, recR, Cm.v, C.v, Cp.v, a.limiter, lambda_half, DIR);
    const typename P::Rec recRm = ShflUp(recR, 1);
    // face c (cells c-1 and c)
    Flx F;
    if constexpr (kFilter) {
      SweepFluxOnly<P>(eq, F.v, recRm, recL, DIR);
    } else {
      const typename P::Wave W = P::MakeWave(eq, C.v, DIR);
      const typename P::Wave Wm = ShflUp(W, 1);
      const R sp = SweepFace<P>(eq, F.v, recRm, recL, Wm, W, DIR, stats);
      if (own) smax = sp > smax ? sp : smax;
    }
    const Flx Fr = ShflDown(F, 1);  // face c + 1
    if (own) {
      const int cap_end = row->cap_end;
      for (int q = row->cap_begin; q < cap_end; ++q) {
        const Cap cp = a.caps[q];
        if (cp.face != c) continue;
        double* dst = a.reg + int64_t(cp.dst) * K;
#pragma unroll
        for (int k = 0; k < K; ++k) dst[k] = dst[k] + split_dt * FluxWiden(F.v[k]);
      }
      if (c < n) {
        const int64_t off = int64_t(row->base) + int64_t(c + kGhost) * (DIR == 0 ? 1 : row->stride);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const double v = __ldg(in + k * N + off) + dt_dx * FluxDiff(F.v[k], Fr.v[k]);
          out[k * N + off] = v;
          if (k == 0 && __double_as_longlong(v) <= 0) status |= kStatusNonPositiveDensity;
        }
      }
    }
  }
  const double smax_d = static_cast<double>(smax);
  BlockMaxAtomic<1>(a.smax_out, &smax_d);
  if (status) atomicOr(&a.ctrl->step_status, status);
}

template <template <int> class PT>
cudaError_t LaunchPatchRowWarpT(int dir, const PatchSweepArgs& a, int grid, int block,
                                cudaStream_t s) {
  if (a.nslots == 0) return cudaSuccess;
  if constexpr (EinfeldtCfl<PT<2>>::value) {
    if (dir == 1) {
      PatchRowWarpKernel<1, PT><<<grid, block, 0, s>>>(a);
      return cudaGetLastError();
    }
  }
  PatchRowWarpKernel<0, PT><<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

// Max signal speed over the faces 0..n of every row (the stable dt of the
// level in that direction is dx / max): one cell and the face on its left per
// lane over the slots of PatchRowWarpKernel.
template <int DIR, template <int> class PT>
__global__ void __launch_bounds__(128) PatchMaxSpeedKernel(MaxSpeedArgs a) {
  using P = PT<2>;
  using R = typename P::Real;
  const typename P::Gas eq = P::MakeGas(a.gamma);
  const int lane = threadIdx.x & 31;
  R smax = R(0);
  const int64_t nwarps = a.nslots > 1 ? (a.nslots - 1 + kLaneFaces - 1) / kLaneFaces : 0;
  const int64_t wstride = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < nwarps;
       w += wstride) {
    const int64_t s = w * kLaneFaces + lane;
    const int64_t sc = s < a.nslots ? s : a.nslots - 1;
    const int32_t r = a.slot_row[sc];
    const Seg* row = a.segs + r;
    const int c = static_cast<int>(sc - a.row_slot0[r]) - 1;
    double u[kComp];
    LoadRowCell<DIR>(u, row, row->n, c, a.in, a.ncells, a.coarse, a.coarse_ncells);
    R v[kComp];
    P::ToCell(v, u);
    const bool own = s < a.nslots && lane >= 1 && c >= 0;
    LaneFaceSpeed<DIR, P, R>(eq, v, a.gamma, a.smax_out, own, smax);
  }
  const double smax_d = static_cast<double>(smax);
  BlockMaxAtomic<1>(a.smax_out, &smax_d);
}

template <template <int> class PT>
cudaError_t LaunchPatchSweepT(int dir, const PatchSweepArgs& a, int grid, int block,
                              cudaStream_t s) {
  if (a.nsegs == 0) return cudaSuccess;
  if (dir == 0)
    PatchSweepKernel<0, PT><<<grid, block, 0, s>>>(a);
  else
    PatchSweepKernel<1, PT><<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

template <template <int> class PT>
cudaError_t LaunchPatchMaxSpeedT(int dir, const MaxSpeedArgs& a, int grid, int block,
                                 cudaStream_t s) {
  if (a.nslots == 0) return cudaSuccess;
  if (dir == 0)
    PatchMaxSpeedKernel<0, PT><<<grid, block, 0, s>>>(a);
  else
    PatchMaxSpeedKernel<1, PT><<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace amr
}  // namespace fvs

// fvs_amr_exact.cu -- AMR patch kernels with the reference's exact FP64
// arithmetic, and the table-driven kernels of the AMR step (reflux,
// average-down, dt selection, per-sweep checks).  Compiled with
// -fmad=false: the results are bit-identical to the CPU oracle's
// restatement (oracle/fvs_oracle_amr.cpp).
#include "fvs_amr.h"
#include "fvs_amr_kernels.cuh"
#include "fvs_policy_exact.cuh"

namespace fvs {
namespace amr {

cudaError_t LaunchPatchSweepExact(int dir, const PatchSweepArgs& a, int grid, int block,
                                  cudaStream_t s) {
  if (a.nslots > 0) return LaunchPatchRowWarpT<ExactPolicy>(dir, a, grid, block, s);
  return LaunchPatchSweepT<ExactPolicy>(dir, a, grid, block, s);
}

cudaError_t LaunchPatchMaxSpeedExact(int dir, const MaxSpeedArgs& a, int grid, int block,
                                     cudaStream_t s) {
  return LaunchPatchMaxSpeedT<ExactPolicy>(dir, a, grid, block, s);
}

// U += s * (0.5 * (F1 + F2) - Fc) / dx for each register slot of the cell,
// in slot order (register entry 3k: coarse sum, 3k+1 and 3k+2: the fine
// sub-faces' sums).  A thread per cell and component: what bounds it is the
// latency of its few slots, not bandwidth (15 us with a thread per cell and
// four IEEE divisions per slot).
__global__ void RefluxKernel(double* coarse, int32_t n_coarse, const double* reg,
                             const RefluxCell* cells, int32_t ncells, const float* signs,
                             double dx) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / kComp, c = t % kComp;
  if (i >= ncells) return;
  const RefluxCell rc = cells[i];
  const ieee64::Divisor ddx = ieee64::MakeDivisor(dx);
  double* cell = coarse + int64_t(c) * n_coarse + rc.cell;
  double U = *cell;
  for (int k = rc.first; k < rc.first + rc.count; ++k) {
    const double sign = static_cast<double>(signs[k]);
    const double* e = reg + int64_t(3 * k) * kComp;
    const double delta = 0.5 * (e[kComp + c] + e[2 * kComp + c]) - e[c];
    U = U + ieee64::Div(sign * delta, ddx);
  }
  *cell = U;
}

cudaError_t LaunchReflux(double* coarse, int32_t n_coarse, const double* reg,
                         const RefluxCell* cells, int32_t ncells, const float* signs, double dx,
                         cudaStream_t s) {
  if (ncells == 0) return cudaSuccess;
  RefluxKernel<<<(int64_t(ncells) * kComp + 127) / 128, 128, 0, s>>>(coarse, n_coarse, reg, cells,
                                                                     ncells, signs, dx);
  return cudaGetLastError();
}

// U_c = (((f(2i,2j) + f(2i+1,2j)) + f(2i,2j+1)) + f(2i+1,2j+1)) * 0.25
__global__ void AverageDownKernel(double* coarse, int32_t n_coarse, const double* fine,
                                  int32_t n_fine, const AvgDown* e, int32_t count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const AvgDown a = e[i];
#pragma unroll
  for (int c = 0; c < kComp; ++c) {
    const double* f = fine + int64_t(c) * n_fine + a.fine;
    const double v = (((f[0] + f[1]) + f[a.pitch]) + f[a.pitch + 1]) * 0.25;
    coarse[int64_t(c) * n_coarse + a.coarse] = v;
  }
}

cudaError_t LaunchAverageDown(double* coarse, int32_t n_coarse, const double* fine,
                              int32_t n_fine, const AvgDown* e, int32_t count, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  AverageDownKernel<<<(count + 255) / 256, 256, 0, s>>>(coarse, n_coarse, fine, n_fine, e, count);
  return cudaGetLastError();
}

// The smallest of the lanes' values in lane order (the first of equal ones; a
// NaN is never smaller).
__device__ __forceinline__ double WarpMin(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_down_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return __shfl_sync(0xffffffffu, v, 0);
}

// dt = min(t_end - t, cfl * stable), stable = min over levels l and
// directions d of 2^l * dx_l / smax(l, d), or the failed step's dt
// (SubcycleFineFirstSolver.hpp:100-112, RunSimulation.hpp:126-151).  One
// warp, a lane per level and direction.
__global__ void AmrDtKernel(AmrControl* ctrl, int nlevels, LevelDx dx) {
  const int lane = threadIdx.x;
  double stable = 1.7976931348623157e308;
  if (lane < 2 * nlevels) {
    const int l = lane >> 1, d = lane & 1;
    const double s = BitsToDouble(ctrl->smax_stable[l][d]);
    const double v = double(1 << l) * ieee64::Div(dx.dx[l], s);
    stable = v < stable ? v : stable;
  }
  stable = WarpMin(stable);
  if (lane != 0) return;
  if (ctrl->failure_dt > 0.0) stable = ctrl->failure_dt;
  const double a = ctrl->t_end - ctrl->t;
  const double b = ctrl->cfl * stable;
  ctrl->dt = a < b ? a : b;
  ctrl->step_status = 0;
}

cudaError_t LaunchAmrDt(AmrControl* ctrl, int nlevels, LevelDx dx, cudaStream_t s) {
  AmrDtKernel<<<1, 32, 0, s>>>(ctrl, nlevels, dx);
  return cudaGetLastError();
}

// Per-sweep checks in execution order (the first failing sweep decides the
// retry dt, 2^l times its level's dt), then commit the step.  One warp, 32
// sweeps at a time (28 of a 3-level step took one thread 16 us).
__global__ void AmrEndStepKernel(AmrControl* ctrl, const SweepInfo* sweeps, int nsweeps,
                                 LevelDx dx) {
  const int lane = threadIdx.x;
  const double dt = ctrl->dt;
  for (int base = 0; base < nsweeps; base += 32) {
    const int s = base + lane;
    bool bad = false;
    double retry = 0.0;
    if (s < nsweeps) {
      const int l = sweeps[s].level;
      const double smax = BitsToDouble(ctrl->smax_sweep[s]);
      const double level_dt = ieee64::Div(dx.dx[l], smax);
      bad = level_dt < sweeps[s].scale * dt;
      retry = level_dt * double(1 << l);
    }
    const unsigned failing = __ballot_sync(0xffffffffu, bad);
    if (failing) {
      if (lane == __ffs(failing) - 1) {
        ctrl->failure_dt = retry;
        ctrl->failed = 1;
      }
      return;
    }
  }
  if (lane != 0) return;
  ctrl->failed = 0;
  ctrl->t = ctrl->t + dt;
  ctrl->failure_dt = 0.0;
  ctrl->status |= ctrl->step_status;
}

cudaError_t LaunchAmrEndStep(AmrControl* ctrl, const SweepInfo* sweeps, int nsweeps,
                             LevelDx dx, cudaStream_t s) {
  AmrEndStepKernel<<<1, 32, 0, s>>>(ctrl, sweeps, nsweeps, dx);
  return cudaGetLastError();
}

// One block per part: a part of a patch's interior between the flat host layout
// ([component][ny][nx], patches one after the other) and its level's storage.
__global__ void PatchCopyKernel(const PatchCopy* parts, LevelArrays levels, double* stage,
                                int64_t base, int to_levels) {
  const PatchCopy p = parts[blockIdx.x];
  const int area = p.nx * p.rows;  // of one component: at most kPatchCopyValues, or one row
  double* level = levels.state[p.level] + p.comp * levels.ncells[p.level] + p.first;
  double* flat = stage + (p.flat - base);
  for (int i = threadIdx.x; i < area; i += blockDim.x) {
    const int row = i / p.nx;
    const int64_t at = int64_t(row) * p.pitch + (i - row * p.nx);
    for (int c = 0; c < p.ncomp; ++c) {
      double* f = flat + int64_t(c) * area + i;
      double* q = level + c * levels.ncells[p.level] + at;
      if (to_levels)
        *q = *f;
      else
        *f = *q;
    }
  }
}

cudaError_t LaunchPatchCopy(const PatchCopy* parts, int nparts, const LevelArrays& levels,
                            double* stage, int64_t base, bool to_levels, cudaStream_t s) {
  if (nparts == 0) return cudaSuccess;
  PatchCopyKernel<<<nparts, 256, 0, s>>>(parts, levels, stage, base, to_levels ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace amr
}  // namespace fvs

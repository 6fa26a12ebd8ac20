// fvs_launch_rule.h -- the automatic segment length of the uniform sweeps
// (host code without CUDA, so that a host test can check it).
#pragma once

#include <cstdint>

namespace fvs {

// What the rule depends on.
struct SweepShape {
  int rank = 3;
  int64_t cells = 0;
  int n = 0;           // cells along the sweep direction
  bool mixed = false;
  bool cut_cells = false;
  int variant = 0;     // launch variant of the marching sweep, 0: not chosen
};

// Segments of a line are blocks in the grid's second dimension.
constexpr int kMaxSegments = 65535;
inline int Segments(int n, int seg) { return n / seg + (n % seg ? 1 : 0); }

// The one-cell-per-lane sweep (a segment length of 1): its slots, two more than
// the cells of each line, are counted in 32 bits.
inline bool LanesFit(int64_t cells, int n) {
  return cells / n * (int64_t(n) + 2) < (int64_t(1) << 31);
}

// Cells per thread and segment (1: one cell per lane).
inline int AutoSegment(const SweepShape& s) {
  // Small grids: one cell per lane (SweepLanesKernel) instead of marching
  // segments, whose serial chains leave the chip idle.  Measured per sweep
  // against the best marching segment (16 cells, the shortest default, in
  // brackets): exact FP64 64^3 0.13 / 0.18 ms (0.26), 128^3 0.99 / 1.03 ms,
  // 192^3 3.25 / 2.95 ms; double-float 128^3 0.44 / 0.46 ms; mixed, where
  // lanes along y or z load a sector per value: 64^2 25 / 31 us (38), 32^3
  // equal, 64^3 20 / 11 us.  Not where the caller has chosen a variant of the
  // marching sweep.
  if (!s.cut_cells && s.variant == 0 &&
      (s.mixed ? s.rank == 1 || s.cells <= (int64_t(1) << 14)
               : s.cells <= (int64_t(1) << 22)) &&
      LanesFit(s.cells, s.n))
    return 1;
  // Enough threads for several waves of resident blocks on 152 SMs
  // (~60K threads per wave at 150 registers per thread); never shorter than
  // 16 cells, mixed 8 (the 2-cell halo of a segment is recomputed), nor more
  // segments than a launch takes.
  const int64_t target = 262144;
  const int64_t ntrans = s.cells / s.n;
  const int shortest = s.mixed && !s.cut_cells ? 8 : 16;
  int seg = s.n;
  while (seg > shortest && ntrans * Segments(s.n, seg) < target &&
         Segments(s.n, (seg + 1) / 2) <= kMaxSegments)
    seg = (seg + 1) / 2;
  return seg;
}

}  // namespace fvs

// fvs_launch_rule.h -- the automatic segment length of the uniform sweeps
// (host code without CUDA, so that a host test can check it).
#pragma once

#include <cstdint>

namespace fvs {

// The flux methods by what their sweeps cost.
enum class SweepFamily : int { kHlle = 0, kHllem = 1, kGodunov = 2 };

// What the rule depends on.
struct SweepShape {
  int rank = 3;
  SweepFamily family = SweepFamily::kHlle;
  int64_t cells = 0;
  int n = 0;           // cells along the sweep direction
  bool exact = false;  // exact FP64
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

// Whether a sweep takes one cell per lane (SweepLanesKernel) unasked: on small
// grids, whose marching segments are serial chains that leave the chip idle.
// Measured (time of a step marching at its default segments, 16 cells at these
// sizes, over that with one cell per lane; 1-D: of a sweep):
//   HLLE, exact / fast / double-float: 1-D 2^10 cells 5 / 4 / 3, 2^22 cells
//     59 / 55 / 77; 2-D 1024^2 1.32 / 1.24 / 1.20, 1448^2 1.18 / 1.10 / 1.06,
//     1500^2 1.13 / 1.07 / 1.02, 1600^2 1.08 / 1.02 / 1.01, 1800^2 1.03 / 0.97 /
//     0.99, 2048^2 1.01 / 0.95 / 0.93; 3-D 64^3 1.7 / 1.6 / 1.9, 128^3 1.08 /
//     1.07 / 1.09, 160^3 1.02 / 1.01 / 1.06
//   HLLEM and its reconstructions: 2-D 2048^2 1.06 to 1.10, 3-D 64^3 1.5 to 1.7,
//     160^3 1.03 to 1.16
//   Godunov / MUSCL-Godunov: 1-D 2^22 cells 96 / 90; 2-D 512^2 1.6 / 1.6, 1024^2
//     1.12 / 1.04, 2048^2 1.08 / 1.02 (from the mean start the first steps of
//     1024^2 0.92, twenty 1.06), but along the lines of 64 cells of 8192 x
//     64 (sweeps) 0.5 / 0.4, where a lane beside a line's end solves a Riemann
//     problem of two unrelated cells and its warp waits; 3-D 64^3 1.19 / 1.13,
//     80^3 1.06 / 1.02, 96^3 0.87 / 0.80
//   mixed, where lanes along y or z load a sector per value (sweeps): 2-D 64^2
//     1.4, 3-D 32^3 1.0, 64^3 0.6
inline bool LanesPay(const SweepShape& s) {
  constexpr int64_t k1 = 1;
  if (s.mixed) return s.rank == 1 || s.cells <= (k1 << 14);
  if (s.family == SweepFamily::kGodunov) {
    if (s.rank == 3) return s.cells <= (k1 << 19);
    if (s.rank == 2 && s.cells > (k1 << 18) && s.n < 256) return false;
  }
  if (s.family == SweepFamily::kHlle && s.rank == 2 && !s.exact) return s.cells <= 5 * (k1 << 19);
  return s.cells <= (k1 << 22);
}

// Cells per thread and segment (1: one cell per lane).
inline int AutoSegment(const SweepShape& s) {
  // not where the caller has chosen a variant of the marching sweep
  if (!s.cut_cells && s.variant == 0 && LanesPay(s) && LanesFit(s.cells, s.n)) return 1;
  // Enough threads for several waves of resident blocks on 152 SMs
  // (~60K threads per wave at 150 registers per thread); never shorter than
  // 16 cells, mixed 8 (the 2-cell halo of a segment is recomputed), FP64 cut
  // cells 8, a tile (exact / fast, two steps of 256^2: 1.80 / 1.00 ms, at 16
  // cells 2.98 / 1.58; 900^2 4.74 / 3.48 against 5.13 / 3.51; 1024^2 5.26 / 3.89
  // against 5.39 / 3.72); nor more segments than a launch takes.
  const int64_t target = 262144;
  const int64_t ntrans = s.cells / s.n;
  const int shortest = s.mixed != s.cut_cells ? 8 : 16;
  int seg = s.n;
  while (seg > shortest && ntrans * Segments(s.n, seg) < target &&
         Segments(s.n, (seg + 1) / 2) <= kMaxSegments)
    seg = (seg + 1) / 2;
  return seg;
}

}  // namespace fvs

// How the flux launches cut a grid into CTAs, from the sizes of its blocks and
// the number of SMs alone.
#pragma once

#include <algorithm>
#include <array>
#include <cmath>
#include <vector>

namespace ostc {

constexpr int kTX = 32, kTY = 4, kTZ = 1;  // per-cell tile (threads)
constexpr int kXSeg = 31;                  // cells per warp of the FP32-bulk x pass
constexpr int kFluxKC = 8;                 // k planes per column of the FP64 kernel at most

// The variants of the FP32-bulk direction passes an autotuner chooses from:
// resident CTAs per SM the register allocator is asked to allow and the cells a
// thread of the y / z pass marches over at most (fewer where the grid would leave
// SMs idle).  Every variant computes the same values.
struct FluxVariant {
  int min_blocks, march;
};
constexpr int kFluxVariants = 4;
constexpr FluxVariant kFluxVariant[kFluxVariants] = {{8, 8}, {8, 16}, {6, 8}, {4, 8}};

using BlockDims = std::array<int, 3>;  // cells of a block

constexpr int tiles_of(int cells, int per_tile) { return (cells + per_tile - 1) / per_tile; }

// Tiles of FP32-bulk pass d over a block: (x) i-segments x row groups x k,
// (y) i-groups x k-groups x j-segments, (z) i-groups x j-groups x k-segments of
// `march` cells.
inline BlockDims dir_tile_counts(int d, int march, const BlockDims &m) {
  if (d == 0) return {tiles_of(m[0], kXSeg), tiles_of(m[1], kTY), m[2]};
  if (d == 1) return {tiles_of(m[0], kTX), tiles_of(m[2], kTY), tiles_of(m[1], march)};
  return {tiles_of(m[0], kTX), tiles_of(m[1], kTY), tiles_of(m[2], march)};
}
// FP64: columns of kTX x kTY cells over kc planes, rows of 32 cells
inline BlockDims col_tile_counts(int kc, const BlockDims &m) {
  return {tiles_of(m[0], kTX), tiles_of(m[1], kTY), tiles_of(m[2], kc)};
}
inline BlockDims row_tile_counts(const BlockDims &m) { return {tiles_of(m[0], 32), m[1], m[2]}; }

template <class Count>
int ctas_of(const std::vector<BlockDims> &blocks, Count &&count) {
  int n = 0;
  for (const BlockDims &m : blocks) {
    const BlockDims t = count(m);
    n += t[0] * t[1] * t[2];
  }
  return n;
}

// The time of a flux launch in units of one face evaluation on an idle SM:
// a thread evaluates `serial` faces one after another, which take up to 1 + a
// times as long once every slot (SMs x resident CTAs) is taken, and waves of
// CTAs follow each other (a wave's end overlaps the next one by about half).
inline double flux_cost(double serial, int ctas, int slots, double a) {
  const double w = static_cast<double>(ctas) / slots;
  return serial * (1 + a * std::min(1.0, w)) * (w <= 1 ? 1.0 : 0.5 * (w + std::ceil(w)));
}

// Long columns or marches evaluate the fewest faces, short ones keep the SMs
// of a small grid busy; the constants are from event times on one B200.  FP64
// (reacting layer, in us; taken before the divisions by constants became
// products (div_by), which made a full grid 17 % faster, 160 x 96 x 64 with 4 planes
// 2.72 ms; the constants were not fitted again):
//   24 x 16 x 8:    8 / 4 / 2 / 1 planes 652 / 344 / 190 / 112, rows 24
//   45 x 37 x 21:                        707 / 381 / 225 / 240, rows 217
//   96 x 64 x 32:                        909 / 872 / 724 / 768, rows 868
//   160 x 96 x 64:                     3432 / 3291 / 3328 / 3537, rows 4199
// laminar ramp (columns, rows): 128 x 64 21, 11; 256 x 128 21, 25.
struct Fp64Cut {
  bool rows;  // k_flux_row, else ...
  int kc;     // ... k_flux_col over columns of kc planes
};
inline Fp64Cut fp64_flux_cut(const std::vector<BlockDims> &blocks, int sms, bool air) {
  bool three_d = false;
  for (const BlockDims &m : blocks) three_d = three_d || m[2] > 1;
  double best = 0;
  Fp64Cut cut{false, 0};
  for (int kc = three_d ? kFluxKC : 1; kc >= 1; kc /= 2) {
    const int ctas = ctas_of(blocks, [kc](const BlockDims &m) { return col_tile_counts(kc, m); });
    const double cost = flux_cost(three_d ? 6 * kc + 2 : 4, ctas, 2 * sms, 0.35);
    if (cut.kc && cost >= best) continue;
    best = cost;
    cut.kc = kc;
  }
  const int ctas = ctas_of(blocks, row_tile_counts);
  const double cost = flux_cost(1.5, ctas, (air ? 2 : 1) * sms, 0) + (three_d ? 0.0 : 0.9);
  cut.rows = cost < best;
  return cut;
}

// Cells a thread of FP32-bulk pass d (1 y, 2 z) marches over.  y pass, in us
// (march 8 / 4 / 2 / 1):
//   24 x 16 x 8: 153 / 88 / 54 / 39     96 x 64 x 32: 222 / 141 / 102 / 131
//   160 x 96 x 64: 336 / 364 / 412 / 457
inline int march_cut(const std::vector<BlockDims> &blocks, int d, const FluxVariant &v, int sms) {
  double best = 0;
  int march = 0;
  for (int m = v.march; m >= 1; m /= 2) {
    const int ctas = ctas_of(blocks, [d, m](const BlockDims &b) { return dir_tile_counts(d, m, b); });
    const double cost = flux_cost(m + 1, ctas, sms * v.min_blocks, 1.25);
    if (march && cost >= best) continue;
    best = cost;
    march = m;
  }
  return march;
}

}  // namespace ostc

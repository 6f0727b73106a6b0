// Which boundary or inner faces may share a launch: the points each one's
// kernel (k_bc, k_inner) reads or writes, and the grouping by them.
#pragma once

#include <algorithm>
#include <vector>

#include "engine.hpp"

namespace ostc {

// A box of points that a face kernel reads or writes in a block.
struct Touch {
  int block, lo[3], hi[3];
  bool meets(const Touch &o) const {
    if (block != o.block) return false;
    for (int d = 0; d < 3; ++d)
      if (hi[d] < o.lo[d] || o.hi[d] < lo[d]) return false;
    return true;
  }
};

struct FacePoints {
  std::vector<Touch> touch;
  int points;  // threads of its launch; 0: no face
};

// k_bc touches ngg layers on both sides of its face
inline FacePoints face_points(const HostBc &f, int ngg) {
  Touch t{f.block, {f.start[0], f.start[1], f.start[2]}, {f.end[0], f.end[1], f.end[2]}};
  t.lo[f.face] -= ngg;
  t.hi[f.face] += ngg;
  const int n = (f.end[0] - f.start[0] + 1) * (f.end[1] - f.start[1] + 1) * (f.end[2] - f.start[2] + 1);
  return {{t}, std::max(0, n)};
}

// k_inner touches its own points (plane and ghosts, with exact faces also tg
// tangential ghost rows) and the points they map to in the other block
inline FacePoints face_points(const HostInner &f, int tg) {
  Touch own{f.block, {}, {}}, other{f.target_block, {}, {}};
  int lo[3], hi[3], np = 1;  // range of d = loop_dir * n
  for (int q = 0; q < 3; ++q) {
    const int wide = q != f.face && f.n_point[q] > 1 ? tg : 0;
    const int e0 = f.loop_dir[q] * -wide, e1 = f.loop_dir[q] * (f.n_point[q] - 1 + wide);
    lo[q] = std::min(e0, e1);
    hi[q] = std::max(e0, e1);
    own.lo[q] = f.start[q] + lo[q];
    own.hi[q] = f.start[q] + hi[q];
    np *= f.n_point[q] + 2 * wide;
  }
  for (int q = 0; q < 3; ++q) {
    const int e0 = f.tstart[q] + f.tloop_dir[q] * lo[f.src_tar[q]], e1 = f.tstart[q] + f.tloop_dir[q] * hi[f.src_tar[q]];
    other.lo[q] = std::min(e0, e1);
    other.hi[q] = std::max(e0, e1);
  }
  return {{own, other}, f.n_point[0] * f.n_point[1] * f.n_point[2] > 0 ? np : 0};
}

// The launch of each face (-1: none): a face goes into the launch after the
// last earlier face that touches one of its points, so that every pair of faces
// whose order could matter keeps it.
inline std::vector<int> face_launch(const std::vector<FacePoints> &faces) {
  const int n = static_cast<int>(faces.size());
  std::vector<int> launch(n, -1);
  for (int q = 0; q < n; ++q) {
    if (faces[q].points <= 0) continue;
    launch[q] = 0;
    for (int e = 0; e < q; ++e) {
      if (faces[e].points <= 0) continue;
      bool meet = false;
      for (const Touch &x : faces[q].touch)
        for (const Touch &y : faces[e].touch) meet = meet || x.meets(y);
      if (meet) launch[q] = std::max(launch[q], launch[e] + 1);
    }
  }
  return launch;
}

}  // namespace ostc

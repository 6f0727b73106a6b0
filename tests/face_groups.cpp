// Reads faces, one per line, and prints each one's launch (face_groups.hpp):
//   b ngg  block face start[3] end[3]
//   i tg   block target face start[3] loop_dir[3] tstart[3] tloop_dir[3] src_tar[3] n_point[3]
#include <cstdio>

#include "device/face_groups.hpp"

int main() {
  std::vector<ostc::FacePoints> faces;
  char kind;
  int g;
  while (std::scanf(" %c %d", &kind, &g) == 2) {
    auto read = [](int *v) { return std::scanf("%d %d %d", v, v + 1, v + 2); };
    if (kind == 'b') {
      ostc::HostBc f{};
      if (std::scanf("%d %d", &f.block, &f.face) != 2 || read(f.start) != 3 || read(f.end) != 3) return 1;
      faces.push_back(ostc::face_points(f, g));
    } else {
      ostc::HostInner f{};
      if (std::scanf("%d %d %d", &f.block, &f.target_block, &f.face) != 3) return 1;
      for (int *v : {f.start, f.loop_dir, f.tstart, f.tloop_dir, f.src_tar, f.n_point})
        if (read(v) != 3) return 1;
      faces.push_back(ostc::face_points(f, g));
    }
  }
  for (int l : ostc::face_launch(faces)) std::printf("%d\n", l);
}

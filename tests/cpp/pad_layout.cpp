// Every address the quad kernels read from padded images -- 24- and 16-row tiles,
// quads of four halo rows, the Sobel margin around them, the slices around a z
// chunk, 64 columns of prefetch -- against the voxels k_presample and k_pad write:
// inside the allocation, and a voxel of the grid exactly where it is that voxel.
#include <cstdio>
#include <set>
#include <vector>

#include "../../lc2registration_gb300/csrc/lc2_quad_plan.hpp"

int main() {
  long long bad = 0, reads = 0;
  for (int r = 1; r <= 4; ++r)
    for (int vx : {1, 31, 32, 33, 70})
      for (int vy : {1, 15, 16, 17, 24, 25, 40, 41, 49, 60})
        for (int vz : {1, 2, 5}) {
          const lc2::PadLayout L = lc2::pad_layout(vx, vy, vz, r);
          const int images = 2, ntx = (vx + 31) / 32;
          std::vector<int> voxel(L.total(images), -1);  // which voxel of which image
          auto id = [&](int k, int x, int y, int z) { return ((k * vz + z) * vy + y) * vx + x; };
          for (int k = 0; k < images; ++k)
            for (int z = 0; z < vz; ++z)
              for (int y = 0; y < vy; ++y)
                for (int x = 0; x < vx; ++x)
                  voxel[L.first() + L.origin() + k * L.volume() + z * L.slice() + (size_t)y * L.px + x] =
                      id(k, x, y, z);
          // tile rows: 24-row tiles over the grid, or 16-row ones for the rest
          std::set<std::pair<int, int>> tiles;
          for (int y = 0; y < vy; y += 24) tiles.insert({y, 24});
          if (vy > 24 && vy % 24 > 0 && vy % 24 <= 16) tiles.insert({vy / 24 * 24, 16});
          for (int k = 0; k < images; ++k)
            for (auto& t : tiles) {
              const int quads = (t.second + 2 * r + 3) / 4, y_lo = t.first - r - 1, y_hi = t.first - r + 4 * quads;
              for (int z = -r - 1; z <= vz + r + 1; ++z)
                for (int y = y_lo; y <= y_hi; ++y)
                  for (int x = -r - 1; x <= 32 * ntx + r; ++x) {
                    const long long a = (long long)L.first() + (long long)L.origin() + k * (long long)L.volume() +
                                        z * (long long)L.slice() + (long long)y * L.px + x;
                    ++reads;
                    if (a < 0 || a >= (long long)voxel.size()) {
                      ++bad;
                      continue;
                    }
                    const bool in = x >= 0 && x < vx && y >= 0 && y < vy && z >= 0 && z < vz;
                    bad += voxel[a] != (in ? id(k, x, y, z) : -1);
                  }
              // prefetches reach 64 columns beyond a tile's first, in the grid's slices
              const long long last = (long long)L.first() + (long long)L.origin() + k * (long long)L.volume() +
                                     (vz - 1) * (long long)L.slice() + (long long)(y_hi - 1) * L.px +
                                     32 * (ntx - 1) - r + 64;
              bad += last >= (long long)voxel.size();
            }
        }
  std::printf("%lld wrong of %lld\n", bad, reads);
  return 0;
}

// lc2_quad_plan.hpp -- layout and launch plans of the quad kernels (host only).
#pragma once

#include <algorithm>
#include <cstddef>

namespace lc2 {

// Presampled images and the static ultrasound's fields in the layout
// k_fused_quad reads: every image has a border of zeros wide enough for the
// halo and the Sobel margin of every tile, so the kernel's loads need no bounds
// test. All have the same strides, so one offset addresses them all. The border
// after a row, a slice or an image is the one before the next: a read beyond the
// end of one lands there (at 96^3, radius 3, 1.17 times the grid's voxels; with
// borders of their own 1.73 times).
struct PadLayout {
  int px, py, pz;   // strides: voxels per row, rows per slice, slices per image
  int b;            // border voxels before x = 0, y = 0 and z = 0
  size_t slice() const { return (size_t)px * py; }
  size_t volume() const { return slice() * pz; }  // from one image to the next
  size_t first() const { return slice() * b; }          // of slice 0
  size_t origin() const { return (size_t)px * b + b; }  // of voxel (0, 0) in a slice
  // of n images: the border before the first, and the rows a read of the last
  // image's last slice runs on into
  size_t total(int n) const { return first() + volume() * n + slice(); }
};

// Reads of tiles of 24 and 16 rows at radius r: columns -r-1 .. 32 ntx + r, rows
// -r-1 .. rows + r, 2 more at odd radii (whole quads of the halo), where `rows`
// of 24-row tiles cover the grid, slices -r-1 .. vz+r+1.
inline PadLayout pad_layout(int vx, int vy, int vz, int r) {
  PadLayout L;
  L.b = r + 1;
  L.px = ((vx + 31) / 32 * 32 + L.b + 3) / 4 * 4;
  L.py = (vy + 23) / 24 * 24 + 2 * (r & 1) + L.b;
  L.pz = vz + 1 + L.b;
  return L;
}

// How the tiles of a group of transforms cover the grid: 24-row tiles, and one
// row of 16-row tiles below them or none, each in its own launch and z chunks.
struct QuadPlan {
  int rows24 = 0, rows16 = 0;  // rows of tiles
  int z24 = 0, z16 = 0;        // slices per CTA
  long long cost = 0;          // estimated duration: kQuadW24 per slice of a 24-row tile
};
// One weight for both kernels and all radii, between the times they measure for
// a slice of a 24- and a 16-row tile: 1.84 and 1.51 us at radius 2, 1.91 and 1.95
// at 3 and 4 (the moments threads' serial chain is the same); k_fixed_quad 1.57
// and 1.38, 1.41 and 1.41, 1.74 and 1.41.
constexpr int kQuadW24 = 12, kQuadW16 = 11;

// Plans for a grid. The plan of a number of transforms is the one with the
// least estimated duration, for one CTA per SM at a time and 2R + 3 slices per
// CTA beside its output (the windows' run-up, filling and draining). The 1-16
// rows that 24-row tiles leave over go to 16-row tiles, which fill the gaps of
// the 24-row launch's last wave, or, where that gains less than 2 %, to 24-row
// tiles that reach beyond the grid: one transform at 256^3, radius 4, takes 3
// waves of 63 slices either way, and the second launch costs 36 us of 398.
// Moments against two launches one after the other, the second's chunks chosen
// by itself: that case 402 -> 362 us, 25 transforms at 135 x 109 x 122, radius 2,
// 1049 -> 991.
class QuadPlanner {
 public:
  QuadPlanner(int vx, int vy, int vz, int r, int sms, int zchunk)
      : ntx_((vx + 31) / 32), vy_(vy), vz_(vz), h_(2 * r + 3), sms_(sms < 1 ? 1 : sms) {
    // the chunk sizes to consider, each once, with the fewest chunks that give it
    if (zchunk > 0) {
      add(1, zchunk < vz ? zchunk : vz);
      return;
    }
    for (int nz = 1; nz <= vz && nz <= kMax; ++nz) {
      const int zc = (vz + nz - 1) / nz;
      if (count_ == 0 || zc != c_[count_ - 1].zc) add(nz, zc);
    }
  }

  QuadPlan plan(int cnt) const {
    QuadPlan best;
    const int all24 = (vy_ + 23) / 24, rest = vy_ % 24;
    const long long n24 = ntx_ * all24 * cnt;
    for (int i = 0; i < considered(n24); ++i) {
      const Launch a = launch(n24, i, kQuadW24);
      const long long end = a.part ? a.whole + a.length : a.whole;
      if (i == 0 || end < best.cost) best = {all24, 0, c_[i].zc, vz_, end};
    }
    if (vy_ <= 24 || rest == 0 || rest > 16) return best;
    // two launches have to save 2 %
    const long long n = ntx_ * (vy_ / 24) * cnt, m = ntx_ * cnt;
    long long bar = best.cost - best.cost / 50;
    Launch second[kMax];
    const int seconds = considered(m);
    for (int i = 0; i < seconds; ++i) second[i] = launch(m, i, kQuadW16);
    for (int i = 0; i < considered(n); ++i) {
      const Launch a = launch(n, i, kQuadW24);
      const long long first = a.part ? a.whole + a.length : a.whole;  // both take longer
      if (first >= bar) continue;
      for (int j = 0; j < seconds; ++j) {
        const long long d = duration(a, second[j]);
        if (d >= bar) continue;
        best = {vy_ / 24, 1, c_[i].zc, c_[j].zc, d};
        bar = d;
      }
    }
    return best;
  }

 private:
  static constexpr int kMax = 64;
  struct Chunk {
    int nz, zc, chunks;
  } c_[kMax];
  // CTAs of one length as the SMs take them: whole rounds, and the rest
  struct Launch {
    long long whole, part, length;
  };
  int count_ = 0;
  long long ntx_;
  int vy_, vz_;
  long long h_, sms_;

  void add(int nz, int zc) { c_[count_++] = {nz, zc, (vz_ + zc - 1) / zc}; }
  // chunk sizes considered for n columns: at most eight CTAs per SM
  int considered(long long n) const {
    int k = 1;
    while (k < count_ && n * c_[k].nz <= 8 * sms_) ++k;
    return k;
  }
  Launch launch(long long n, int i, int weight) const {
    const long long ctas = n * c_[i].chunks, length = (c_[i].zc + h_) * weight;
    return {ctas / sms_ * length, ctas % sms_, length};
  }
  // End of launch a followed by b's CTAs as SMs come free.
  long long duration(const Launch& a, const Launch& b) const {
    const long long t0 = a.whole, t1 = t0 + a.length;
    const long long late = b.whole;  // whole rounds: every SM later by one
    const long long end = (a.part ? t1 : t0) + late;
    if (b.part > sms_ - a.part) return t1 + late + b.length;
    if (b.part && t0 + late + b.length > end) return t0 + late + b.length;
    return end;
  }
};

// Transforms per group of a batch of cnt in a buffer of cap slots, from half of
// them on: the least cost(n), summed over the groups; ties go to larger groups.
// Each n is asked for once. A launch of 100 transforms outside a graph, radius 3,
// takes 16, 26 and 50 us of host time at 64^3, 20 x 40 x 64 and 32 x 40 x 200; with
// every n asked for again and every pair of chunk sizes tried 91, 180 and 382.
template <typename Cost>
int group_size(int cnt, int cap, Cost cost) {
  constexpr int kKnown = 128;
  long long known[kKnown];
  std::fill(known, known + kKnown, -1);
  auto of = [&](int n) -> long long {
    if (n <= 0) return 0;
    if (n >= kKnown) return cost(n);
    if (known[n] < 0) known[n] = cost(n);
    return known[n];
  };
  int best_g = cap;
  long long best = -1;
  for (int g = cap; g >= (cap + 1) / 2; --g) {
    long long total = (long long)(cnt / g) * of(g);
    if (best >= 0 && total >= best) continue;
    total += of(cnt % g);
    if (best < 0 || total < best) {
      best = total;
      best_g = g;
    }
  }
  return best_g;
}

}  // namespace lc2

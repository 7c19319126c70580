// Launch plans of the quad kernels against the search they stand for, every pair
// of chunk sizes tried, over grids, radii, batches and fixed chunk sizes; then the
// host time of a batch's grouping against the same search.
#include <chrono>
#include <cstdio>
#include <random>

#include "../../lc2registration_gb300/csrc/lc2_quad_plan.hpp"

using lc2::QuadPlan;

static QuadPlan search(int vx, int vy, int vz, int r, int cnt, int sms, int zchunk) {
  QuadPlan best;
  const long long ntx = (vx + 31) / 32, h = 2 * r + 3;
  auto end = [&](long long a, long long la, long long b, long long lb) {
    const long long part = a % sms, t0 = a / sms * la, t1 = t0 + la, late = b / sms * lb, left = b % sms;
    long long e = (part ? t1 : t0) + late;
    if (left > sms - part)
      e = t1 + late + lb;
    else if (left && t0 + late + lb > e)
      e = t0 + late + lb;
    return e;
  };
  auto chunks = [&](int zc) { return (vz + zc - 1) / zc; };
  auto each = [&](long long n, auto f) {
    if (zchunk > 0) return f(zchunk < vz ? zchunk : vz);
    for (int nz = 1, last = 0; nz <= vz && nz <= 64 && (nz == 1 || n * nz <= 8LL * sms); ++nz) {
      const int zc = (vz + nz - 1) / nz;
      if (zc != last) f(zc);
      last = zc;
    }
  };
  const int all = (vy + 23) / 24, rest = vy % 24;
  const long long n24 = ntx * all * cnt;
  each(n24, [&](int z) {
    const long long d = end(n24 * chunks(z), (z + h) * lc2::kQuadW24, 0, 0);
    if (!best.z24 || d < best.cost) best = {all, 0, z, vz, d};
  });
  if (vy > 24 && rest > 0 && rest <= 16) {
    const long long n = ntx * (vy / 24) * cnt, m = ntx * cnt, bar = best.cost - best.cost / 50;
    each(n, [&](int z) {
      each(m, [&](int zz) {
        const long long d = end(n * chunks(z), (z + h) * lc2::kQuadW24, m * chunks(zz), (zz + h) * lc2::kQuadW16);
        if (d < bar && d < best.cost) best = {vy / 24, 1, z, zz, d};
      });
    });
  }
  return best;
}

static int search_group(int vx, int vy, int vz, int r, int cnt, int cap, int sms) {
  auto cost = [&](int n) { return n <= 0 ? 0 : search(vx, vy, vz, r, n, sms, 0).cost; };
  int best_g = cap;
  long long best = -1;
  for (int g = cap; g >= (cap + 1) / 2; --g) {
    const long long total = (cnt / g) * cost(g) + cost(cnt % g);
    if (best < 0 || total < best) {
      best = total;
      best_g = g;
    }
  }
  return best_g;
}

static int group(int vx, int vy, int vz, int r, int cnt, int cap, int sms) {
  const lc2::QuadPlanner p(vx, vy, vz, r, sms, 0);
  return lc2::group_size(cnt, cap, [&](int n) { return p.plan(n).cost; });
}

template <typename F>
static double best_us(F f) {
  double best = 1e30;
  for (int i = 0; i < 20; ++i) {
    const auto t0 = std::chrono::steady_clock::now();
    f();
    const std::chrono::duration<double, std::micro> d = std::chrono::steady_clock::now() - t0;
    if (d.count() < best) best = d.count();
  }
  return best;
}

int main() {
  std::mt19937 rng(1);
  auto upto = [&](int lo, int hi) { return (int)std::uniform_int_distribution<int>(lo, hi)(rng); };
  int bad = 0, two = 0;
  for (int i = 0; i < 20000; ++i) {
    const int vx = upto(1, 300), vy = upto(1, 300), vz = upto(1, 300), r = upto(1, 4);
    const int cnt = upto(0, 1) ? upto(1, 4) : upto(1, 64), sms = upto(0, 3) ? 152 : upto(1, 200);
    const int zchunk = upto(0, 4) ? 0 : upto(1, 320);
    const QuadPlan a = search(vx, vy, vz, r, cnt, sms, zchunk);
    const QuadPlan b = lc2::QuadPlanner(vx, vy, vz, r, sms, zchunk).plan(cnt);
    two += a.rows16;
    bad += a.rows24 != b.rows24 || a.rows16 != b.rows16 || a.z24 != b.z24 || a.z16 != b.z16 || a.cost != b.cost;
  }
  for (int i = 0; i < 150; ++i) {
    const int vx = upto(1, 200), vy = upto(1, 200), vz = upto(1, 200), r = upto(1, 4), cap = upto(1, 64);
    const int cnt = upto(1, 600);
    bad += search_group(vx, vy, vz, r, cnt, cap, 152) != group(vx, vy, vz, r, cnt, cap, 152);
  }
  volatile int sink = 0;
  double t[2] = {0, 0};
  const int grids[3][3] = {{64, 64, 64}, {20, 40, 64}, {32, 40, 200}};
  for (auto& g : grids) {
    t[0] += best_us([&] { sink = sink + search_group(g[0], g[1], g[2], 3, 100, 64, 152); });
    t[1] += best_us([&] { sink = sink + group(g[0], g[1], g[2], 3, 100, 64, 152); });
  }
  std::printf("%d wrong, %d with two launches, %.1f us searched, %.1f us planned\n", bad, two, t[0], t[1]);
  return 0;
}

// Host-side checks of plan_segments and filter_batch
// (fft3dcl_gb300/csrc/f3d_batch_plan.hpp) over the planes engines ask for, one
// block row a segment included: the segments are those of the smallest
// waves x (rows + 1.5) over every number of rows, each has a block row, one
// plane alone stays within one wave, and long planes are planned in less than a
// fifth of the time that trying every number of rows takes; the filter's groups
// cover every block row of every plane once. Built and run by
// tests/test_batch_rows_cpu.py; prints "ok" or the failed case.
#include "f3d_batch_plan.hpp"

#include <chrono>
#include <cstdio>
#include <vector>

using namespace f3d;

static SweepArgs plane(int w, int h, int n, int slots) {
  SweepArgs a{};
  const int c = n / 2, tj = 256 / n - 1;
  a.inv.g.bw = a.inv.g.bh = n;
  a.inv.g.W = w;
  a.inv.g.H = h;
  a.inv.bm = 3;
  a.cells_x = (w + c - 1) / c;
  a.cells_y = (h + c - 1) / c;
  a.inv.g.ncols = a.cells_x + 2;
  a.strips = (a.cells_x + tj - 1) / tj;
  a.segs = most_segments(slots, a.strips, a.cells_y);
  return a;
}

// Every number of rows in turn.
static void plan_all_rows(SweepArgs* p, int n, int slots) {
  int most = 1, best = 0;
  for (int i = 0; i < n; i++)
    if (p[i].cells_y + 1 > most) most = p[i].cells_y + 1;
  auto segs_of = [](const SweepArgs& a, int rows) {
    const int s = (a.cells_y + rows) / rows;
    return s < a.segs ? s : a.segs;
  };
  long long best_cost = 0;
  for (int rows = 1; rows <= most; rows++) {
    long long ctas = 0;
    int longest = 0;
    for (int i = 0; i < n; i++) {
      const int s = segs_of(p[i], rows), r = (p[i].cells_y + s) / s;
      ctas += (long long)p[i].strips * s;
      longest = r > longest ? r : longest;
    }
    const long long cost = (ctas + slots - 1) / slots * (2 * longest + 3);
    if (!best || cost <= best_cost) best = rows, best_cost = cost;
  }
  for (int i = 0; i < n; i++) p[i].segs = segs_of(p[i], best);
}

static bool filter_ok(std::vector<SweepArgs> v, int n) {
  static SweepBatch Bf, Bs, Bm;
  static FilterBatch F;
  const int k = (int)v.size(), group = 256 / n;
  for (SweepArgs& a : v) {
    a.tab = reinterpret_cast<const uint8_t*>(16);
    a.err = reinterpret_cast<int*>(16);
    a.img = reinterpret_cast<uint8_t*>(16);
  }
  if (!sweep_batches(v.data(), k, Bf, Bs, Bm)) return false;
  const int ctas = filter_batch(Bs, group, F);
  int at = 0;
  for (int i = 0; i < k; i++) {
    const int blocks = (v[i].cells_y + 1) * v[i].inv.g.ncols;
    if (F.cta0[i] != at || F.p[i].nblk != blocks || F.run[i] != Bs.run[i] || F.rlen[i] != Bs.rlen[i]) return false;
    at += (blocks + group - 1) / group;
    // A run's CTAs are dealt to its planes in turn: each must have the same number.
    if (F.run[i] < i && blocks != F.p[F.run[i]].nblk) return false;
  }
  for (int i = k; i <= kMaxBatch; i++)
    if (F.cta0[i] != at) return false;
  return ctas == at && F.shifted == Bs.shifted && F.n == k;
}

int main() {
  const int sizes[][2] = {{16, 16}, {17, 33}, {64, 360}, {640, 360}, {854, 480}, {1280, 720}, {1919, 1079}, {3840, 2160}, {7680, 4320}, {96, 4096}, {4096, 96}};
  for (int slots : {3, 148 * 3, 152 * 3})
    for (int n : {8, 16, 32})
      for (const auto& s : sizes)
        for (int k = 1; k <= kMaxBatch; k++)
          for (int chroma = 0; chroma < 2; chroma++) {
            std::vector<SweepArgs> v;
            for (int i = 0; i < k; i++)
              v.push_back(chroma && i % 3 ? plane(s[0] / 2 + 1, s[1] / 2 + 1, n, slots) : plane(s[0], s[1], n, slots));
            std::vector<SweepArgs> w = v;
            const std::vector<SweepArgs> own = v;
            plan_segments(v.data(), k, slots);
            plan_all_rows(w.data(), k, slots);
            bool good = n == 8 || filter_ok(v, n);
            for (int i = 0; i < k; i++) {
              const int nrow = v[i].cells_y + 1;
              good = good && v[i].segs == w[i].segs && v[i].segs >= 1 && v[i].segs <= own[i].segs;
              for (int g = 0; g < v[i].segs; g++)  // the kernels' rows of a segment
                good = good && (long long)(g + 1) * nrow / v[i].segs > (long long)g * nrow / v[i].segs;
            }
            if (k == 1) good = good && (v[0].strips > slots || v[0].strips * v[0].segs <= slots);
            if (!good) {
              std::printf("FAILED %d slots, %dx%d blocks, %dx%d plane, %d entries, chroma %d\n", slots, n, n, s[0], s[1], k, chroma);
              return 1;
            }
          }
  auto us = [](void (*plan)(SweepArgs*, int, int)) {
    double best = 1e30;
    for (int rep = 0; rep < 20; rep++) {
      std::vector<SweepArgs> v(kMaxBatch, plane(64, 16384, 8, 456));
      const auto t0 = std::chrono::steady_clock::now();
      plan(v.data(), kMaxBatch, 456);
      const double t = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count();
      best = t < best ? t : best;
    }
    return best;
  };
  const double fast = us(plan_segments), slow = us(plan_all_rows);
  if (fast > slow / 5) {
    std::printf("FAILED plan of long planes: %.1f us, every number of rows %.1f us\n", fast, slow);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}

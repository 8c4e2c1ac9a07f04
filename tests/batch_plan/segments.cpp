// Host-side checks of plan_segments (fft3dcl_gb300/csrc/f3d_batch_plan.hpp):
// every plane keeps at least one segment and at most those its seam buffers
// hold, no plan costs more waves x (rows + 1.5) than the planes' own segments,
// and one plane alone fills one wave. Built and run by
// tests/test_segment_plan_cpu.py; prints "ok" or the failed case.
#include "f3d_batch_plan.hpp"

#include <cstdio>
#include <vector>

using namespace f3d;

static SweepArgs plane(int w, int h, int n, int slots) {
  SweepArgs a{};
  const int c = n / 2, tj = 256 / n - 1;
  a.cells_x = (w + c - 1) / c;
  a.cells_y = (h + c - 1) / c;
  a.strips = (a.cells_x + tj - 1) / tj;
  int s = slots / a.strips;
  if (s > (a.cells_y + 1) / 2) s = (a.cells_y + 1) / 2;
  a.segs = s < 1 ? 1 : s;
  return a;
}

static double cost(const std::vector<SweepArgs>& v, int slots) {
  long long ctas = 0;
  int longest = 0;
  for (const SweepArgs& a : v) {
    ctas += (long long)a.strips * a.segs;
    const int r = (a.cells_y + 1 + a.segs - 1) / a.segs;
    longest = r > longest ? r : longest;
  }
  return (double)((ctas + slots - 1) / slots) * (longest + 1.5);
}

int main() {
  const int sizes[][2] = {{16, 16}, {17, 33}, {64, 360}, {640, 360}, {854, 480}, {1280, 720}, {1919, 1079}, {3840, 2160}, {7680, 4320}};
  for (int slots : {3, 148 * 3, 152 * 3})
    for (int n : {16, 32})
      for (const auto& s : sizes)
        for (int k = 1; k <= kMaxBatch; k++)
          for (int chroma = 0; chroma < 2; chroma++) {
            std::vector<SweepArgs> v;
            for (int i = 0; i < k; i++)
              v.push_back(chroma && i % 3 ? plane(s[0] / 2 + 1, s[1] / 2 + 1, n, slots) : plane(s[0], s[1], n, slots));
            const std::vector<SweepArgs> own = v;
            plan_segments(v.data(), k, slots);
            bool good = cost(v, slots) <= cost(own, slots) + 1e-9;
            for (int i = 0; i < k; i++) good = good && v[i].segs >= 1 && v[i].segs <= own[i].segs;
            if (!good) {
              std::printf("FAILED %d slots, %dx%d blocks, %dx%d plane, %d entries, chroma %d\n", slots, n, n, s[0], s[1], k, chroma);
              return 1;
            }
          }
  std::printf("ok\n");
  return 0;
}

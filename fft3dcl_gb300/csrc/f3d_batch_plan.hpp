// f3d_batch_plan.hpp -- host-side planning of the batched tensor-core
// launches: the by-value batch parameters of the forward and of the filter
// and inverse kernels, with each kernel's per-plane prefix of CTA (or
// block-group) counts, the filter's runs of one geometry and its
// shifted-window bits. Plain host code, also compiled by the CPU tests.
#pragma once

#include "f3d_kernels.hpp"

namespace f3d {

// Blocks per tensor-core forward group: one M = 128 tile of blocks x n/2
// packed columns (8 blocks of 32 x 32, 16 of 16 x 16).
constexpr int tc_group_size(int bw) { return 256 / bw; }

// The forward batch parameter of `planes` (false: not one batch).
inline bool forward_batch(const TcFwdArgs* planes, int n, TcFwdBatch& B) {
  if (n < 1 || n > kMaxBatch) return false;
  B = TcFwdBatch{};
  B.n = n;
  for (int i = 0; i < n; i++) {
    const TcFwdArgs& a = planes[i];
    if ((a.g.bw != 16 && a.g.bw != 32) || a.g.bh != a.g.bw || a.g.bw != planes[0].g.bw || a.g.mode != 1 ||
        a.fmt != planes[0].fmt)
      return false;
    B.p[i] = a;
    const int gs = tc_group_size(a.g.bw);
    B.grp0[i + 1] = B.grp0[i] + (a.g.nb + gs - 1) / gs;
  }
  for (int i = n + 1; i <= kMaxBatch; i++) B.grp0[i] = B.grp0[n];
  return true;
}

// The sweep-side batch parameters (by (row, strip) group, by CTA of the sweep,
// by seam row) of `planes`: the same planes, with the prefix of each one's
// counts. tc: the tensor-core sweep (16x16 or 32x32 blocks, tables, block
// images); otherwise the fast form's fused sweep (8x8 to 32x32 blocks; only Bs
// is used).
inline bool sweep_batches(const SweepArgs* planes, int n, SweepBatch& Bf, SweepBatch& Bs, SweepBatch& Bm,
                          bool tc = true) {
  if (n < 1 || n > kMaxBatch) return false;
  SweepBatch B{};
  B.n = n;
  for (int i = 0; i < n; i++) {
    const SweepArgs& a = planes[i];
    const int bw = a.inv.g.bw;
    const bool size_ok = tc ? (bw == 16 || bw == 32) : (bw == 8 || bw == 16 || bw == 32);
    if (!size_ok || a.inv.g.bh != bw || bw != planes[0].inv.g.bw || (tc && (!a.tab || !a.err || !a.img)) ||
        a.inv.bm != planes[0].inv.bm || a.inv.half != planes[0].inv.half)
      return false;
    B.p[i] = a;
  }
  // Runs of consecutive planes of one geometry (the same group and segment
  // counts). A run of consecutive outputs of one plane is shifted: every
  // window frame but the newest is the previous entry's (the same spectrum
  // buffers). The filter kernel interleaves the CTAs of a run's planes.
  const int nf = B.p[0].inv.bm >= 2 ? B.p[0].inv.bm : 1;
  B.shifted = 0;
  for (int i = 0; i < n; i++) {
    const SweepArgs& a = B.p[i];
    const bool same = i > 0 && a.inv.g.W == B.p[i - 1].inv.g.W && a.inv.g.H == B.p[i - 1].inv.g.H &&
                      a.strips == B.p[i - 1].strips && a.segs == B.p[i - 1].segs;
    B.run[i] = same ? B.run[i - 1] : i;
    B.rlen[i] = 0;
    B.rlen[B.run[i]]++;
    bool shift = same && nf > 1;
    for (int k = 0; k + 1 < nf && shift; k++) shift = a.inv.s[k] == B.p[i - 1].inv.s[k + 1];
    if (shift) B.shifted |= 1 << i;
  }
  auto prefix = [&](SweepBatch& out, auto count) {
    out = B;
    for (int i = 0; i < n; i++) out.cta0[i + 1] = out.cta0[i] + count(out.p[i]);
    for (int i = n + 1; i <= kMaxBatch; i++) out.cta0[i] = out.cta0[n];
  };
  prefix(Bf, [](const SweepArgs& a) { return a.strips * (a.cells_y + 1); });  // (row, strip) groups
  prefix(Bs, [](const SweepArgs& a) { return a.strips * a.segs; });          // (strip, segment)
  prefix(Bm, [](const SweepArgs& a) { return a.segs > 1 ? a.segs - 1 : 0; });  // seams
  return true;
}

// The switches all planes of a batch share (kSwAny where they differ).
inline int filter_switches(const SweepBatch& S) {
  int sw = filter_switches(S.p[0].inv);
  for (int i = 1; i < S.n; i++)
    if (filter_switches(S.p[i].inv) != sw) sw = kSwAny;
  return sw;
}

// The most segments a plane's strips are cut into: at most one wave of `slots`
// resident CTAs (a partial second wave would double the time); one block row a
// segment where they still fit (360p 8-bit bt=3, 72 -> 144 CTAs: 27.6 -> 26.8 us
// a pass; every row is then read and written once more, in L2).
inline int most_segments(int slots, int strips, int cells_y) {
  int s = slots / strips;
  if (s > cells_y + 1) s = cells_y + 1;
  return s < 1 ? 1 : s;
}

// Segments of each plane's strips (written to its segs, at most what it comes
// with) for one launch of all planes' sweeps, `slots` CTAs of which run at a
// time. A CTA costs its block rows plus about one and a half for its set-up
// and its seams, and a last wave costs as much as a full one: the rows per
// segment with the smallest waves x (rows + 1.5), the largest such. Each
// plane's own plan fills one wave by itself: a 1080p 4:2:0 frame then had 756
// CTAs of 2 to 3 rows for 456 slots and 56 seams, here 378 CTAs of 5 rows and
// 25 seams (its step, with the seams finished in the sweep: 123.5 -> 120.7
// us; ten 4K outputs 1750 -> 1738 us).
//
// rows goes from one change of any plane's segments to the next: every number
// of rows in turn took most of a long plane's host time (eight outputs of
// 64x16384 with 8x8 blocks: 160 us a step, 56 before there was a plan; sixteen
// planned in 282 us on an x86 host, 4 this way).
inline void plan_segments(SweepArgs* planes, int n, int slots) {
  if (slots < 1) return;
  int most = 1;
  for (int i = 0; i < n; i++) most = planes[i].cells_y + 1 > most ? planes[i].cells_y + 1 : most;
  auto segs_of = [&](const SweepArgs& a, int rows) {
    const int s = (a.cells_y + 1 + rows - 1) / rows;
    return s < a.segs ? s : a.segs;
  };
  int best = 0;
  long long best_cost = 0;
  for (int rows = 1, next; rows <= most; rows = next) {
    long long ctas = 0;
    int longest = 0, s = 1;
    next = most + 1;
    for (int i = 0; i < n; i++) {
      const SweepArgs& a = planes[i];
      if (i == 0 || a.cells_y != planes[i - 1].cells_y || a.segs != planes[i - 1].segs) {
        const int all = a.cells_y + 1;
        s = segs_of(a, rows);
        const int r = (all + s - 1) / s, fewer = s > 1 ? (all + s - 2) / (s - 1) : next;  // rows with s - 1 segments
        longest = r > longest ? r : longest;
        next = fewer < next ? fewer : next;
      }
      ctas += (long long)a.strips * s;
    }
    const long long cost = (ctas + slots - 1) / slots * (2 * longest + 3);
    if (best == 0 || cost <= best_cost) best = rows, best_cost = cost;
  }
  for (int i = 0; i < n; i++) planes[i].segs = segs_of(planes[i], best);
}

// The filter's batch parameter of the planes of a sweep batch (sweep_batches):
// the same runs, with the prefix of the planes' groups of `group` blocks.
// Returns the CTAs (groups) of the launch.
inline int filter_batch(const SweepBatch& S, int group, FilterBatch& F) {
  F.n = S.n;
  F.shifted = S.shifted;
  F.clk = S.p[0].clk;
  F.cta0[0] = 0;
  for (int i = 0; i < S.n; i++) {
    const SweepArgs& a = S.p[i];
    F.p[i].f = a.inv;
    F.p[i].img = a.img;
    F.p[i].nblk = (a.cells_y + 1) * a.inv.g.ncols;
    F.run[i] = S.run[i];
    F.rlen[i] = S.rlen[i];
    F.cta0[i + 1] = F.cta0[i] + (F.p[i].nblk + group - 1) / group;
  }
  for (int i = S.n + 1; i <= kMaxBatch; i++) F.cta0[i] = F.cta0[S.n];
  return F.cta0[S.n];
}

// Autotuner choice among n timed launch shapes (fastest[i]: the fastest of
// shape i's runs; shape 0 is the default): the fastest shape, unless the
// default is within `margin` of it (single-step timings vary by about 1 %).
inline int autotune_pick(const float* fastest, int n, float margin = 0.01f) {
  int pick = 0;
  for (int c = 1; c < n; c++)
    if (fastest[c] < fastest[pick]) pick = c;
  return fastest[0] <= (1.0f + margin) * fastest[pick] ? 0 : pick;
}

}  // namespace f3d

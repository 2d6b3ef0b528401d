// How many tiles of a chunk's sweep one thread block of the tensor-core kernels takes.
//
// One block per chunk lasts as long as the longest sweep, whatever the chip has idle; many short blocks pay their start-up each.
// Both are reckoned here: the launch is played through on 148 SMs with a block time of start + cost * tiles, for whole sweeps and
// for segments of 1, 2, 4 .. tiles, and the shortest wins (whole sweeps unless another is at least 5 % shorter).  The constants are
// microseconds, fitted to forwards and backwards of 1 to 4 query heads at head_dim 64 and 128 on one to 64 (batch, head) units; of the
// shapes measured, with every segment length tried, the choice is the best one or within 5 % of it.  A plan depends on the shape
// alone and the last ones are kept per thread: a call asks for it several times.
#pragma once
#include <algorithm>
#include <functional>
#include <vector>

#include "ua_common.cuh"

namespace ua {
namespace sm100 {

constexpr int kSms = 148;

// 128-row tiles in the sweep of chunk i (chunks of 64 keys start a tile at their own first row)
inline int sweep_tiles(const Shape& s, int i) { return (s.L - i * s.C + 127) / 128; }
// ... and 64-row half tiles, the backward's unit
inline int sweep_halves(const Shape& s, int i) { return (s.L - i * s.C) / 64; }

// End of the last block when every chunk i of every (batch, head) unit takes len(i) units in blocks of seg (0: all of them), launched
// chunk by chunk; skip: blocks at the start of each chunk's list that have nothing to do.
template <typename Len>
double play(const Shape& s, Len len, int seg, int skip, double start, double cost) {
  static thread_local std::vector<double> free_at;
  free_at.assign(kSms, 0.0);                          // a heap, earliest first
  double end = 0;
  for (int i = 0; i < s.N; ++i) {
    const int n = len(i), step = seg ? seg : n;
    for (int t = skip * step; t < n; t += step) {
      const double d = start + cost * std::min(step, n - t);
      for (int bh = 0; bh < s.B * s.H; ++bh) {
        std::pop_heap(free_at.begin(), free_at.end(), std::greater<double>());
        free_at.back() += d;
        end = std::max(end, free_at.back());
        std::push_heap(free_at.begin(), free_at.end(), std::greater<double>());
      }
    }
  }
  return end;
}

struct SplitPlan {
  Shape s;
  int fwd, bwd;
};
inline SplitPlan make_split_plan(const Shape& s) {
  SplitPlan p{s, 0, 0};
  const double BH = (double)s.B * s.H, R = s.R, narrow = s.C == 64 ? 0.7 : 1.0;
  double tiles = 0;
  for (int i = 0; i < s.N; ++i) tiles += sweep_tiles(s, i);
  // enough work for every SM behind the longest sweep: nothing to gain, and nothing to play through
  if (BH * tiles > 1.3 * kSms * sweep_tiles(s, 0) || BH * tiles > 8192) return p;
  {
    const double start = 9.0, cost = narrow * (s.D == 64 ? 3.8 + 0.8 * R : 3.2 + 1.35 * R), totals = 3.0 + BH * tiles * (s.D == 64 ? 0.01 : 0.018);
    auto len = [&](int i) { return sweep_tiles(s, i); };
    double best = 0.95 * play(s, len, 0, 0, start, cost);
    for (int t = 1; t < len(0); t *= 2) {
      const double est = totals + play(s, len, t, 0, start, cost);
      if (est < best) { best = est; p.fwd = t; }
    }
  }
  {
    const double start = 12.0, cost = narrow * (s.D == 64 ? 3.3 + 0.9 * R : 3.4 + 1.9 * R), corr_start = 6.0, corr = narrow * (s.D == 64 ? 2.2 : 2.6);
    auto len = [&](int i) { return sweep_halves(s, i); };
    double best = 0.95 * play(s, len, 0, 0, start, cost);
    for (int t = 2; t < len(0); t *= 2) {
      const double est = 2.0 + play(s, len, t, 0, start, cost) + play(s, len, t, 1, corr_start, corr);
      if (est < best) { best = est; p.bwd = t; }
    }
  }
  return p;
}
inline const SplitPlan& split_plan(const Shape& s) {
  static thread_local SplitPlan kept[16] = {};
  static thread_local int next = 0;
  for (const SplitPlan& p : kept)
    if (p.s.B == s.B && p.s.H == s.H && p.s.R == s.R && p.s.N == s.N && p.s.C == s.C && p.s.D == s.D) return p;
  kept[next] = make_split_plan(s);
  const SplitPlan& p = kept[next];
  next = (next + 1) % 16;
  return p;
}
// row tiles per block of the forward, half tiles per block of the backward; 0: a block sweeps its whole chunk
inline int fwd_split(const Shape& s) { return split_plan(s).fwd; }
inline int bwd_split(const Shape& s) { return split_plan(s).bwd; }

inline size_t fwd_totals_bytes(const Shape& s) { return (size_t)s.B * s.H * s.N * sweep_tiles(s, 0) * 128 * sizeof(float); }
inline int bwd_max_segments(const Shape& s, int seg) { return seg ? (s.L / 64 + seg - 1) / seg : 0; }

}  // namespace sm100
}  // namespace ua

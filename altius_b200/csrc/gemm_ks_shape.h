// Tile width, K split and shared memory of the kernel for products of few rows (gemm_ks.cu): host arithmetic only.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

namespace ac {
namespace gemm_ks {

constexpr int BM = 128, KB = 64, kMaxStages = 4;
constexpr int kAHalf = BM * KB * 2;           // bytes of A's hi (or lo) tile: rows of 128 bytes
constexpr size_t kSmemMax = 231000;

struct Shape {
  int bn = 0, split = 0;                      // columns of a tile, blocks that share it along K
  int kper = 0, stages = 0;                   // K-blocks of a block, ring entries
  int inv = 0;                                // c * inv >> 20: the block that finishes quad c of the tile
  size_t smem = 0;
  double clocks = 1e30;
};

inline int k_blocks(int64_t k, bool wide) {
  const int step = wide ? KB / 2 : KB;
  return (int)((k + step - 1) / step);
}

// The one place that kper, stages, inv and smem come from. False: no kernel of that width and split, as a block of the cluster would
// have no K-block, a column no owner, or the ring no room.
inline bool make_shape(int bn, int split, int64_t k, bool wide, Shape* s) {
  const int nkb = k_blocks(k, wide);
  if ((bn != 32 && bn != 64 && bn != 96 && bn != 128) || (split != 1 && split != 2 && split != 4 && split != 8) || nkb < 1) return false;
  const int kper = (nkb + split - 1) / split;
  if ((split - 1) * kper >= nkb || (bn % (4 * split)) != 0) return false;
  const int quads = bn / split / 4;
  const size_t stage = (wide ? 1 : 2) * (size_t)kAHalf + (size_t)bn * KB * 4, ex = (size_t)split * quads * (BM + 1) * 16;
  const int stages = (int)std::min<size_t>(std::min(kper, kMaxStages), (kSmemMax - 1024 - (split > 1 ? ex : 0)) / stage);
  if (stages < std::min(2, kper)) return false;
  s->bn = bn;
  s->split = split;
  s->kper = kper;
  s->stages = stages;
  s->inv = ((1 << 20) + quads - 1) / quads;
  s->smem = std::max(stages * stage + (split > 1 ? ex : 0), ex) + 1024;
  return true;
}

// By clocks, from stamps in the kernel: a K-block costs its twelve MMAs (45 to 65 clocks
// each) or its bytes at 60 a clock, whichever is more; first loads and drain 2700; exchange 1600 and 18
// per column; epilogue 1500 and 40 per column that a block finishes. A launch as timed takes 1.4 to 2 times as long
// (launch, cold code; operands arrive at 34 bytes a clock when all SMs load at once).
//
// Fp32 operands: a K-block of 32 costs 1190 clocks up to 96 columns, 1370 with 128. `slots(split)`: clusters that run at once.
template <typename Slots>
Shape pick_shape(int64_t m, int64_t n, int64_t k, bool wide, Slots slots) {
  Shape best;
  const long long mt = (m + BM - 1) / BM;
  for (int bn : {32, 64, 96, 128}) {
    for (int split : {1, 2, 4, 8}) {
      Shape s;
      if (!make_shape(bn, split, k, wide, &s)) continue;
      const double waves = std::ceil((double)mt * ((n + bn - 1) / bn) / slots(split));
      const double kb = wide ? (bn > 96 ? 1370.0 : 1190.0)
                             : std::max(12 * (32.0 + 0.26 * bn), (2.0 * kAHalf + (double)bn * KB * 4) / 60.0);
      s.clocks = waves * (s.kper * kb + 4200.0 + (split > 1 ? 1600.0 + 18.0 * bn : 0.0) + 40.0 * bn / split);
      if (s.clocks < best.clocks) best = s;
    }
  }
  return best;
}

}  // namespace gemm_ks
}  // namespace ac

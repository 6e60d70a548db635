// Tile shape of the tensor-core convolution kernel (conv_tc.cu): host arithmetic only.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <array>
#include <cmath>

#include "kernels.h"

namespace ac {
namespace conv_tc {

constexpr int PX = 128, KB = 32;             // pixels per tile, floats of K per step (128-byte rows)
constexpr int kMaxStages = 3;
constexpr int kABytes = PX * KB * 4;         // one of hi / lo

struct Shape {
  int bn, tiles, split, kper, stages, resident, ctas;
  int set, mains, bufs, cols;                // tensor memory: see the end of pick_shape
  size_t smem;
  double rounds;                             // of the blocks (clusters) that run at once
};

constexpr size_t kSmemSm = 233472;           // shared memory of an SM
constexpr size_t kSmemMax = 231000;          // dynamic shared memory of one block
constexpr size_t kSmemBeside = 2304;         // beside it: 1120 static bytes, 1024 of the system, rounding

// Picks channels per tile and K split among those that fit a block's shared memory with two stages. Times in clocks, from measurements of the kernel's parts: a K step
// costs its loads and stores to shared memory (about 420 when blocks overlap) or its MMAs (12 per
// full step at 65 or 0.8 per channel, whichever is more), the epilogue about 4 per channel, start
// and end 2500 and a cluster's exchange 1500.
inline Shape pick_shape(const ConvParams& q, const std::array<int, 4>& slots) {
  const int sms = slots[0];
  const int k = q.c * q.kh * q.kw, nkb = (k + KB - 1) / KB;
  const long long px = ((long long)q.n * q.oh * q.ow + PX - 1) / PX;
  const bool window = q.kh != 1 || q.kw != 1 || q.sh != 1 || q.sw != 1 || q.pad_t || q.pad_l || q.oh != q.ih || q.ow != q.iw;
  const size_t table = window ? (size_t)k * sizeof(int2) : 0;
  // Shared memory of a block: ring, filter tile where it stays, sums of the cluster, table, alignment.
  auto bytes = [&](int bn, int split, int kper, int stages, bool resident) {
    const size_t bb = (size_t)bn * KB * 8;
    return stages * (2 * (size_t)kABytes + (resident ? 0 : bb)) + (resident ? kper * bb : 0) +
           (split > 1 ? (size_t)bn * PX * 4 : 0) + table + 1024;
  };
  Shape best{};
  double best_t = 1e30;
  for (int tiles = (q.oc + 255) / 256; tiles <= (q.oc + 15) / 16; ++tiles) {
    const int bn = ((q.oc + tiles - 1) / tiles + 15) / 16 * 16;
    if ((bn * (tiles - 1)) >= q.oc) continue;
    for (int split = 1; split <= 8; split *= 2) {
      const int kper = (nkb + split - 1) / split;
      if ((split - 1) * kper >= nkb || bytes(bn, split, kper, std::min(2, kper), false) > kSmemMax) continue;
      const double step = std::max(420.0, 12 * std::max(65.0, 0.8 * bn) * std::min(1.0, k / 32.0));
      const double body = kper * step + 4.0 * bn, waves = std::ceil((double)px * tiles / slots[split <= 1 ? 0 : split <= 2 ? 1 : split <= 4 ? 2 : 3]);
      const double t = waves * body + 2500 + (split > 1 ? 1500 : 0);
      if (t < best_t * 0.98) { best_t = t; best.bn = bn; best.tiles = tiles; best.split = split; best.kper = kper; }
    }
    if (bn <= 32) break;
  }
  // Blocks walk tiles when there are more than two per SM (and nothing is cut over a cluster), two blocks to an SM:
  // each has half of tensor memory, which holds the accumulators of up to 128 channels.
  const bool walk = best.split == 1 && px * best.tiles > 2 * sms;
  if (walk && best.bn > 128) {
    best.tiles = (q.oc + 127) / 128;
    best.bn = ((q.oc + best.tiles - 1) / best.tiles + 15) / 16 * 16;
  }
  // A walking block keeps its filter tile in shared memory where that leaves room for two stages.
  const size_t half = kSmemSm / 2 - kSmemBeside;
  best.resident = walk && bytes(best.bn, 1, best.kper, 2, true) <= half;
  best.stages = std::min(best.kper * (walk ? 2 : 1), kMaxStages);
  auto need = [&](int st) { return bytes(best.bn, best.split, best.kper, st, best.resident); };
  // As many stages as leave room for a second block on the SM, at least two when there are two steps.
  while (best.stages > 2 && need(best.stages) > half) --best.stages;
  // Accumulators: `set` columns each. The tensor core truncates its sum at every instruction by up to an ulp of
  // the sum, an error that grows with the instructions behind one another: so the cross terms, 2^-11 of the
  // result, have an accumulator of their own, and the main terms of narrow tiles, and of a K cut eight times, are
  // dealt to two, K step by K step. (All on one: 1.3e-6 of the result at 2048 x 7 x 7 into 512, 5.9e-7 at
  // 480 x 32 x 32 into 480; the GEMM on a column buffer, with its up to 32 slices of K, 3.4e-7 and 2.7e-7; this way
  // 2.5e-7 and 2.3e-7.) A single K step, or two of a block that walks, need none of it, all terms are on one
  // (mains 0): that GEMM has no shorter slices, and cuts K only where it has few tiles (64 x 56 x 56 into 256, one
  // image: two steps on one 2.6e-7, this way 1.1e-7, that GEMM 1.9e-7). Walking blocks have a second buffer of
  // accumulators, so that the products of the next tile run under the stores of a tile, as far as the columns go.
  best.set = best.bn <= 32 ? 32 : best.bn <= 64 ? 64 : best.bn <= 128 ? 128 : 256;
  best.mains = best.kper == 1 || (walk && best.kper == 2) ? 0 : walk || best.set == 256 || (best.set == 128 && best.split < 8) ? 1 : 2;
  best.bufs = walk && best.set * (best.mains + 1) <= 128 ? 2 : 1;   // mains 0: always two
  best.cols = 32;
  while (best.cols < best.set * (best.mains + 1) * best.bufs) best.cols *= 2;
  // Shared memory in proportion to the columns, so that whatever blocks share an SM find theirs. (With 2048 bytes
  // for what lies beside it two blocks of 256 columns missed the SM by 192 bytes, and half of a grid of two
  // blocks per SM started when the other half had finished.)
  best.smem = std::max(need(best.stages), best.cols == 512 ? kSmemSm / 2 : kSmemSm * best.cols / 512 - kSmemBeside);
  const int resident_blocks = sms * (best.smem <= half ? 2 : 1);
  best.rounds = (double)px * best.tiles / (best.split == 1 ? resident_blocks : slots[best.split == 2 ? 1 : best.split == 4 ? 2 : 3]);
  best.ctas = (int)(walk ? std::min<long long>(px, std::max(1, resident_blocks / best.tiles)) : px);
  return best;
}

}  // namespace conv_tc
}  // namespace ac

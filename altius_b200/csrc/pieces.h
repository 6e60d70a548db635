// Runs from host memory in pieces of the batch: the steps at the front of a schedule that treat images one by one start on
// the first images while the others are still on their way to the device. Host logic only.
#pragma once
#include <stddef.h>

#include <algorithm>
#include <vector>

namespace ac {

struct PiecePlan {
  int steps = 0;      // steps [0, steps) run piece by piece; 0: the whole schedule at once
  int images = 0;     // of the batch
  int per = 0;        // of a piece, the last one may be smaller
  int count() const { return per ? (images + per - 1) / per : 0; }
  int begin(int k) const { return k * per; }
  int end(int k) const { return std::min(images, (k + 1) * per); }
};

// `front`: steps at the front that can run on a part of the batch. Pieces are multiples of four images (so that their
// data stays 16-byte aligned whatever an image's size), four at most, of 2 MB or more. Below 8 MB, or with fewer than
// three steps to hide, the launches cost what the overlap gives.
inline PiecePlan plan_pieces(int front, int images, size_t input_bytes) {
  PiecePlan p;
  if (front < 3 || images < 8 || input_bytes < (size_t(8) << 20)) return p;
  const size_t image = input_bytes / (size_t)images;
  const int least = (int)(((size_t(2) << 20) + image - 1) / image);
  const int per = (std::max((images + 3) / 4, least) + 3) / 4 * 4;
  if (per >= images) return p;
  p.steps = front;
  p.images = images;
  p.per = per;
  return p;
}

}  // namespace ac

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

// A step at the front that can run on a part of the batch: its time on all of it, and for how many rounds its blocks fill the device.
struct FrontStep {
  double us = 0, rounds = 1;
  // On a share of the batch: the launch, and at least one round of the blocks.
  double part(double share) const { return kLaunch + std::max(0.0, us - kLaunch) * std::max(1.0, rounds * share) / std::max(1.0, rounds); }
  static constexpr double kLaunch = 2.5;
};

// Pieces are multiples of four images (so that their data stays 16-byte aligned whatever an image's size), four at most, of 2 MB or more;
// inputs below 8 MB stay whole. The front ends where the run would end first: a step in it runs once a piece, which is lost
// time where a piece does not fill the device or its images have all arrived (128 images of 512 x 7 x 7 through 60 pointwise
// convolutions 1.5 ms, with all of them in the front 4.5), and gained where it runs under the upload. Less than 20 us is
// not worth the launches. (64 images of 256 x 14 x 14 through 20 pointwise convolutions 774 us whole, 995 with all in the front, 727 so;
// MobileNetV3-Large, 32 images, 1268 whole, 1058 with the eleven steps up to the first squeeze-and-excite block, which it chooses.)
inline PiecePlan plan_pieces(const std::vector<FrontStep>& front, int images, size_t input_bytes) {
  PiecePlan p;
  if (front.empty() || images < 8 || input_bytes < (size_t(8) << 20)) return p;
  const size_t image = input_bytes / (size_t)images;
  const int least = (int)(((size_t(2) << 20) + image - 1) / image);
  const int per = (std::max((images + 3) / 4, least) + 3) / 4 * 4;
  if (per >= images) return p;
  const double upload = (double)input_bytes / 45e3;          // us at 45 GB/s
  double whole = upload;
  for (const FrontStep& s : front) whole += s.us;
  PiecePlan cut;
  cut.images = images;
  cut.per = per;
  double best = whole - 20.0, rest = whole - upload;
  std::vector<double> piece((size_t)cut.count(), 0.0);       // time of a piece's steps
  for (int steps = 1; steps <= (int)front.size(); ++steps) {
    const FrontStep& s = front[(size_t)steps - 1];
    rest -= s.us;
    double t = 0.0;
    for (int k = 0; k < cut.count(); ++k) {
      piece[(size_t)k] += s.part((double)(cut.end(k) - cut.begin(k)) / images);
      t = std::max(t, upload * cut.end(k) / images) + piece[(size_t)k];
    }
    if (t + rest < best) {
      best = t + rest;
      p = cut;
      p.steps = steps;
    }
  }
  return p;
}

}  // namespace ac

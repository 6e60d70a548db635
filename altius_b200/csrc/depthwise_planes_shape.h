// Split of the depthwise kernel that works on whole planes (depthwise_planes.cu): host arithmetic only.
#pragma once
#include <stddef.h>

#include <algorithm>

#include "kernels.h"

namespace ac {
namespace depthwise_planes {

constexpr int kMaxThreads = 512;
constexpr size_t kMaxSmem = 100 << 10;       // two blocks an SM

struct Shape {
  int per;                   // planes a block
  int stride;                // floats from plane to plane in shared memory
  int rows, segs;            // output rows a thread, threads down a column
  int threads;
  size_t smem;
};

inline bool supported(const ConvParams& p) {
  const long long ihw = (long long)p.ih * p.iw;
  return p.kh == p.kw && (p.kh == 3 || p.kh == 5) && p.sh == 1 && p.sw == 1 && p.dh == 1 && p.dw == 1 &&
         (p.act == ACT_NONE || p.act == ACT_RELU || p.act == ACT_HARDSWISH) && p.ow <= kMaxThreads / 4 &&
         (ihw + 32) * (long long)sizeof(float) * ((ihw & 3) ? 4 : 1) <= (long long)kMaxSmem && (long long)p.n * p.c < (1ll << 30) &&
         p.oh >= 1 && p.ow >= 1;
}

// For a batch of q.n images. The order in which a plane's mean is added up follows from rows and segs, so a launch on a
// part of the batch takes the shape of the whole.
inline Shape pick_shape(const ConvParams& q, int sms) {
  Shape s{};
  const int planes = q.n * q.c, ihw = q.ih * q.iw, unit = (ihw & 3) ? 4 : 1;
  // Neighbouring lanes walk neighbouring columns, then the next plane's: its banks follow on those of the row (in
  // whole float4s where the copies are).
  const int step = (ihw & 3) ? 1 : 4;
  s.stride = ihw;
  while ((((s.stride - q.iw) % 32) + 32) % 32 >= step) s.stride += step;
  // About 14 rows a thread and 256 threads a block; fewer planes and shorter columns while the SMs hold more threads
  // than that gives (32 images, 200 planes of 14 x 14: 8.7 us with 600 threads an SM, 6.1 with 1200).
  s.segs = std::max(1, std::min((q.oh + 13) / 14, kMaxThreads / (unit * q.ow)));
  const int fit = std::max(1, (int)(kMaxSmem / 2 / sizeof(float)) / (s.stride * unit));
  int units = std::max(1, std::min(256 / (s.segs * q.ow * unit), fit));
  while (units > 1 && (planes + units * unit - 1) / (units * unit) < 2 * sms) units /= 2;
  s.per = units * unit;
  while ((q.oh + s.segs - 1) / s.segs > 4 && (long long)planes * s.segs * q.ow < (long long)sms * 1024 &&
         2 * s.per * s.segs * q.ow <= kMaxThreads)
    s.segs *= 2;
  s.rows = (q.oh + s.segs - 1) / s.segs;
  s.segs = (q.oh + s.rows - 1) / s.rows;
  s.threads = (s.per * s.segs * q.ow + 31) / 32 * 32;
  s.smem = (size_t)s.per * s.stride * sizeof(float);
  return s;
}

}  // namespace depthwise_planes
}  // namespace ac

// Split of the depthwise kernel that works on whole planes (depthwise_planes.cu), and where it is taken: host arithmetic only.
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

// Microseconds of a launch behind another one: this kernel's (a column's chain of rows, or the instructions of all threads, whichever is
// more, and most of the other), and those of the kernel that reads global memory (depthwise_rows_kernel, four pixels a thread).
// Fitted over 630 layers of 1 to 64 images, 16 to 960 planes, rows of 3 to 126 that are no whole float4s.
inline double planes_us(const ConvParams& q, int sms) {
  const Shape s = pick_shape(q, sms);
  const bool wide = q.kh == 5;
  const double steps = s.rows + q.kh - 1, blocks = (double)(((long long)q.n * q.c + s.per - 1) / s.per);
  const double chain = steps * (wide ? 0.16 : 0.115), issue = blocks * s.threads * steps * (wide ? 0.46 : 0.36) / (1000.0 * sms);
  return 2.5 + std::max(chain, issue) + 0.6 * std::min(chain, issue);
}
inline double rows_us(const ConvParams& q, int sms) {
  const double quads = (double)q.n * q.c * q.oh * ((q.ow + 3) / 4);
  return std::max(2.8, 2.6 + quads * (q.kh == 5 ? 27.7e-6 : 12.9e-6) * 148 / sms);
}

// Whether this kernel is the faster one. Only for rows that are no whole float4s: of those the other takes a value a load, but with them,
// and at stride two, it is the faster one (32 images, 240 planes of 28 x 28, 3 x 3, stride two: 7.3 us against 9.3). Few or large
// planes leave a thread a long column and most SMs idle (us, rows -> planes: one image, 16 planes of 75 x 75, 3 x 3 3.1 -> 16.5, 72 of
// 61 x 61, 5 x 5 4.3 -> 11.3; 32 images, 72 of 61 x 61, 5 x 5 63.9 -> 34.5, 960 of 7 x 7 14.1 -> 9.3, 480 of 14 x 14, 3 x 3 13.7 -> 10.0,
// 16 of 75 x 75 12.2 -> 19.2). Over the 630 the choice takes 5 % less than the other kernel alone, 0.7 % more than the better one each
// time would. `gain`: us that the means of the planes are worth where only this kernel leaves them.
inline bool wins(const ConvParams& q, int sms, double gain = 0.0) {
  return (q.iw & 3) != 0 && supported(q) && planes_us(q, sms) < 0.95 * rows_us(q, sms) + gain;
}

}  // namespace depthwise_planes
}  // namespace ac

"""The depthwise kernel on whole planes (depthwise_planes_shape.h): its split over a sweep of layers, the choice between it and the
kernel that reads global memory at layers timed with both, and its results where it is chosen."""
import os
import subprocess

import numpy as np
import pytest
import torch

from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# images, planes, height, width, filter, padding: planes of whole float4s and others, a remainder of planes, one and several
# segments of a column, rectangles, results larger and smaller than the planes, rows of one and two values
CHOSEN = [(32, 480, 14, 14, 3, 1), (31, 333, 9, 9, 5, 2), (24, 64, 122, 122, 3, 1), (21, 72, 37, 61, 5, 2), (32, 120, 27, 31, 5, 0),
          (64, 501, 9, 10, 5, 4), (33, 960, 7, 7, 5, 2), (64, 997, 11, 1, 5, 2), (64, 960, 12, 2, 5, 2)]
HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "depthwise_planes_shape.h"
using namespace ac;
static ConvParams layer(int n, int c, int h, int w, int k, int p) {
  ConvParams q{};
  q.n = n; q.c = q.oc = q.group = c; q.ih = h; q.iw = w; q.kh = q.kw = k; q.sh = q.sw = q.dh = q.dw = 1; q.pad_t = q.pad_l = p;
  q.oh = h + 2 * p - k + 1; q.ow = w + 2 * p - k + 1; q.act = ACT_RELU;
  return q;
}
int main(int argc, char** argv) {
  for (int i = 1; i + 5 < argc; i += 6) {
    int v[6];
    for (int j = 0; j < 6; ++j) v[j] = std::atoi(argv[i + j]);
    std::printf("%d\n", depthwise_planes::wins(layer(v[0], v[1], v[2], v[3], v[4], v[5]), 148) ? 1 : 0);
  }
  if (argc > 1) return 0;
  for (int k : {3, 5})
    for (int p = 0; p < k; ++p)
      for (int h : {1, 2, 5, 7, 14, 15, 28, 57, 113, 128, 300})
        for (int w : {1, 2, 3, 7, 10, 14, 31, 57, 75, 113, 126})
          for (int c : {1, 16, 121, 960})
            for (int n : {1, 7, 64}) {
              const ConvParams q = layer(n, c, h, w, k, p);
              if (q.oh < 1 || q.ow < 1 || !depthwise_planes::supported(q)) continue;
              const depthwise_planes::Shape s = depthwise_planes::pick_shape(q, 148);
              const int unit = (h * w) % 4 ? 4 : 1;      // a block's planes start on 16 bytes
              if (s.threads < 1 || s.threads > depthwise_planes::kMaxThreads || s.threads % 32 || s.per % unit || s.per * s.segs * q.ow > s.threads ||
                  s.rows * s.segs < q.oh || s.rows * (s.segs - 1) >= q.oh || s.stride < h * w || s.smem > depthwise_planes::kMaxSmem ||
                  s.smem != (size_t)s.per * s.stride * 4) {
                std::printf("n %d c %d %d x %d filter %d pad %d: per %d rows %d segs %d threads %d smem %zu\n", n, c, h, w, k, p, s.per, s.rows, s.segs,
                            s.threads, s.smem);
                return 1;
              }
            }
  std::puts("ok");
}
"""
# us of the kernel on global memory and on whole planes (square, padding k / 2): the choice may cost a twentieth at most
TIMED = [(1, 16, 75, 3, 3.1, 16.5), (1, 72, 61, 5, 4.3, 11.3), (1, 16, 114, 3, 3.5, 8.2), (4, 480, 15, 3, 3.9, 5.2), (32, 16, 75, 3, 12.2, 19.2),
         (8, 64, 75, 3, 12.0, 18.9), (32, 72, 61, 5, 63.9, 34.5), (32, 960, 7, 5, 14.1, 9.3), (32, 480, 14, 3, 13.7, 10.0),
         (32, 64, 114, 3, 93.4, 71.5), (8, 72, 37, 5, 8.6, 7.6), (32, 120, 22, 5, 16.6, 12.2)]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("planes")
    (d / "p.cpp").write_text(HARNESS)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-I", os.path.join(cuda, "include"),
                    str(d / "p.cpp"), "-o", str(d / "p")], check=True)
    return lambda *a: subprocess.run([str(d / "p"), *map(str, a)], capture_output=True, text=True).stdout.split("\n")[:-1]


def test_every_split_can_be_launched(harness):
    assert harness() == ["ok"]


def test_choice(harness):
    assert harness(*[v for q in CHOSEN for v in q]) == ["1"] * len(CHOSEN)
    picks = harness(*[v for n, c, h, k, _, _ in TIMED for v in (n, c, h, h, k, k // 2)])
    for pick, (*layer, rows, planes) in zip(picks, TIMED):
        assert (planes if pick == "1" else rows) <= 1.05 * min(planes, rows), layer


@pytest.mark.gpu
@pytest.mark.parametrize("n,c,h,w,k,p", CHOSEN)
def test_convolution_on_whole_planes(cuda_lib, n, c, h, w, k, p):
    rng = np.random.default_rng(h * w + k)
    x, f, b = (rng.standard_normal(d).astype(np.float32) for d in ((n, c, h, w), (c, 1, k, k), (c,)))
    g = ir.Graph()
    y = g.op("Conv2d", g.add_input("x", x.shape), g.new_init(f), g.new_init(b), kernel_shape=[k, k], strides=[1, 1], padding=[p] * 4,
             dilations=[1, 1], group=c, auto_pad="")
    g.outputs.append(g.op("ReLU", y))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        assert [e["kind"] for e in sess.schedule()] == ["conv_depthwise"]
        got = torch.from_numpy(sess.run([x])[0]).cuda()
    finally:
        sess.close()
    conv = lambda *a: torch.nn.functional.conv2d(*(torch.from_numpy(t).cuda().double() for t in a), padding=p, groups=c)
    # k * k products and the bias: k * k + 2 roundings of terms bounded by the sum of magnitudes
    assert ((got - conv(x, f, b).clamp_min(0)).abs() <= (k * k + 2) * 2.0 ** -24 * conv(np.abs(x), np.abs(f), np.abs(b))).all()

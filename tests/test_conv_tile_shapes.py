"""Host arithmetic of the tensor-core convolution's tile choice (conv_tc_shape.h), compiled and swept
over layers, batches and numbers of clusters that run at once: every shape it returns can be launched, and
the blocks that walk tiles run at once."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SWEEP = r"""
#include <cstdio>
#include "conv_tc_shape.h"
using namespace ac;
int main() {
  long long tried = 0, bad = 0;
  for (std::array<int, 4> slots : {std::array<int, 4>{148, 74, 33, 15}, {148, 74, 36, 18}, {148, 64, 32, 16}, {132, 66, 28, 12}})
    for (int kk : {1, 3, 5, 7})
      for (int c : {1, 3, 16, 21, 24, 40, 64, 72, 96, 128, 160, 240, 256, 448, 455, 512, 672, 960, 1024, 2048, 4096})
        for (int oc : {1, 16, 24, 64, 80, 112, 128, 160, 176, 208, 224, 240, 255, 256, 300, 384, 480, 512, 960, 1280, 2048, 16384})
          for (int h : {1, 7, 14, 28, 32, 56, 112, 224})
            for (int n : {1, 2, 3, 4, 8, 9, 13, 16, 32, 64}) {
              if ((long long)c * kk * kk > 4096 || (long long)n * h * h >= (1ll << 24)) continue;
              ConvParams q{};
              q.n = n; q.c = c; q.ih = q.iw = q.oh = q.ow = h; q.oc = oc; q.kh = q.kw = kk; q.sh = q.sw = q.dh = q.dw = 1;
              q.pad_t = q.pad_l = kk / 2; q.group = 1;
              const conv_tc::Shape s = conv_tc::pick_shape(q, slots);
              const int k = c * kk * kk, nkb = (k + 31) / 32;
              ++tried;
              // What lives on an SM together: 1120 static bytes and 1024 of the system beside the dynamic ones.
              const long long px = ((long long)n * h * h + 127) / 128;
              const int per_sm = (int)std::min<size_t>(7, 233472 / ((s.smem + 1120 + 127) / 128 * 128 + 1024));
              const bool walks = s.ctas < px;
              const bool fits = per_sm * s.cols <= 512 && s.cols >= s.set * (s.mains + 1) * s.bufs && s.set >= s.bn && s.cols >= 32 &&
                                (s.mains > 0 || s.kper == 1 || (walks && s.kper == 2)) && (s.mains > 0 || !walks || s.bufs == 2) && (!walks || s.ctas == 1 || s.ctas * s.tiles <= per_sm * slots[0]);
              const bool ok = fits && s.bn >= 16 && s.bn <= 256 && s.bn % 16 == 0 && s.tiles >= 1 && s.tiles <= 65535 && (long long)s.tiles * s.bn >= oc &&
                              s.split * s.kper >= nkb && (s.split - 1) * s.kper < nkb && s.ctas >= 1 &&
                              s.stages >= std::min(2, s.kper) && s.stages <= 3 && s.smem <= conv_tc::kSmemMax;
              if (!ok && ++bad <= 12)
                std::printf("n %d c %d h %d oc %d filter %d slots %d: bn %d split %d stages %d smem %zu blocks %d x %d, %d an SM\n", n, c, h, oc, kk,
                            slots[3], s.bn, s.split, s.stages, s.smem, s.ctas, s.tiles, per_sm);
            }
  std::printf("%lld tried, %lld bad\n", tried, bad);
  return bad != 0;
}
"""


def test_every_convolution_tile_can_be_launched(tmp_path):
    src = tmp_path / "sweep.cpp"
    src.write_text(SWEEP)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-I", os.path.join(cuda, "include"),
                    str(src), "-o", str(tmp_path / "sweep")], check=True)
    r = subprocess.run([str(tmp_path / "sweep")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

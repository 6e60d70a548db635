"""The split of a batch into pieces whose first steps run while the others' images are still on their way (pieces.h): the
plan, the arena's part in it, and runs from host memory against runs on device buffers."""
import os
import subprocess

import numpy as np
import pytest

from altius_b200 import configs, ir
from altius_b200.session import CudaSessionBuilder

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <cstdio>
#include "pieces.h"
using ac::FrontStep;
int main() {
  int cut = 0, tried = 0;
  for (int n = 0; n < 30; ++n)
    for (double us : {3.0, 10.0, 40.0, 200.0})
      for (double rounds : {0.3, 1.0, 2.5, 20.0})
        for (int images = 1; images < 200; images += images < 40 ? 1 : 13)
          for (size_t image : {size_t(12), size_t(40000), size_t(602112), size_t(3) << 20}) {
            const std::vector<FrontStep> front((size_t)n, FrontStep{us, rounds});
            const ac::PiecePlan p = ac::plan_pieces(front, images, image * images);
            ++tried;
            if (!p.steps) { if (p.count()) return 1; continue; }
            ++cut;
            if (p.steps > n || image * images < (size_t(8) << 20) || p.per % 4 || p.count() < 2 || p.count() > 4) return 2;
            if ((size_t)p.per * image < (size_t(2) << 20) || p.begin(0) != 0 || p.end(p.count() - 1) != images) return 3;
            for (int k = 0; k + 1 < p.count(); ++k) if (p.end(k) != p.begin(k + 1) || p.end(k) <= p.begin(k)) return 4;
            if (p.end(p.count() - 1) <= p.begin(p.count() - 1)) return 5;
            if (rounds <= 1.0) return 6;        // a piece takes as long as the batch: nothing to gain
          }
  if (cut < tried / 50) return 7;
  // Steps that fill the device many times over run in pieces while the rest is under way, not far beyond: 100 MB are 2.2 ms.
  for (int n : {5, 30, 300}) {
    const ac::PiecePlan p = ac::plan_pieces(std::vector<FrontStep>((size_t)n, FrontStep{40.0, 20.0}), 100, 100000000);
    if (p.steps < std::min(n, 30) || p.steps > 90) return 8;
  }
  // Half of the steps are worth it, none of those behind.
  std::vector<FrontStep> front(10, FrontStep{30.0, 8.0});
  front.insert(front.end(), 10, FrontStep{30.0, 0.7});
  if (ac::plan_pieces(front, 64, 40000000).steps != 10) return 9;
  std::puts("ok");
}
"""


def test_plan(tmp_path):
    src = tmp_path / "p.cpp"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-o", str(tmp_path / "p"), str(src)], check=True)
    assert subprocess.run([str(tmp_path / "p")], capture_output=True, text=True).stdout == "ok\n"


ARENA = r"""
#include <cstdio>
#include <random>
#include "arena.h"
using ac::Slot;
int main() {
  std::mt19937 rng(1);
  auto at = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  for (int round = 0; round < 2000; ++round) {
    std::vector<Slot> fixed, slots;
    const int steps = at(1, 30), n = at(1, 40);
    size_t sum = 0;
    for (int i = 0; i < n; ++i) {
      const int a = at(0, steps - 1), b = at(a, steps - 1);
      slots.push_back({(size_t)at(0, 5000), a, b, 0});
      sum += (slots.back().bytes + 255) / 256 * 256;
    }
    for (int i = at(0, 5), o = at(0, 4) * 256; i > 0; --i, o += at(0, 9) * 256) {
      fixed.push_back({(size_t)at(1, 3000), 0, steps - 1, (size_t)o});
      o = (int)fixed.back().end();
    }
    const std::vector<Slot> before = slots;
    const size_t top = ac::place_slots(slots, fixed), gap = fixed.empty() ? 0 : fixed.back().end();
    size_t end = 0;
    for (size_t i = 0; i < slots.size(); ++i) {
      const Slot& s = slots[i];
      end = std::max(end, s.end());
      if (s.bytes != before[i].bytes || s.first != before[i].first || s.last != before[i].last || s.offset % 256) return 1;
      for (size_t j = 0; j < i; ++j)
        if (s.bytes && slots[j].bytes && s.meets(slots[j]) && s.offset < slots[j].end() && slots[j].offset < s.end()) return 2;
      for (const Slot& f : fixed)
        if (s.bytes && s.offset < f.end() && f.offset < s.end()) return 3;
    }
    if (end != top || top > sum + gap) return 4;
  }
  std::puts("ok");
}
"""


def test_slots_with_common_steps_do_not_overlap(tmp_path):
    src = tmp_path / "a.cpp"
    src.write_text(ARENA)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-o", str(tmp_path / "a"), str(src)], check=True)
    r = subprocess.run([str(tmp_path / "a")], capture_output=True, text=True)
    assert r.stdout == "ok\n", r.returncode


def _convolutions(batch, layers=24, c=64, px=56):
    """A net that is all front: with every value in a place of its own it would take `layers` times its input."""
    g = ir.Graph()
    x = g.add_input("x", (batch, c, px, px))
    w = g.new_init(np.full((c, c, 1, 1), 1 / c, np.float32))
    for _ in range(layers):
        x = g.op("ReLU", g.op("Conv2d", x, w, kernel_shape=[1, 1], strides=[1, 1], padding=[0] * 4, dilations=[1, 1], group=1, auto_pad=""))
    g.outputs.append(x)
    return ir.Model(g, 13)


@pytest.mark.parametrize("model,batch,most", [
    (lambda b: configs.mobilenet_v3_large(batch=b, img=224)[0], 14, 73.5 * 2 ** 20), (lambda b: configs.mobilenet_v3_large(batch=b, img=224)[0], 32, 152.5 * 2 ** 20),
    (_convolutions, 32, 4.1 * 32 * 4 * 64 * 56 ** 2)])
def test_pieces_need_no_memory_of_their_own(model, batch, most):
    m = model(batch)
    pieces, whole = (CudaSessionBuilder(m).with_plan_only(True).with_cuda_graph(on).build() for on in (True, False))
    assert pieces.arena_bytes == whole.arena_bytes <= most


# four pieces of which the last has one image, pieces of an odd plane, four even ones
@pytest.mark.gpu
@pytest.mark.parametrize("batch,px", [(25, 224), (21, 193), (32, 224)])
def test_runs_in_pieces(cuda_lib, batch, px):
    import torch
    sess = CudaSessionBuilder(configs.mobilenet_v3_large(batch=batch, img=px)[0]).build()
    try:
        rng = np.random.default_rng(batch)
        for _ in range(3):
            x = rng.standard_normal((batch, 3, px, px)).astype(np.float32)
            want = torch.empty(sess.output_info[0][0], device="cuda")
            xd = torch.from_numpy(x).cuda()
            torch.cuda.synchronize()
            sess.run_device([xd.data_ptr()], [want.data_ptr()])
            want = want.cpu().numpy()
            assert np.array_equal(sess.run([x])[0], want)
            pinned, out = torch.from_numpy(x).pin_memory(), torch.empty(want.shape).pin_memory()
            assert np.array_equal(sess.run([pinned.numpy()], [out.numpy()])[0], want)
            outs = [[np.empty_like(want)], [np.empty_like(want)]]
            sess.run_batches([[x], [x]], outs)
            assert np.array_equal(outs[0][0], want) and np.array_equal(outs[1][0], want)
    finally:
        sess.close()


# A front whose last layers leave means of narrow planes: their sums follow the split over the whole batch, not a piece's.
@pytest.mark.gpu
@pytest.mark.parametrize("batch,c,px,k", [(128, 200, 14, 3), (104, 200, 15, 5)])
def test_pieces_give_the_bits_of_the_whole(cuda_lib, batch, c, px, k):
    import torch
    rng = np.random.default_rng(c)
    f = lambda *sh: (rng.standard_normal(sh) / np.sqrt(np.prod(sh[1:]))).astype(np.float32)
    g = ir.Graph()

    def conv(x, w, group=1):
        return g.op("Conv2d", x, g.new_init(w), kernel_shape=list(w.shape[2:]), strides=[1, 1], padding=[w.shape[2] // 2] * 4,
                    dilations=[1, 1], group=group, auto_pad="")
    y = conv(g.add_input("x", (batch, 2 * c, px, px)), f(c, 2 * c, 1, 1))
    y = g.op("ReLU", conv(y, f(c, 1, 3, 3), c))
    y = g.op("ReLU", conv(conv(y, f(c, c, 1, 1)), f(c, 1, k, k), c))
    z = conv(g.op("ReLU", conv(g.op("GlobalAveragePool", y), f(48, c, 1, 1))), f(c, 48, 1, 1))
    gate = g.op("HardSigmoid", z, alpha=0.2, beta=0.5)
    g.outputs += [gate, conv(g.op("Mul", y, gate), f(c, c, 1, 1))]
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        kinds = [e["kind"] for e in sess.schedule()]
        assert kinds == ["gemm_tf32x3_tcgen05", "conv_depthwise", "gemm_tf32x3_tcgen05", "conv_depthwise", "squeeze_excite",
                         "gemm_tf32x3_tcgen05"]
        x = rng.standard_normal((batch, 2 * c, px, px)).astype(np.float32)
        outs = [torch.empty(s, device="cuda") for s, _ in sess.output_info]
        xd = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        sess.run_device([xd.data_ptr()], [o.data_ptr() for o in outs])
        for got, want in zip(sess.run([x]), outs):
            assert np.array_equal(got, want.cpu().numpy())
    finally:
        sess.close()

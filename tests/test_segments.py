"""Runs on the caller's device buffers (segments.h): which buffers are taken, and the segments of the schedule,
with a stand-in for the capture that fails where the test says."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <cstdio>
#include <set>
#include "segments.h"
using namespace ac;
int main() {
  const std::vector<char> touches = {1, 0, 0, 1, 1, 0, 1, 0};
  for (int fails = 0; fails < 5; ++fails) {        // the capture that fails; 4: none
    std::vector<Segment> segs = split_segments(touches);
    if (segs.size() != 6 || segs[1].first != 1 || segs[1].last != 3 || segs[5].last != 8 || !segs[0].direct || segs[1].direct) return 1;
    std::set<cudaGraph_t> live;
    long made = 0;
    auto capture = [&](Segment& g) {
      const bool half = made == fails;             // a graph, but no executable
      g.graph = reinterpret_cast<cudaGraph_t>(0x1000 + 16 * made++);
      live.insert(g.graph);
      if (half) return cudaErrorMemoryAllocation;
      g.exec = reinterpret_cast<cudaGraphExec_t>(g.graph);
      return cudaSuccess;
    };
    bool unknown = false;
    auto destroy = [&](Segment& g) { unknown = unknown || live.erase(g.graph) != 1; };
    capture_segments(segs, capture, destroy);
    if (fails < 3 && (!segs.empty() || !live.empty())) return 2;
    if (fails >= 3) {
      if (segs.size() != 6 || live.size() != 3) return 3;
      for (const Segment& g : segs)
        if (g.direct ? g.exec != nullptr : g.exec == nullptr) return 4;
      destroy_segments(segs, destroy);
      if (!live.empty()) return 5;
    }
    if (unknown) return 6;
  }
  return split_segments({}).empty() ? 0 : 7;
}
"""


BUFFERS = r"""
#include "segments.h"
using namespace ac;
using B = std::pair<uintptr_t, size_t>;
int main() {
  // memory of this device from 0x10000 on, of another one from 0x20000 on, the host's from 0x30000 on
  auto local = [](uintptr_t p) { return p >= 0x10000 && p < 0x20000; };
  auto ok = [&](std::vector<B> in, std::vector<B> out) {
    return can_bind_buffers((int)in.size(), [&](int i) { return in[i]; }, (int)out.size(), [&](int i) { return out[i]; }, local);
  };
  if (!ok({{0x10000, 64}}, {{0x10040, 64}, {0x10080, 4}})) return 1;
  if (ok({{0x20000, 64}}, {{0x10040, 64}}) || ok({{0x10000, 64}}, {{0x20040, 64}})) return 2;      // another device's
  if (ok({{0x30000, 64}}, {{0x10040, 64}}) || ok({{0x10000, 64}}, {{0x10040, 64}, {0x30000, 4}})) return 3;
  if (ok({{0x10004, 60}}, {{0x10040, 64}}) || ok({{0x10000, 64}}, {{0x10048, 64}})) return 4;      // alignment
  if (ok({{0x10000, 64}}, {{0x10030, 64}}) || ok({{0x10030, 64}}, {{0x10000, 64}})) return 5;      // an input under a result
  if (ok({{0x10000, 64}}, {{0x10100, 64}, {0x10130, 64}}) || ok({{0x10000, 64}}, {{0x10000, 64}})) return 6;
  if (!ok({{0, 0}}, {{0x10040, 64}})) return 7;                                                   // nothing to read
  return 0;
}
"""


def _run(tmp_path, text):
    (tmp_path / "h.cpp").write_text(text)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-I", os.path.join(cuda, "include"),
                    str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")], check=True)
    assert subprocess.run([str(tmp_path / "h")]).returncode == 0


def test_buffers_a_run_takes_in_place(tmp_path):
    _run(tmp_path, BUFFERS)


def test_a_capture_that_fails_leaves_no_segments(tmp_path):
    _run(tmp_path, HARNESS)

"""The segments of a schedule that runs on the caller's device buffers (segments.h), with a stand-in for the
capture that fails where the test says."""
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


def test_a_capture_that_fails_leaves_no_segments(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "altius_b200", "csrc"), "-I", os.path.join(cuda, "include"),
                    str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")], check=True)
    assert subprocess.run([str(tmp_path / "h")]).returncode == 0

// Consecutive steps of a schedule for runs on bound buffers (session.cu): host logic only.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>
#include <vector>

namespace ac {

// Steps that touch a graph input or output are launched one by one on the caller's pointers, the others
// replay a graph.
struct Segment {
  int first = 0, last = 0;         // steps [first, last)
  bool direct = false;
  cudaGraph_t graph = nullptr;     // of a segment that is not direct, once captured
  cudaGraphExec_t exec = nullptr;
};

inline std::vector<Segment> split_segments(const std::vector<char>& touches) {
  std::vector<Segment> segs;
  for (int i = 0; i < (int)touches.size(); ++i) {
    if (segs.empty() || segs.back().direct != (touches[i] != 0)) {
      Segment g;
      g.first = i;
      g.direct = touches[i] != 0;
      segs.push_back(g);
    }
    segs.back().last = i + 1;
  }
  return segs;
}

template <typename Destroy>
void destroy_segments(std::vector<Segment>& segs, Destroy destroy) {
  for (Segment& g : segs)
    if (g.graph || g.exec) destroy(g);
  segs.clear();
}

// Captures the graph segments; if one fails, those made so far are destroyed and no segment is left (the
// session then runs its complete graph on copies).
template <typename Capture, typename Destroy>
void capture_segments(std::vector<Segment>& segs, Capture capture, Destroy destroy) {
  for (Segment& g : segs)
    if (!g.direct && capture(g) != cudaSuccess) return destroy_segments(segs, destroy);
}

// Whether the schedule may run on these buffers, `in(i)` and `out(i)` being their addresses and sizes.
// Kernels read and write with 16-byte accesses; a result may not land on a buffer that a later kernel
// still reads; and `local(address)` says whether the memory is the device's own -- a copy also takes
// page-locked host memory and another device's, which kernels cannot reach or reach over a link.
template <typename In, typename Out, typename Local>
bool can_bind_buffers(int n_in, In in, int n_out, Out out, Local local) {
  auto usable = [&](std::pair<uintptr_t, size_t> b) { return (b.first & 15) == 0 && (b.second == 0 || local(b.first)); };
  auto meet = [](std::pair<uintptr_t, size_t> a, std::pair<uintptr_t, size_t> b) {
    return a.first < b.first + b.second && b.first < a.first + a.second;
  };
  for (int i = 0; i < n_in; ++i)
    if (!usable(in(i))) return false;
  for (int i = 0; i < n_out; ++i) {
    if (!usable(out(i))) return false;
    for (int j = 0; j < n_in; ++j)
      if (meet(out(i), in(j))) return false;
    for (int j = 0; j < i; ++j)
      if (meet(out(i), out(j))) return false;
  }
  return true;
}

}  // namespace ac

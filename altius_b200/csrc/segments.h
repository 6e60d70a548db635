// Consecutive steps of a schedule for runs on bound buffers (session.cu): host logic only.
#pragma once
#include <cuda_runtime.h>

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

}  // namespace ac

// C ABI of the CUDA session (include/altius_session_cuda.h): parse the graph
// description, infer shapes, lower to the kernel schedule, plan one device
// arena from value lifetimes, upload the weights once, capture the schedule in
// a CUDA graph and replay it per run.
//
// Replaces InterpreterSessionBuilder::build
// (crates/session_interpreter/src/builder.rs:37-65) and InterpreterSession::run
// (crates/session_interpreter/src/session.rs:66-134). Where the reference
// allocates every node output per run (`Tensor::uninit_of_type`, :159-162) and
// frees by last use (crates/session/src/plan.rs:14-58), the same last-use
// analysis here assigns fixed arena offsets at build time.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <functional>
#include <mutex>
#include <set>

#include "session.h"

using namespace ac;

namespace {

thread_local std::string g_create_error;

#define AC_CUDA(expr)                                                                     \
  do {                                                                                    \
    cudaError_t e__ = (expr);                                                             \
    if (e__ != cudaSuccess)                                                               \
      fail(AC_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e__));             \
  } while (0)

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Reads a buffer twice the size of L2: afterwards L2 holds clean lines of that buffer only,
// so the next kernel's reads miss and its evictions cost no write-back.
constexpr size_t kSweepBytes = size_t(256) << 20;
__global__ void l2_sweep_kernel(const float4* __restrict__ p, size_t n4, float* sink) {
  float acc = 0.f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    const float4 v = __ldg(p + i);
    acc += v.x + v.y + v.z + v.w;
  }
  if (acc == 123.25f) *sink = acc;   // never true for a zeroed buffer; keeps the loads alive
}

void parse_graph(AcSession& s, const AcGraphDesc& g) {
  if (g.n_values < 0 || g.n_nodes < 0 || (g.n_values && !g.values) || (g.n_nodes && !g.nodes))
    fail(AC_ERR_INVALID, "malformed graph description");
  s.opset = g.opset_version;
  s.values.resize(g.n_values);
  for (int i = 0; i < g.n_values; ++i) {
    const AcValueDesc& d = g.values[i];
    Value& v = s.values[i];
    if (d.elem_ty < 0 || d.elem_ty > AC_I64) fail(AC_ERR_INVALID, "bad element type");
    v.elem_ty = d.elem_ty;
    v.rank = d.rank < 0 ? -1 : d.rank;
    if (d.rank > AC_MAX_RANK) fail(AC_ERR_SHAPE, "rank above 8 is not supported");
    for (int k = 0; k < v.rank; ++k) {
      if (d.dims[k] < 0) fail(AC_ERR_SHAPE, "Must be fixed dimension");  // shape.rs:675
      v.dims[k] = d.dims[k];
    }
  }
  auto check_val = [&](int v, bool allow_missing) {
    if (v == -1 && allow_missing) return;
    if (v < 0 || v >= g.n_values) fail(AC_ERR_INVALID, "value id out of range");
  };
  s.nodes.resize(g.n_nodes);
  for (int i = 0; i < g.n_nodes; ++i) {
    const AcNodeDesc& d = g.nodes[i];
    Node& n = s.nodes[i];
    if (d.op < 0 || d.op >= AC_OP_COUNT) fail(AC_ERR_INVALID, "bad operator code");
    n.op = d.op;
    for (int k = 0; k < d.n_inputs; ++k) { check_val(d.inputs[k], true); n.inputs.push_back(d.inputs[k]); }
    for (int k = 0; k < d.n_outputs; ++k) { check_val(d.outputs[k], false); n.outputs.push_back(d.outputs[k]); }
    if (n.outputs.empty()) fail(AC_ERR_INVALID, "node without outputs");
    if (d.n_ints > 0) n.ints.assign(d.ints, d.ints + d.n_ints);
    if (d.n_floats > 0) n.floats.assign(d.floats, d.floats + d.n_floats);
    if (d.name) n.name = d.name;
  }
  for (int i = 0; i < g.n_inits; ++i) {
    const AcInitDesc& d = g.inits[i];
    check_val(d.value, false);
    Value& v = s.values[d.value];
    if (v.rank < 0) fail(AC_ERR_SHAPE, "initializer without a static shape");
    if (d.bytes != v.bytes() || (!d.data && d.bytes)) fail(AC_ERR_INVALID, "initializer size mismatch");
    v.is_init = true;
    if (d.location == 0) {
      v.host = d.data;  // valid during create(); small shape tensors are kept below
      if (v.elem_ty == AC_I64 || v.numel() <= 16) {
        v.host_owned.assign(static_cast<const char*>(d.data), static_cast<const char*>(d.data) + d.bytes);
      }
    }
  }
  for (int i = 0; i < g.n_inputs; ++i) {
    check_val(g.inputs[i], false);
    if (s.values[g.inputs[i]].rank < 0) fail(AC_ERR_SHAPE, "graph input without a static shape");
    s.inputs.push_back(g.inputs[i]);
  }
  for (int i = 0; i < g.n_outputs; ++i) { check_val(g.outputs[i], false); s.outputs.push_back(g.outputs[i]); }
  if (s.outputs.empty()) fail(AC_ERR_INVALID, "graph without outputs");
}

// The steps at the front that follow one another on the batch of the one input, image by image.
void plan_front(AcSession& s) {
  s.pieces = PiecePlan{};
  if (s.opt.disable_cuda_graph || s.opt.enable_profiling || s.inputs.size() != 1) return;
  const Value& in = s.values[s.inputs[0]];
  if (in.rank < 1 || s.storages[in.storage].weight) return;
  std::vector<FrontStep> front;
  for (const Step& st : s.steps) {
    if (!st.part || st.images != in.dims[0]) break;
    // Convolutions: 4 TB/s, or 80 TFLOP/s of the products.
    front.push_back({FrontStep::kLaunch + std::max(st.bytes / 4e6, st.flops / 80e6), st.rounds});
  }
  s.pieces = plan_pieces(front, (int)std::min<int64_t>(in.dims[0], 1 << 30), in.bytes());
}

// Where a piece's steps put the values that none but they read: a piece runs behind the one before it, so such a value needs
// the room of one piece, in what the arena has free beside the input and the values that the rest reads, which
// collect the whole batch. The arena does not grow for it; if it would have to, there are no pieces.
void plan_piece_slots(AcSession& s) {
  s.piece_slots.clear();
  if (!s.pieces.steps) return;
  const int last_front = s.pieces.steps - 1;
  std::vector<Slot> fixed, own;
  for (int i = 0; i < (int)s.storages.size(); ++i) {
    const Storage& st = s.storages[i];
    if (st.weight || st.last < 0 || st.first > last_front) continue;
    if (st.first < 0 || st.last > last_front) {
      fixed.push_back({st.bytes, 0, last_front, st.offset});
    } else {
      if (st.bytes % (size_t)s.pieces.images) { s.pieces = PiecePlan{}; s.piece_slots.clear(); return; }
      own.push_back({st.bytes / (size_t)s.pieces.images * (size_t)s.pieces.per, st.first, st.last, 0});
      s.piece_slots.push_back({i, 0});
    }
  }
  const size_t top = place_slots(own, fixed);
  for (size_t i = 0; i < own.size(); ++i) s.piece_slots[i].second = own[i].offset;
  if (top > s.arena_bytes) { s.pieces = PiecePlan{}; s.piece_slots.clear(); }
}

// Lifetimes by step index, then the placement.
void plan_arena(AcSession& s) {
  const int nsteps = (int)s.steps.size();
  for (Storage& st : s.storages) { st.first = 1 << 30; st.last = -1; }
  auto touch = [&](int sid, int step) {
    Storage& st = s.storages[sid];
    st.first = std::min(st.first, step);
    st.last = std::max(st.last, step);
  };
  for (int i = 0; i < nsteps; ++i) {
    for (int r : s.steps[i].reads) touch(r, i);
    for (int w : s.steps[i].writes) touch(w, i);
  }
  for (const Step& st : s.init_steps) {
    for (int r : st.reads) s.storages[r].pinned_live = s.storages[r].pinned_live || !s.storages[r].weight;
    for (int w : st.writes) s.storages[w].pinned_live = true;
  }
  size_t woff = 0;
  std::vector<int> live;
  std::vector<Slot> slots;
  for (int i = 0; i < (int)s.storages.size(); ++i) {
    Storage& st = s.storages[i];
    if (st.weight) {
      st.offset = woff;
      woff += align_up(st.bytes, 256);
      continue;
    }
    if (st.pinned_live) { st.first = -1; st.last = nsteps; }
    if (st.last < 0) continue;  // never touched
    live.push_back(i);
    slots.push_back({st.bytes, st.first, st.last, 0});
  }
  s.weight_bytes = woff;
  s.arena_bytes = std::max<size_t>(place_slots(slots), 256);
  for (size_t i = 0; i < live.size(); ++i) s.storages[live[i]].offset = slots[i].offset;
  plan_front(s);
  plan_piece_slots(s);
}

void upload_weights(AcSession& s, const AcGraphDesc& g) {
  AC_CUDA(cudaMalloc(&s.weights, std::max<size_t>(s.weight_bytes, 256)));
  for (int i = 0; i < g.n_inits; ++i) {
    const AcInitDesc& d = g.inits[i];
    if (!d.bytes) continue;
    void* dst = s.weights + s.storages[s.values[d.value].storage].offset;
    AC_CUDA(cudaMemcpyAsync(dst, d.data, d.bytes,
                            d.location == 1 ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                            s.stream));
  }
  AC_CUDA(cudaStreamSynchronize(s.stream));
  // Host pointers of large initializers belong to the caller: forget them.
  for (Value& v : s.values)
    if (v.is_init) v.host = v.host_owned.empty() ? nullptr : v.host_owned.data();
}

cudaError_t replay(AcSession* s, cudaStream_t st, int first, int last) {
  for (int i = first; i < last; ++i) {
    cudaError_t e = s->steps[i].fn(st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t replay(AcSession* s, cudaStream_t st) { return replay(s, st, 0, (int)s->steps.size()); }

template <typename Launches>
cudaError_t capture(AcSession* s, Launches launches, cudaGraph_t* graph, cudaGraphExec_t* exec) {
  cudaError_t e = cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  e = launches();
  const cudaError_t e2 = cudaStreamEndCapture(s->stream, graph);
  if (e != cudaSuccess) return e;
  if (e2 != cudaSuccess) return e2;
  return cudaGraphInstantiate(exec, *graph, 0);
}

cudaError_t capture(AcSession* s, int first, int last, cudaGraph_t* graph, cudaGraphExec_t* exec) {
  return capture(s, [&] { return replay(s, s->stream, first, last); }, graph, exec);
}

cudaError_t launch_all(AcSession* s) { return s->graph_exec ? cudaGraphLaunch(s->graph_exec, s->stream) : replay(s, s->stream); }

void destroy_segment(Segment& g) {
  if (g.exec) cudaGraphExecDestroy(g.exec);
  if (g.graph) cudaGraphDestroy(g.graph);
}

// A run on device buffers need not copy them in and out of the arena (115 of the 200 us that the
// tensor-op micrograph spent on the GPU): the kernels that read a graph input or write a graph
// output take the caller's pointers. Their launches cannot be in a graph then, so this is done where
// they are few and together: at most six segments, at most eight such steps (a launch
// costs the host about 3 us, a graph of any size 1 us).
void plan_segments(AcSession& s) {
  std::vector<char> io(s.storages.size(), 0);
  std::set<int> seen;
  auto bindable = [&](int v) {
    const int sid = s.values[v].storage;
    if (s.values[v].is_const || s.storages[sid].weight || !seen.insert(sid).second) return false;
    io[sid] = 1;
    return true;
  };
  for (int v : s.inputs)
    if (!bindable(v)) return;
  for (int v : s.outputs)
    if (!bindable(v)) return;
  for (const Step& st : s.init_steps)
    for (int w : st.writes)
      if (io[w]) return;
  std::vector<char> touches(s.steps.size(), 0);
  for (size_t i = 0; i < s.steps.size(); ++i) {
    for (int r : s.steps[i].reads) touches[i] |= io[r];
    for (int w : s.steps[i].writes) touches[i] |= io[w];
  }
  std::vector<Segment> segs = split_segments(touches);
  if (segs.size() > 6 || std::count(touches.begin(), touches.end(), 1) > 8) return;
  capture_segments(segs, [&](Segment& g) { return capture(&s, g.first, g.last, &g.graph, &g.exec); }, destroy_segment);
  (void)cudaGetLastError();
  s.segments = std::move(segs);
}

// The graphs of a run in pieces; without them the session runs its complete one.
void capture_pieces(AcSession& s) {
  const PiecePlan& p = s.pieces;
  if (!p.steps) return;
  cudaError_t e = cudaStreamCreateWithFlags(&s.up_stream, cudaStreamNonBlocking);
  for (int k = 0; k <= p.count() && e == cudaSuccess; ++k) {
    Segment g;
    if (k == p.count()) {
      e = capture(&s, p.steps, (int)s.steps.size(), &g.graph, &g.exec);
    } else {
      cudaEvent_t up = nullptr;
      e = cudaEventCreateWithFlags(&up, cudaEventDisableTiming);
      if (e == cudaSuccess) s.piece_up.push_back(up);
      auto launches = [&] {
        cudaError_t l = cudaSuccess;
        for (int i = 0; i < p.steps && l == cudaSuccess; ++i) l = s.steps[i].part(s.stream, p.begin(k), p.end(k) - p.begin(k));
        return l;
      };
      // The steps count from the batch's first image: that far in front of its slot a value of the piece's own begins.
      for (auto& [id, offset] : s.piece_slots) {
        const size_t image = s.storages[id].bytes / (size_t)p.images;
        s.storages[id].bound = reinterpret_cast<void*>(reinterpret_cast<uintptr_t>(s.arena) + offset - (size_t)p.begin(k) * image);
      }
      if (e == cudaSuccess) e = capture(&s, launches, &g.graph, &g.exec);
      for (auto& slot : s.piece_slots) s.storages[slot.first].bound = nullptr;
    }
    s.piece_graphs.push_back(g);
  }
  if (e == cudaSuccess) return;
  (void)cudaGetLastError();
  destroy_segments(s.piece_graphs, destroy_segment);
}

bool can_bind(const AcSession* s, const void* const* ins, void* const* outs) {
  if (s->segments.empty()) return false;
  auto local = [&](uintptr_t p) {
    cudaPointerAttributes pa{};
    if (cudaPointerGetAttributes(&pa, reinterpret_cast<const void*>(p)) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    return pa.type == cudaMemoryTypeDevice && pa.device == s->device;
  };
  return can_bind_buffers(
      (int)s->inputs.size(), [&](int i) { return std::make_pair(reinterpret_cast<uintptr_t>(ins[i]), s->values[s->inputs[i]].bytes()); },
      (int)s->outputs.size(), [&](int i) { return std::make_pair(reinterpret_cast<uintptr_t>(outs[i]), s->values[s->outputs[i]].bytes()); },
      local);
}

// The schedule with device buffers in place of the arena slots of the graph's inputs (and outputs,
// unless outs is null).
cudaError_t launch_bound(AcSession* s, const void* const* ins, void* const* outs) {
  auto bind = [&](bool on) {
    for (size_t i = 0; i < s->inputs.size(); ++i)
      s->storages[s->values[s->inputs[i]].storage].bound = on ? const_cast<void*>(ins[i]) : nullptr;
    for (size_t i = 0; outs && i < s->outputs.size(); ++i)
      s->storages[s->values[s->outputs[i]].storage].bound = on ? outs[i] : nullptr;
  };
  bind(true);
  cudaError_t e = cudaSuccess;
  for (const Segment& g : s->segments) {
    e = g.direct ? replay(s, s->stream, g.first, g.last) : cudaGraphLaunch(g.exec, s->stream);
    if (e != cudaSuccess) break;
  }
  bind(false);
  return e;
}

constexpr size_t kSmallIo = size_t(1) << 20;   // inputs (outputs) up to this go through the session's staging block

// Host inputs into the arena. Small ones are gathered in the page-locked block first: the driver's own
// path from pageable memory costs a call of up to 35 us there, the copy into the block 1 to 13.
cudaError_t upload_inputs(AcSession* s, const void* const* ins) {
  size_t at = 0;
  for (size_t i = 0; i < s->inputs.size(); ++i) {
    const size_t bytes = s->values[s->inputs[i]].bytes();
    void* dst = s->ptr(s->inputs[i]);
    cudaError_t e;
    if (s->stage_in) {
      std::memcpy(s->stage_in + at, ins[i], bytes);
      e = cudaMemcpyAsync(dst, s->stage_in + at, bytes, cudaMemcpyHostToDevice, s->stream);
      at += align_up(bytes, 256);
    } else {
      cudaPointerAttributes pa{};
      bool pageable = bytes > kSmallIo;
      if (pageable) {
        if (cudaPointerGetAttributes(&pa, ins[i]) == cudaSuccess) pageable = pa.type == cudaMemoryTypeUnregistered;
        else (void)cudaGetLastError();       // not left for the next launch to report
      }
      if (pageable && !s->host_stage) s->host_stage = HostStage::of_device(s->device);
      e = pageable && s->host_stage ? s->host_stage->upload(dst, ins[i], bytes, s->stream)
                                    : cudaMemcpyAsync(dst, ins[i], bytes, cudaMemcpyHostToDevice, s->stream);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// A whole run of the schedule from one large host input: the copies go on a stream of their own, and each piece's front steps
// start when its images are there (MobileNetV3-Large, 32 images: 470 us of copies in front of 750 of kernels, 250 of them here).
cudaError_t run_pieces(AcSession* s, const void* in) {
  const PiecePlan& p = s->pieces;
  const size_t bytes = s->values[s->inputs[0]].bytes(), image = bytes / (size_t)p.images;
  char* dst = static_cast<char*>(s->ptr(s->inputs[0]));
  int next = 0;
  auto sent = [&](size_t n) {
    cudaError_t e = cudaSuccess;
    for (; next < p.count() && (size_t)p.end(next) * image <= n && e == cudaSuccess; ++next) {
      e = cudaEventRecord(s->piece_up[next], s->up_stream);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(s->stream, s->piece_up[next], 0);
      if (e == cudaSuccess) e = cudaGraphLaunch(s->piece_graphs[next].exec, s->stream);
    }
    return e;
  };
  cudaPointerAttributes pa{};
  bool pageable = true;
  if (cudaPointerGetAttributes(&pa, in) == cudaSuccess) pageable = pa.type == cudaMemoryTypeUnregistered;
  else (void)cudaGetLastError();
  if (pageable && !s->host_stage) s->host_stage = HostStage::of_device(s->device);
  cudaError_t e = cudaSuccess;
  if (pageable && s->host_stage) {
    e = s->host_stage->upload(dst, in, bytes, s->up_stream, std::ref(sent));   // no allocation, so nothing thrown
  } else {
    for (int k = 0; k < p.count() && e == cudaSuccess; ++k) {
      const size_t from = (size_t)p.begin(k) * image, to = (size_t)p.end(k) * image;
      e = cudaMemcpyAsync(dst + from, static_cast<const char*>(in) + from, to - from, cudaMemcpyHostToDevice, s->up_stream);
      if (e == cudaSuccess) e = sent(to);
    }
  }
  return e == cudaSuccess ? cudaGraphLaunch(s->piece_graphs.back().exec, s->stream) : e;
}

}  // namespace

namespace ac {
// Lets other translation units of the library report through altius_cuda_last_error(NULL).
void set_thread_error(const std::string& msg) { g_create_error = msg; }
}  // namespace ac

namespace {

int set_err(AcSession* s, int status, const std::string& msg) {
  if (s) s->err = msg;
  else g_create_error = msg;
  return status;
}

std::unique_ptr<GraphCopy> copy_graph(const AcGraphDesc& g) {
  std::unique_ptr<GraphCopy> c(new GraphCopy());
  c->opset = g.opset_version;
  c->values.assign(g.values, g.values + g.n_values);
  c->nodes.resize(g.n_nodes);
  for (int i = 0; i < g.n_nodes; ++i) {
    const AcNodeDesc& d = g.nodes[i];
    GraphCopy::NodeCopy& n = c->nodes[i];
    n.op = d.op;
    if (d.n_inputs > 0) n.inputs.assign(d.inputs, d.inputs + d.n_inputs);
    if (d.n_outputs > 0) n.outputs.assign(d.outputs, d.outputs + d.n_outputs);
    if (d.n_ints > 0) n.ints.assign(d.ints, d.ints + d.n_ints);
    if (d.n_floats > 0) n.floats.assign(d.floats, d.floats + d.n_floats);
    n.has_name = d.name != nullptr;
    if (d.name) n.name = d.name;
  }
  if (g.n_inits > 0) c->inits.assign(g.inits, g.inits + g.n_inits);
  for (AcInitDesc& d : c->inits) d.data = nullptr;
  if (g.n_inputs > 0) c->inputs.assign(g.inputs, g.inputs + g.n_inputs);
  if (g.n_outputs > 0) c->outputs.assign(g.outputs, g.outputs + g.n_outputs);
  return c;
}

int create_session(const AcGraphDesc* graph, const AcOptions* options, AcSession** out, bool wide = false);

// What a session holds on the device for its runs.
void release_runs(AcSession* s) {
  if (s->graph_exec) cudaGraphExecDestroy(s->graph_exec);
  if (s->graph) cudaGraphDestroy(s->graph);
  s->graph_exec = nullptr;
  s->graph = nullptr;
  destroy_segments(s->segments, destroy_segment);
  destroy_segments(s->piece_graphs, destroy_segment);
  for (int k = 0; k < 2; ++k) {
    for (void*& p : s->staging[k]) {
      if (p) cudaFree(p);
      p = nullptr;
    }
  }
  if (s->arena) cudaFree(s->arena);
  if (s->weights) cudaFree(s->weights);
  s->arena = s->weights = nullptr;
}

// The session that takes over when an operand has left the fp16 range, built from the kept description; its
// initializers are read from this session's weight blob (or the host copies of the small ones). A plan with
// operands on the fixed scale that could do without it (|x| <= 255: the cluster GEMM, attention in blocks
// of keys) gives way to the same mode without these, whose range is 65504 there; only a plan that has left that
// too, to the 3xTF32 one. The session that is left keeps no memory.
int create_fallback(AcSession* s) {
  if (s->fallback) return AC_OK;
  if (!s->desc) return set_err(s, AC_ERR_CUDA, "an operand exceeds the fp16 range and no fallback description was kept");
  GraphCopy& c = *s->desc;
  std::vector<AcNodeDesc> nodes(c.nodes.size());
  for (size_t i = 0; i < c.nodes.size(); ++i) {
    GraphCopy::NodeCopy& n = c.nodes[i];
    nodes[i] = AcNodeDesc{n.op, (int32_t)n.inputs.size(), n.inputs.data(), (int32_t)n.outputs.size(), n.outputs.data(),
                          (int32_t)n.ints.size(), n.ints.data(), (int32_t)n.floats.size(), n.floats.data(),
                          n.has_name ? n.name.c_str() : nullptr};
  }
  std::vector<AcInitDesc> inits = c.inits;
  for (AcInitDesc& d : inits) {
    const Value& v = s->values[d.value];
    if (!v.host_owned.empty()) { d.location = 0; d.data = v.host_owned.data(); }
    else { d.location = 1; d.data = s->ptr(d.value); }
  }
  AcGraphDesc g{};
  g.opset_version = c.opset;
  g.n_values = (int32_t)c.values.size(); g.values = c.values.data();
  g.n_nodes = (int32_t)nodes.size(); g.nodes = nodes.data();
  g.n_inits = (int32_t)inits.size(); g.inits = inits.data();
  g.n_inputs = (int32_t)c.inputs.size(); g.inputs = c.inputs.data();
  g.n_outputs = (int32_t)c.outputs.size(); g.outputs = c.outputs.data();
  AcOptions o = s->opt;
  const bool same_mode = s->narrow && !s->wide;
  if (!same_mode) o.gemm_mode = 3;
  int rc = create_session(&g, &o, &s->fallback, same_mode);
  if (rc == -kGemmRangeCode) {
    o.gemm_mode = 3;
    rc = create_session(&g, &o, &s->fallback);
  }
  if (rc != AC_OK) return set_err(s, rc, "building the fallback failed: " + g_create_error);
  release_runs(s);
  return AC_OK;
}

// The error word after a run: 0 fine; the range code switches to the fallback session
// (returns 1: the caller re-runs there); anything else is a kernel that gave up a wait.
int check_err_word(AcSession* s) {
  const int code = *s->err_host;
  if (code == 0) return AC_OK;
  *s->err_host = 0;      // the stream has been drained: no kernel writes it now
  if (code == kGemmRangeCode && s->opt.gemm_mode == 0) {
    const int rc = create_fallback(s);
    if (rc != AC_OK) return rc;
    s->use_fallback = true;
    return 1;
  }
  return set_err(s, AC_ERR_CUDA, "a kernel gave up a bounded wait (code " + std::to_string(code) + ")");
}

int run_common(AcSession* s, const void* const* ins, void* const* outs, bool device_io) {
  if (!s) return set_err(s, AC_ERR_INVALID, "null argument");
  std::lock_guard<std::recursive_mutex> lock(s->run_mutex);
  if ((!ins && !s->inputs.empty()) || !outs) return set_err(s, AC_ERR_INVALID, "null argument");
  if (s->opt.plan_only) return set_err(s, AC_ERR_NO_DEVICE, "session was created with plan_only");
  // Every buffer is checked before anything is enqueued: an error return leaves no copy or
  // kernel in flight that could still write into the caller's memory.
  for (size_t i = 0; i < s->inputs.size(); ++i)
    if (!ins[i]) return set_err(s, AC_ERR_INVALID, "null input buffer");
  for (size_t i = 0; i < s->outputs.size(); ++i)
    if (!outs[i]) return set_err(s, AC_ERR_INVALID, "null output buffer");
  if (s->use_fallback) {
    const int rc = run_common(s->fallback, ins, outs, device_io);
    if (rc != AC_OK) s->err = s->fallback->err;
    return rc;
  }
  cudaError_t e = cudaSetDevice(s->device);
  if (e != cudaSuccess) return set_err(s, AC_ERR_CUDA, cudaGetErrorString(e));
  // An error after this point drains the stream before returning, for the same reason.
  auto fail_cuda = [&](const std::string& what, cudaError_t err) {
    if (s->up_stream) cudaStreamSynchronize(s->up_stream);
    cudaStreamSynchronize(s->stream);
    return set_err(s, AC_ERR_CUDA, what + cudaGetErrorString(err));
  };
  const bool bound = device_io && can_bind(s, ins, outs), in_pieces = !device_io && !s->piece_graphs.empty();
  if (!bound && !in_pieces) {
    if (device_io) {
      for (size_t i = 0; i < s->inputs.size() && e == cudaSuccess; ++i)
        e = cudaMemcpyAsync(s->ptr(s->inputs[i]), ins[i], s->values[s->inputs[i]].bytes(), cudaMemcpyDeviceToDevice, s->stream);
    } else {
      e = upload_inputs(s, ins);
    }
    if (e != cudaSuccess) return fail_cuda("input copy: ", e);
  }
  if (s->opt.enable_profiling) {
    const size_t n = s->steps.size();
    for (size_t i = 0; i < n; ++i) {
      // enable_profiling 2: every step starts on a cold L2 that holds no dirty lines.
      if (s->sweep_buf) l2_sweep_kernel<<<device_sm_count() * 8, 256, 0, s->stream>>>(
          reinterpret_cast<const float4*>(s->sweep_buf), kSweepBytes / 16, reinterpret_cast<float*>(s->sweep_buf));
      cudaEventRecord(s->events[2 * i], s->stream);
      e = s->steps[i].fn(s->stream);
      if (e != cudaSuccess) return fail_cuda(s->steps[i].kind + ": ", e);
      cudaEventRecord(s->events[2 * i + 1], s->stream);
    }
  } else {
    e = in_pieces ? run_pieces(s, ins[0]) : bound ? launch_bound(s, ins, outs) : launch_all(s);
    if (e != cudaSuccess) return fail_cuda(in_pieces ? "input copy and kernel launch: " : "kernel launch: ", e);
  }
  size_t at = 0;
  for (size_t i = 0; i < s->outputs.size() && !bound; ++i) {
    const size_t bytes = s->values[s->outputs[i]].bytes();
    const bool staged = !device_io && s->stage_out;
    e = cudaMemcpyAsync(staged ? s->stage_out + at : outs[i], s->ptr(s->outputs[i]), bytes,
                        device_io ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s->stream);
    if (e != cudaSuccess) return fail_cuda("output copy: ", e);
    at += align_up(bytes, 256);
  }
  e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return set_err(s, AC_ERR_CUDA, std::string("run: ") + cudaGetErrorString(e));
  if (const int rc = check_err_word(s)) return rc == 1 ? run_common(s, ins, outs, device_io) : rc;
  if (!device_io && s->stage_out) {
    at = 0;
    for (size_t i = 0; i < s->outputs.size(); ++i) {
      const size_t bytes = s->values[s->outputs[i]].bytes();
      std::memcpy(outs[i], s->stage_out + at, bytes);
      at += align_up(bytes, 256);
    }
  }
  if (s->opt.enable_profiling) {
    for (size_t i = 0; i < s->steps.size(); ++i) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, s->events[2 * i], s->events[2 * i + 1]);
      ProfileAcc& acc = s->profile[s->steps[i].kind];
      acc.launches += s->steps[i].launches;
      acc.ms += ms;
      acc.bytes += s->steps[i].bytes;
      acc.flops += s->steps[i].flops;
    }
  }
  return AC_OK;
}

}  // namespace

extern "C" {

int altius_cuda_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) return -AC_ERR_NO_DEVICE;
  return n;
}

}  // extern "C"

namespace {
int create_session(const AcGraphDesc* graph, const AcOptions* options, AcSession** out, bool wide) {
  if (!graph || !out) return set_err(nullptr, AC_ERR_INVALID, "null argument");
  *out = nullptr;
  AcSession* s = new AcSession();
  try {
    if (options) s->opt = *options;
    s->device = s->opt.device;
    s->wide = wide;
    if (s->opt.plan_only) {
      parse_graph(*s, *graph);
      infer_shapes(*s);
      lower_graph(*s);
      plan_arena(*s);
      *out = s;
      return AC_OK;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
      fail(AC_ERR_NO_DEVICE, "no CUDA device is visible: this backend has no CPU fallback");
    if (s->device < 0 || s->device >= ndev) fail(AC_ERR_NO_DEVICE, "device ordinal out of range");
    int major = 0;
    AC_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, s->device));
    if (major != 10)
      fail(AC_ERR_NO_DEVICE, "device is not sm_100 (the kernels are built for sm_100a only)");
    AC_CUDA(cudaSetDevice(s->device));
    AC_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    parse_graph(*s, *graph);
    infer_shapes(*s);
    {
      size_t in = 0, out = 0;
      for (int v : s->inputs) in += align_up(s->values[v].bytes(), 256);
      for (int v : s->outputs) out += align_up(s->values[v].bytes(), 256);
      if (in > kSmallIo) in = 0;
      if (out > kSmallIo) out = 0;
      AC_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&s->host_block), 256 + in + out, cudaHostAllocMapped));
      s->err_host = reinterpret_cast<int*>(s->host_block);
      *s->err_host = 0;
      AC_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&s->err_word), s->host_block, 0));
      if (in) s->stage_in = s->host_block + 256;
      if (out) s->stage_out = s->host_block + 256 + in;
    }
    lower_graph(*s);
    plan_arena(*s);
    AC_CUDA(cudaMalloc(&s->arena, s->arena_bytes));
    upload_weights(*s, *graph);
    for (Step& st : s->init_steps) AC_CUDA(st.fn(s->stream));
    AC_CUDA(cudaStreamSynchronize(s->stream));
    if (*s->err_host == kGemmRangeCode) fail(-kGemmRangeCode, "a constant operand exceeds the fp16 range");
    if (*s->err_host != 0) fail(AC_ERR_CUDA, "a kernel gave up a bounded wait while preparing constants");
    if (s->opt.gemm_mode == 0) s->desc = copy_graph(*graph);
    if (s->opt.enable_profiling) {
      s->events.resize(2 * s->steps.size());
      for (cudaEvent_t& ev : s->events) AC_CUDA(cudaEventCreate(&ev));
      if (s->opt.enable_profiling == 2) {
        AC_CUDA(cudaMalloc(&s->sweep_buf, kSweepBytes));
        AC_CUDA(cudaMemset(s->sweep_buf, 0, kSweepBytes));
      }
    } else if (!s->opt.disable_cuda_graph && !s->steps.empty()) {
      const cudaError_t e = capture(s, 0, (int)s->steps.size(), &s->graph, &s->graph_exec);
      if (e != cudaSuccess) fail(AC_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
      plan_segments(*s);
      capture_pieces(*s);
    }
  } catch (const BuildError& e) {
    set_err(nullptr, e.status, e.msg);
    altius_cuda_destroy(s);
    return e.status;
  } catch (const std::exception& e) {
    set_err(nullptr, AC_ERR_INVALID, e.what());
    altius_cuda_destroy(s);
    return AC_ERR_INVALID;
  }
  *out = s;
  return AC_OK;
}
}  // namespace

extern "C" {

int altius_cuda_create(const AcGraphDesc* graph, const AcOptions* options, AcSession** out) {
  int rc = create_session(graph, options, out);
  if (rc == -kGemmRangeCode) {
    // A weight does not fit the fp16 split: lower everything on the 3xTF32 path instead.
    AcOptions o{};
    if (options) o = *options;
    o.gemm_mode = 3;
    rc = create_session(graph, &o, out);
  }
  return rc;
}

int altius_cuda_run(AcSession* s, const void* const* ins, void* const* outs) {
  return run_common(s, ins, outs, false);
}

int altius_cuda_run_device(AcSession* s, const void* const* d_ins, void* const* d_outs) {
  return run_common(s, d_ins, d_outs, true);
}

int altius_cuda_run_batches(AcSession* s, int32_t n_batches, const void* const* ins, void* const* outs) {
  if (!s) return set_err(s, AC_ERR_INVALID, "bad argument");
  std::lock_guard<std::recursive_mutex> lock(s->run_mutex);
  if (n_batches < 0 || (!ins && !s->inputs.empty() && n_batches) || (!outs && n_batches))
    return set_err(s, AC_ERR_INVALID, "bad argument");
  if (s->opt.plan_only) return set_err(s, AC_ERR_NO_DEVICE, "session was created with plan_only");
  const size_t ni = s->inputs.size(), no = s->outputs.size();
  // All buffers of all batches are checked before the first copy is enqueued.
  for (size_t i = 0; i < (size_t)n_batches * ni; ++i)
    if (!ins[i]) return set_err(s, AC_ERR_INVALID, "null input buffer");
  for (size_t i = 0; i < (size_t)n_batches * no; ++i)
    if (!outs[i]) return set_err(s, AC_ERR_INVALID, "null output buffer");
  // Sessions that profile, or that have switched to their fallback plan, take the plain path.
  if (s->opt.enable_profiling || s->use_fallback || n_batches < 2) {
    for (int b = 0; b < n_batches; ++b) {
      const int rc = run_common(s, ins + (size_t)b * ni, outs + (size_t)b * no, false);
      if (rc != AC_OK) return rc;
    }
    return AC_OK;
  }
  cudaError_t e = cudaSetDevice(s->device);
  if (e == cudaSuccess && !s->copy_stream) {
    e = cudaStreamCreateWithFlags(&s->copy_stream, cudaStreamNonBlocking);
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
      s->staging[k].assign(ni, nullptr);
      for (size_t i = 0; i < ni && e == cudaSuccess; ++i)
        e = cudaMalloc(&s->staging[k][i], std::max<size_t>(s->values[s->inputs[i]].bytes(), 16));
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->staged[k], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->consumed[k], cudaEventDisableTiming);
    }
  }
  for (int b = 0; b < n_batches && e == cudaSuccess; ++b) {
    const int k = b & 1;
    // copy stream: inputs of batch b into staging set k (free again once batch b-2 has left it)
    if (b >= 2) e = cudaStreamWaitEvent(s->copy_stream, s->consumed[k], 0);
    for (size_t i = 0; i < ni && e == cudaSuccess; ++i) {
      const void* src = ins[(size_t)b * ni + i];
      e = cudaMemcpyAsync(s->staging[k][i], src, s->values[s->inputs[i]].bytes(), cudaMemcpyHostToDevice, s->copy_stream);
    }
    if (e == cudaSuccess) e = cudaEventRecord(s->staged[k], s->copy_stream);
    // compute stream: the schedule on the staging set, or staging -> arena and the schedule; outputs to the host
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s->stream, s->staged[k], 0);
    if (!s->segments.empty()) {
      if (e == cudaSuccess) e = launch_bound(s, s->staging[k].data(), nullptr);
      if (e == cudaSuccess) e = cudaEventRecord(s->consumed[k], s->stream);
    } else {
      for (size_t i = 0; i < ni && e == cudaSuccess; ++i)
        e = cudaMemcpyAsync(s->ptr(s->inputs[i]), s->staging[k][i], s->values[s->inputs[i]].bytes(),
                            cudaMemcpyDeviceToDevice, s->stream);
      if (e == cudaSuccess) e = cudaEventRecord(s->consumed[k], s->stream);
      if (e == cudaSuccess) e = launch_all(s);
    }
    for (size_t i = 0; i < no && e == cudaSuccess; ++i) {
      void* dst = outs[(size_t)b * no + i];
      e = cudaMemcpyAsync(dst, s->ptr(s->outputs[i]), s->values[s->outputs[i]].bytes(), cudaMemcpyDeviceToHost, s->stream);
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) {
    // Whatever was enqueued before the failure finishes before the caller gets its buffers back.
    if (s->copy_stream) cudaStreamSynchronize(s->copy_stream);
    cudaStreamSynchronize(s->stream);
    return set_err(s, AC_ERR_CUDA, std::string("run_batches: ") + cudaGetErrorString(e));
  }
  if (const int rc = check_err_word(s))   // out of fp16 range somewhere: all batches again on the fallback plan
    return rc == 1 ? altius_cuda_run_batches(s, n_batches, ins, outs) : rc;
  return AC_OK;
}

int altius_cuda_time_device_runs(AcSession* s, const void* const* d_ins, void* const* d_outs,
                                 int32_t iters, float* elapsed_ms) {
  if (!s) return set_err(s, AC_ERR_INVALID, "bad argument");
  std::lock_guard<std::recursive_mutex> lock(s->run_mutex);
  if (!elapsed_ms || iters <= 0 || !d_outs || (!d_ins && !s->inputs.empty()))
    return set_err(s, AC_ERR_INVALID, "bad argument");
  if (s->opt.plan_only) return set_err(s, AC_ERR_NO_DEVICE, "session was created with plan_only");
  if (s->opt.enable_profiling) return set_err(s, AC_ERR_INVALID, "not available on a profiling session");
  for (size_t i = 0; i < s->inputs.size(); ++i)
    if (!d_ins[i]) return set_err(s, AC_ERR_INVALID, "null input buffer");
  for (size_t i = 0; i < s->outputs.size(); ++i)
    if (!d_outs[i]) return set_err(s, AC_ERR_INVALID, "null output buffer");
  if (s->use_fallback) {
    const int rc = altius_cuda_time_device_runs(s->fallback, d_ins, d_outs, iters, elapsed_ms);
    if (rc != AC_OK) s->err = s->fallback->err;
    return rc;
  }
  cudaError_t e = cudaSetDevice(s->device);
  const bool bound = can_bind(s, d_ins, d_outs);
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  if (e == cudaSuccess) e = cudaEventCreate(&t0);
  if (e == cudaSuccess) e = cudaEventCreate(&t1);
  if (e == cudaSuccess) e = cudaEventRecord(t0, s->stream);
  for (int it = 0; it < iters && e == cudaSuccess; ++it) {
    if (bound) {
      e = launch_bound(s, d_ins, d_outs);
      continue;
    }
    for (size_t i = 0; i < s->inputs.size() && e == cudaSuccess; ++i)
      e = cudaMemcpyAsync(s->ptr(s->inputs[i]), d_ins[i], s->values[s->inputs[i]].bytes(),
                          cudaMemcpyDeviceToDevice, s->stream);
    if (e == cudaSuccess) e = launch_all(s);
    for (size_t i = 0; i < s->outputs.size() && e == cudaSuccess; ++i)
      e = cudaMemcpyAsync(d_outs[i], s->ptr(s->outputs[i]), s->values[s->outputs[i]].bytes(),
                          cudaMemcpyDeviceToDevice, s->stream);
  }
  if (e == cudaSuccess) e = cudaEventRecord(t1, s->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e == cudaSuccess && *s->err_host != 0) {
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
    const int rc = check_err_word(s);
    return rc == 1 ? altius_cuda_time_device_runs(s, d_ins, d_outs, iters, elapsed_ms) : rc;
  }
  if (e == cudaSuccess) e = cudaEventElapsedTime(elapsed_ms, t0, t1);
  if (t0) cudaEventDestroy(t0);
  if (t1) cudaEventDestroy(t1);
  if (e != cudaSuccess) return set_err(s, AC_ERR_CUDA, std::string("timed runs: ") + cudaGetErrorString(e));
  return AC_OK;
}

int altius_cuda_num_inputs(const AcSession* s) { return s ? (int)s->inputs.size() : -AC_ERR_INVALID; }
int altius_cuda_num_outputs(const AcSession* s) { return s ? (int)s->outputs.size() : -AC_ERR_INVALID; }
int altius_cuda_input_value(const AcSession* s, int32_t i) {
  return (s && i >= 0 && i < (int)s->inputs.size()) ? s->inputs[i] : -AC_ERR_INVALID;
}
int altius_cuda_output_value(const AcSession* s, int32_t i) {
  return (s && i >= 0 && i < (int)s->outputs.size()) ? s->outputs[i] : -AC_ERR_INVALID;
}

int altius_cuda_value_info(const AcSession* s, int32_t value, AcValueDesc* out) {
  if (!s || !out || value < 0 || value >= (int)s->values.size()) return AC_ERR_INVALID;
  const Value& v = s->values[value];
  out->elem_ty = v.elem_ty;
  out->rank = v.rank;
  for (int i = 0; i < AC_MAX_RANK; ++i) out->dims[i] = i < v.rank ? v.dims[i] : 0;
  return AC_OK;
}

int64_t altius_cuda_launches_per_run(const AcSession* s) {
  while (s && s->use_fallback) s = s->fallback;
  return s ? s->launches_per_run : -1;
}
uint64_t altius_cuda_arena_bytes(const AcSession* s) {
  while (s && s->use_fallback) s = s->fallback;
  return s ? s->arena_bytes : 0;
}

int altius_cuda_profile(AcSession* s, AcProfileEntry* entries, size_t* n) {
  while (s && s->use_fallback) s = s->fallback;
  if (!s || !n) return AC_ERR_INVALID;
  const size_t cap = *n;
  size_t i = 0;
  for (auto& kv : s->profile) {
    if (entries && i < cap) {
      AcProfileEntry& e = entries[i];
      std::memset(&e, 0, sizeof(e));
      std::snprintf(e.name, sizeof(e.name), "%s", kv.first.c_str());
      e.launches = kv.second.launches;
      e.total_ms = kv.second.ms;
      e.bytes = kv.second.bytes;
      e.flops = kv.second.flops;
    }
    ++i;
  }
  *n = i;
  return AC_OK;
}

int altius_cuda_schedule(const AcSession* s, AcProfileEntry* entries, size_t* n) {
  while (s && s->use_fallback) s = s->fallback;
  if (!s || !n) return AC_ERR_INVALID;
  const size_t cap = *n;
  for (size_t i = 0; i < s->steps.size() && entries && i < cap; ++i) {
    AcProfileEntry& e = entries[i];
    std::memset(&e, 0, sizeof(e));
    std::snprintf(e.name, sizeof(e.name), "%s", s->steps[i].kind.c_str());
    e.launches = s->steps[i].launches;
    e.bytes = s->steps[i].bytes;
    e.flops = s->steps[i].flops;
  }
  *n = s->steps.size();
  return AC_OK;
}

int altius_cuda_profile_reset(AcSession* s) {
  while (s && s->use_fallback) s = s->fallback;
  if (!s) return AC_ERR_INVALID;
  s->profile.clear();
  return AC_OK;
}

const char* altius_cuda_last_error(const AcSession* s) {
  return s ? s->err.c_str() : g_create_error.c_str();
}

void altius_cuda_destroy(AcSession* s) {
  if (!s) return;
  if (s->fallback) altius_cuda_destroy(s->fallback);
  if (s->stream) cudaSetDevice(s->device);
  release_runs(s);
  for (cudaEvent_t ev : s->events)
    if (ev) cudaEventDestroy(ev);
  if (s->sweep_buf) cudaFree(s->sweep_buf);
  for (int k = 0; k < 2; ++k) {
    if (s->staged[k]) cudaEventDestroy(s->staged[k]);
    if (s->consumed[k]) cudaEventDestroy(s->consumed[k]);
  }
  for (cudaEvent_t ev : s->piece_up) cudaEventDestroy(ev);
  if (s->copy_stream) cudaStreamDestroy(s->copy_stream);
  if (s->up_stream) cudaStreamDestroy(s->up_stream);
  if (s->host_block) cudaFreeHost(s->host_block);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

int altius_cuda_host_alloc(size_t bytes, void** out) {
  if (!out) return AC_ERR_INVALID;
  cudaError_t e = cudaHostAlloc(out, bytes ? bytes : 1, cudaHostAllocDefault);
  if (e != cudaSuccess) return set_err(nullptr, AC_ERR_CUDA, cudaGetErrorString(e));
  return AC_OK;
}

int altius_cuda_host_free(void* p) {
  if (!p) return AC_OK;
  return cudaFreeHost(p) == cudaSuccess ? AC_OK : AC_ERR_CUDA;
}

}  // extern "C"

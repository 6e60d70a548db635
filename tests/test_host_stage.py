"""The staged upload (host_stage.cpp) against a stand-in for the CUDA runtime: copies are memcpys, events
complete, stay pending or fail as the test says."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>
#include <thread>
#include <vector>
#include "host_stage.h"

static std::atomic<int> query_result{0}, whole_copies{0}, copies{0};
static std::atomic<bool> held{false};       // copies have been handed over but do not finish
static std::atomic<bool> no_memory{false};
void* operator new(size_t n) {
  void* p = no_memory ? nullptr : std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void* operator new[](size_t n) { return operator new(n); }
void* operator new(size_t n, const std::nothrow_t&) noexcept { return no_memory ? nullptr : std::malloc(n); }
void* operator new[](size_t n, const std::nothrow_t& t) noexcept { return operator new(n, t); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return held ? cudaErrorNotReady : (cudaError_t)query_result.load(); }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  ++copies;
  if (n > (size_t(1) << 20)) ++whole_copies;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
}

static bool right(const std::vector<char>& a, const std::vector<char>& b) { return std::memcmp(a.data(), b.data(), a.size()) == 0; }

int main(int argc, char** argv) {
  const std::string what = argv[1];
  if (what == "memory") {                    // nothing to be had: no stage, nothing thrown; later: the driver's path
    no_memory = true;
    if (ac::HostStage::of_device(1)) return 1;
    no_memory = false;
    auto s = ac::HostStage::of_device(1);
    std::vector<char> a(size_t(5) << 20, 7), b(size_t(5) << 20);
    no_memory = true;
    const bool ok = s->upload(b.data(), a.data(), a.size(), nullptr) == cudaSuccess && whole_copies == 1;
    no_memory = false;
    return ok && std::memcmp(a.data(), b.data(), a.size()) == 0 ? 0 : 2;
  }
  auto stage = ac::HostStage::of_device(0);
  const size_t big = (size_t(40) << 20) + 12345;
  std::vector<char> src(big), dst(big), dst2(big);
  for (size_t i = 0; i < big; ++i) src[i] = (char)(i * 2654435761u >> 13);
  if (what == "copies") {
    for (size_t n : {size_t(1), size_t(63), size_t(1) << 20, (size_t(1) << 20) + 1, (size_t(12) << 20), (size_t(13) << 20) + 7, big}) {
      std::fill(dst.begin(), dst.end(), 0);
      if (stage->upload(dst.data(), src.data(), n, nullptr) != cudaSuccess || std::memcmp(dst.data(), src.data(), n)) return 1;
    }
    return 0;
  }
  if (what == "fault") {                     // an earlier fault on the device: the query says so
    query_result = (int)cudaErrorLaunchFailure;
    if (stage->upload(dst.data(), src.data(), big, nullptr) != cudaErrorLaunchFailure) return 1;
    query_result = 0;
    return stage->upload(dst.data(), src.data(), big, nullptr) == cudaSuccess && right(dst, src) ? 0 : 2;
  }
  if (what == "two") {                       // while one upload holds the ring another one goes on
    held = true;
    std::atomic<bool> first{false};
    std::thread t([&] { (void)stage->upload(dst.data(), src.data(), big, nullptr); first = true; });
    while (copies < 12) std::this_thread::yield();           // the ring is full
    const bool ok = stage->upload(dst2.data(), src.data(), big, nullptr) == cudaSuccess && right(dst2, src) && !first;
    held = false;
    t.join();
    return ok && right(dst, src) ? 0 : 1;
  }
  if (what == "sent") {                      // told of what has been handed over, in order; an error ends the upload and is passed on
    size_t last = 0;
    int calls = 0;
    auto told = [&](size_t n) { const bool ok = n > last && std::memcmp(dst.data(), src.data(), n) == 0; last = n; ++calls; return ok ? cudaSuccess : cudaErrorUnknown; };
    if (stage->upload(dst.data(), src.data(), big, nullptr, std::ref(told)) != cudaSuccess || last != big || calls != 41) return 1;
    copies = 0;
    auto stop = [&](size_t n) { return n < (size_t(4) << 20) ? cudaSuccess : cudaErrorLaunchFailure; };
    if (stage->upload(dst.data(), src.data(), big, nullptr, std::ref(stop)) != cudaErrorLaunchFailure || copies != 4) return 2;
    return stage->upload(dst.data(), src.data(), big, nullptr) == cudaSuccess && right(dst, src) ? 0 : 3;
  }
  return 9;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("stage")
    (d / "h.cpp").write_text(HARNESS)
    csrc = os.path.join(ROOT, "altius_b200", "csrc")
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", csrc, "-I", os.path.join(cuda, "include"), str(d / "h.cpp"),
                    os.path.join(csrc, "host_stage.cpp"), "-o", str(d / "h")], check=True)
    return str(d / "h")


@pytest.mark.parametrize("what", ["copies", "fault", "two", "memory", "sent"])
def test_staged_upload(harness, what):
    assert subprocess.run([harness, what], timeout=30).returncode == 0

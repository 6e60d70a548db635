// The squeeze-and-excite block of the MobileNets up to its gate,
//   GlobalAveragePool -> 1 x 1 Conv + act -> 1 x 1 Conv + act,
// in one kernel. As three launches (pool, and two products of a few rows against up to 960 x 240
// weights) it took 20 to 145 us per block of the network at a batch of one: one or two blocks of a
// GEMM walked K alone. The work is 0.5 MFLOP and 2 MB of weights per image, so it is bound by
// latency: a cluster of eight blocks shares one to four images; every block computes an eighth of the hidden units from
// the channels' means and sends them to all eight, then finishes its eighth of the gate. The means come from the
// depthwise convolution in front where that makes them; else every block pools its eighth of the channels
// and leaves them in the shared memory of all eight first.
// Several images per cluster (when the clusters of one image no longer fit the SMs at once) read the weights once for all of them.
// Per block of a MobileNetV3-Large at batch one, from the end of the kernel in front: 8.0 us with the pool, a cluster barrier
// behind each exchange and cold code; 4.0 with given means, sends that count on an mbarrier and a pass ahead of the wait.
// At 32 images 11.4 -> 8.0 over the eight blocks.
#include <cooperative_groups.h>

#include "cluster_send.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"

namespace cg = cooperative_groups;

namespace ac {
namespace {

constexpr int kCluster = 8, kThreads = 1024, kWarps = kThreads / 32;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sum8(float v) {   // over eight neighbouring lanes
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, acc))));
}
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }

template <int G, bool POOL, bool WARM>
__global__ void __launch_bounds__(kThreads) squeeze_excite_kernel(const SqueezeExciteParams p) {
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) uint64_t sent;
  float* mean = smem;                 // [G][c]
  float* hid = smem + G * p.c;        // [G][s]
  cg::cluster_group cl = cg::this_cluster();
  const int rank = blockIdx.z, n0 = blockIdx.x * G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, quarter = lane >> 3;
  const int c = p.c, s = p.s, hw = (int)p.hw;
  const int cper = (c + kCluster - 1) / kCluster, c0 = rank * cper, c1 = min(c, c0 + cper), cn = max(c1 - c0, 0);
  if (threadIdx.x == 0) {             // the hidden units, four bytes each, from all blocks
    tc::mbar_init(&sent, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_arrive_expect_tx(&sent, (uint32_t)(G * s * 4));
  }
  __syncthreads();
  cl.barrier_arrive();
  // The warp's first row of W1 is requested before anything else; eight loads of a lane cover 1024 inputs.
  const int j0 = rank + kCluster * warp;
  float4 w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = lane * 4 + i * 128;
    w[i] = j0 < s && k < c ? ldg4(p.w1 + (long long)j0 * c + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  pdl_trigger();

  // Pass 0 has no channels and no hidden units: it brings the code into the instruction cache while the
  // kernel in front still runs.
#pragma unroll 1
  for (int pass = WARM ? 0 : 1; pass < 2; ++pass) {
    const bool now = !WARM || pass == 1;
    const int js = now ? s : min(s, j0 + 1), cs = now ? c : 0, ss = now ? s : 0, ce = now ? c1 : 0;
    if (now) {
      pdl_wait();
      cl.barrier_wait();              // every block of the cluster runs: its shared memory may be written
    }
    if (POOL) {
      // ---- means of this block's channels: eight lanes each ----
      const bool v4 = (hw & 3) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
      for (int i = warp * 4; i < G * cn && now; i += kWarps * 4) {
        const int item = i + quarter, g = min(item / max(cn, 1), G - 1), ch = c0 + item - g * cn;
        const bool ok = item < G * cn && n0 + g < p.n;
        float acc = 0.f;
        if (ok) {
          const float* row = p.x + ((long long)(n0 + g) * c + ch) * hw;
          if (v4) {
#pragma unroll 8
            for (int j = sub * 4; j < hw; j += 32) {
              const float4 v = *reinterpret_cast<const float4*>(row + j);
              acc = __fadd_rn(acc, __fadd_rn(__fadd_rn(v.x, v.y), __fadd_rn(v.z, v.w)));
            }
          } else {
#pragma unroll 8
            for (int j = sub; j < hw; j += 8) acc = __fadd_rn(acc, row[j]);
          }
        }
        acc = __fdiv_rn(sum8(acc), (float)hw);
        if (item < G * cn) cl.map_shared_rank(mean, sub)[g * c + ch] = acc;
      }
      if (now) cl.sync();
    } else {
      // ---- the means of the cluster's images, made by the kernel in front ----
      const int there = min(G, p.n - n0) * c;
      for (int i = threadIdx.x * 4; i < G * cs; i += kThreads * 4)
        *reinterpret_cast<float4*>(mean + i) =
            i < there ? *reinterpret_cast<const float4*>(p.mean + (long long)n0 * c + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      __syncthreads();
    }

    // ---- hidden units rank, rank + 8, ...: a warp each, all G images at once ----
    for (int j = j0; j < js; j += kCluster * kWarps) {
      float acc[G];
#pragma unroll
      for (int g = 0; g < G; ++g) acc[g] = 0.f;
      const float* row = p.w1 + (long long)j * c;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = lane * 4 + i * 128;
        if (k >= cs) continue;
        const float4 wv = j == j0 ? w[i] : ldg4(row + k);
#pragma unroll
        for (int g = 0; g < G; ++g) acc[g] = dot4(wv, lds4(mean + g * c + k), acc[g]);
      }
      for (int k = 1024 + lane * 4; k < cs; k += 128) {
        const float4 wv = ldg4(row + k);
#pragma unroll
        for (int g = 0; g < G; ++g) acc[g] = dot4(wv, lds4(mean + g * c + k), acc[g]);
      }
      float v = 0.f;                    // lane g * 8 + q sends image g to block q
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float u = warp_sum(acc[g]);
        if (quarter == g) v = u;
      }
      if (p.b1) v = __fadd_rn(v, ld_plain(p.b1 + j));
      v = apply_act(p.act1, v, p.alpha1, p.beta1);
      if (quarter < G && now) send1(cluster_addr(hid + quarter * s + j, sub), cluster_addr(&sent, sub), v);
    }
    // The lane's part of its first row of W2: eight loads cover 256 hidden units.
    const int ch0 = c0 + warp * 4 + quarter;
    if (now) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = sub * 4 + i * 32;
        w[i] = ch0 < c1 && k < s ? ldg4(p.w2 + (long long)ch0 * s + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (!__all_sync(0xffffffffu, wait_sent(&sent, 0))) atomicExch(p.err, 72);
    }

    // ---- gate: eight lanes per channel ----
    for (int ch = ch0; ch - quarter < (now ? c1 : ch0 + 1); ch += kWarps * 4) {
      float acc[G];
#pragma unroll
      for (int g = 0; g < G; ++g) acc[g] = 0.f;
      if (ch < ce) {
        const float* row = p.w2 + (long long)ch * s;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int k = sub * 4 + i * 32;
          if (k >= ss) continue;
          const float4 wv = ch == ch0 ? w[i] : ldg4(row + k);
#pragma unroll
          for (int g = 0; g < G; ++g) acc[g] = dot4(wv, lds4(hid + g * s + k), acc[g]);
        }
        for (int k = 256 + sub * 4; k < ss; k += 32) {
          const float4 wv = ldg4(row + k);
#pragma unroll
          for (int g = 0; g < G; ++g) acc[g] = dot4(wv, lds4(hid + g * s + k), acc[g]);
        }
      }
      float v = 0.f;                    // lane sub == g finishes image g
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float u = sum8(acc[g]);
        if (sub == g) v = u;
      }
      if (ch < ce && sub < G && n0 + sub < p.n) {
        if (p.b2) v = __fadd_rn(v, ld_plain(p.b2 + ch));
        p.gate[(long long)(n0 + sub) * c + ch] = apply_act(p.act2, v, p.alpha2, p.beta2);
      }
    }
  }
}

constexpr int kMaxVector = 3072;      // c + s

template <int G, bool POOL, bool WARM>
cudaError_t launch_form(const SqueezeExciteParams& p, cudaStream_t st) {
  // Four images' vectors are 48 KB, which a kernel may use unasked only without the barrier beside them.
  static unsigned long long done = 0;
  if (cudaError_t e = ensure_dynamic_smem(squeeze_excite_kernel<G, POOL, WARM>, G * kMaxVector * (int)sizeof(float), &done)) return e;
  return launch_pdl(squeeze_excite_kernel<G, POOL, WARM>, dim3((unsigned)((p.n + G - 1) / G), 1, kCluster), dim3(kThreads),
                    (size_t)G * (p.c + p.s) * sizeof(float), st, kCluster, p);
}

template <int G>
cudaError_t launch_g(const SqueezeExciteParams& p, cudaStream_t st) {
  // A block fills an SM: it starts under the kernel in front, and has the time for a pass ahead, only while most SMs are free.
  if (!p.mean) return launch_form<G, true, false>(p, st);
  if (G == 1 && 2 * p.n * kCluster <= device_sm_count()) return launch_form<1, false, true>(p, st);
  return launch_form<G, false, false>(p, st);
}

inline bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

bool squeeze_excite_supported(const SqueezeExciteParams& p) {
  // Rows of the weights (and of the vectors in shared memory) are read as float4s.
  return p.c >= 8 && (p.c % 4) == 0 && p.s >= 4 && (p.s % 4) == 0 && p.c + p.s <= kMaxVector && p.n >= 1 && p.hw >= 1 &&
         p.hw < (1 << 28);
}

cudaError_t launch_squeeze_excite(const SqueezeExciteParams& p, cudaStream_t st) {
  if (!squeeze_excite_supported(p) || !al16(p.w1) || !al16(p.w2) || (p.mean && !al16(p.mean))) return cudaErrorInvalidValue;
  // Clusters that run at once (a block of 1024 threads fills an SM). One more takes a second round: 32 images
  // as 16 clusters of two 19 to 26 us, as 8 clusters of four 12 to 21, as 11 of three another 0.6 to 4 less.
  const int per_wave = cluster_slots(kCluster);
  if (p.n <= per_wave) return launch_g<1>(p, st);
  if (p.n <= 2 * per_wave) return launch_g<2>(p, st);
  return p.n <= 3 * per_wave ? launch_g<3>(p, st) : launch_g<4>(p, st);
}

}  // namespace ac

// Depthwise convolutions (square K x K filter, K 3 or 5, stride 1, dilation 1) over whole planes in shared memory.
// Restates the per-(batch, group) products of crates/session_interpreter/src/conv2d.rs:145-209 for one
// channel a group.
//
// A stencil on global memory reads every value K times (four pixels of a row a thread) and every filter once for
// four pixels: 65 loads a thread of a 5 x 5 filter on rows that are no whole float4s, and the load unit, not
// memory, bounded it. Here a block copies whole neighbouring planes into shared memory (one contiguous piece of the
// tensor, read as float4s), and a thread walks down one output column with the K output rows that an input
// row contributes to in registers: K shared-memory loads and K * K products a pixel, the filter in registers. The
// taps of a result are added in the order of the generic kernel and those outside the plane are
// skipped, so the results are the same bits.
#include "depthwise_planes_shape.h"
#include "kernels.h"
#include "pdl.cuh"
#include "plane_means.cuh"
#include "ref_math.cuh"

namespace ac {
namespace {

using namespace depthwise_planes;

struct PlanesDev {
  const float* x; const float* w; const float* bias; float* out; float* means;
  int planes, c, ih, iw, oh, ow, pad_t, pad_l;
  int per, stride, rows, segs;   // see Shape
  float act_alpha, act_beta;
};

template <int K, int ACT>
__global__ void __launch_bounds__(kMaxThreads) depthwise_planes_kernel(const PlanesDev p) {
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, plane0 = blockIdx.x * p.per, here = min(p.per, p.planes - plane0);
  const int ox = tid % p.ow, t = tid / p.ow, seg = t % p.segs, pl = t / p.segs;
  const bool live = pl < here;
  const int plane = plane0 + (live ? pl : 0), ch = plane % p.c;
  float wk[K][K];
#pragma unroll
  for (int i = 0; i < K * K; ++i) wk[i / K][i % K] = __ldg(p.w + ch * (K * K) + i);   // constants where the launch overlaps
  const float bv = p.bias ? __ldg(p.bias + ch) : 0.f;
  pdl_trigger();
  pdl_wait();

  // ---- planes -> shared memory ----
  const int ihw = p.ih * p.iw, count = here * ihw, gap = p.stride - ihw;
  const float* src = p.x + (long long)plane0 * ihw;        // 16-byte aligned: planes of whole float4s, or four a block
  if ((ihw & 3) == 0) {
#pragma unroll 4
    for (int i = tid * 4; i < count; i += blockDim.x * 4) {
      const float4 v = *reinterpret_cast<const float4*>(src + i);
      *reinterpret_cast<float4*>(smem + i + i / ihw * gap) = v;
    }
  } else {
#pragma unroll 4
    for (int i = tid * 4; i < count; i += blockDim.x * 4) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (i + 3 < count) {
        const float4 f = *reinterpret_cast<const float4*>(src + i);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] = i + j < count ? src[i + j] : 0.f;
      }
      const int q = i / ihw;
      int left = (q + 1) * ihw - i, at = i + q * gap;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (left == 0) { left = ihw; at += gap; }
        if (i + j < count) smem[at] = v[j];
        ++at; --left;
      }
    }
  }
  __syncthreads();

  // ---- one output column, `rows` pixels of it ----
  float sum = 0.f;
  if (live) {
    const int ix = ox - p.pad_l;
    bool in[K];
#pragma unroll
    for (int j = 0; j < K; ++j) in[j] = ix + j >= 0 && ix + j < p.iw;
    const float* col = smem + pl * p.stride + ix;
    const int y0 = seg * p.rows, y1 = min(p.oh, y0 + p.rows);
    float* dst = p.out + ((long long)plane * p.oh) * p.ow + ox;
    float acc[K];                             // of the output rows in work
#pragma unroll
    for (int a = 0; a < K; ++a) acc[a] = 0.f;
    // Output row q - a collects the taps a of input row q - pad_t.
    for (int q = y0; q < y1 + K - 1; ++q) {
      const int iy = q - p.pad_t;
      if (iy >= 0 && iy < p.ih) {
        float v[K];
#pragma unroll
        for (int j = 0; j < K; ++j) v[j] = in[j] ? col[iy * p.iw + j] : 0.f;
#pragma unroll
        for (int a = 0; a < K; ++a)
#pragma unroll
          for (int j = 0; j < K; ++j)
            if (in[j]) acc[a] = fmaf(wk[a][j], v[j], acc[a]);
      }
      if (q - (K - 1) >= y0) {                // output row q - (K - 1) has its last tap
        float r = acc[K - 1];
        if (p.bias) r = __fadd_rn(bv, r);
        r = apply_act(ACT, r, p.act_alpha, p.act_beta);
        dst[(q - (K - 1)) * p.ow] = r;
        sum = __fadd_rn(sum, r);
      }
#pragma unroll
      for (int a = K - 1; a > 0; --a) acc[a] = acc[a - 1];
      acc[0] = 0.f;
    }
  }
  if (!p.means) return;
  __shared__ float sums[kMaxThreads];
  sums[tid] = sum;
  __syncthreads();
  plane_means(sums, (unsigned)here, (unsigned)(p.segs * p.ow), p.means, (unsigned)plane0, (unsigned)p.planes, p.oh * p.ow);
}

template <int K>
cudaError_t launch_act(const PlanesDev& d, int act, int threads, size_t smem, int overlap, cudaStream_t st) {
  const dim3 grid((unsigned)((d.planes + d.per - 1) / d.per)), block((unsigned)threads);
  auto go = [&](auto kernel, unsigned long long* done) -> cudaError_t {
    if (cudaError_t e = ensure_dynamic_smem(kernel, (int)kMaxSmem, done)) return e;
    return launch_pdl(kernel, grid, block, smem, st, overlap, d);
  };
  static unsigned long long done[3] = {0, 0, 0};
  switch (act) {
    case ACT_NONE: return go(depthwise_planes_kernel<K, ACT_NONE>, &done[0]);
    case ACT_RELU: return go(depthwise_planes_kernel<K, ACT_RELU>, &done[1]);
    case ACT_HARDSWISH: return go(depthwise_planes_kernel<K, ACT_HARDSWISH>, &done[2]);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_depthwise_planes(const ConvParams& q, int images, const float* x, const float* w, const float* bias, float* out,
                                    float* means, bool constants, cudaStream_t st) {
  if (!supported(q) || (reinterpret_cast<uintptr_t>(x) & 15)) return cudaErrorInvalidValue;
  const Shape sh = pick_shape(q, device_sm_count());
  PlanesDev d{};
  d.x = x; d.w = w; d.bias = bias; d.out = out; d.means = means;
  d.planes = images * q.c; d.c = q.c; d.ih = q.ih; d.iw = q.iw; d.oh = q.oh; d.ow = q.ow; d.pad_t = q.pad_t; d.pad_l = q.pad_l;
  d.per = sh.per; d.stride = sh.stride; d.rows = sh.rows; d.segs = sh.segs;
  d.act_alpha = q.act_alpha; d.act_beta = q.act_beta;
  const int overlap = constants ? 1 : 0;
  return q.kh == 3 ? launch_act<3>(d, q.act, sh.threads, sh.smem, overlap, st) : launch_act<5>(d, q.act, sh.threads, sh.smem, overlap, st);
}

}  // namespace ac

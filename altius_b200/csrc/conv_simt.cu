// fp32 convolutions on the CUDA cores, as implicit products
//   out[b] (oc x pixels) = W (oc x k) * col[b] (k x pixels)
// over the columns of ALL images at once (column = image * pixels + pixel), with bias, activation
// and residual in the epilogue. Restates what the reference does per image with im2col +
// cblas_sgemm (crates/session_interpreter/src/conv2d.rs:81-209).
//
// For convolutions of up to a few million products (the layers of a small CNN at a batch of one, of
// a digit classifier): 28 K products per SM or fewer are 0.1 us of FMAs, so such a layer costs
// what its launch, its one or two round trips to memory and the chain of its K steps cost. A
// 128 x 128-tile GEMM gives it one to seven blocks that walk K alone (24 to 110 us per layer for
// the 1 x 1 and 3 x 3 layers of a MobileNet at batch one, 13 us for 25 taps into 8 channels of
// 28 x 28); here the work is cut until it covers the SMs, and nothing is split, padded, transposed
// or written as a column buffer first: planes of any size and filters with a window (their
// addresses come from a table in shared memory) take the same loop.
//
// Shape: a group of 128 threads (8 x 16) owns a tile of 8 TM output channels x 64 columns, TM x 4
// in registers. A block has four such groups, which share the tile and take interleaved slices of
// every K step of 32; a cluster of up to eight blocks shares the tile in the same way over ranges
// of K. Partial sums meet in (distributed) shared memory in a fixed order, so results do not
// depend on timing. Operands arrive by cp.async in a ring of four stages; the filter's part of
// the first stages is requested before the kernel in front has finished.
#include <cooperative_groups.h>

#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"

namespace cg = cooperative_groups;

namespace ac {
namespace {

constexpr int GROUP = 128;
enum Load { LOAD_VEC = 0, LOAD_SCALAR, LOAD_WINDOW };

struct ConvDev {
  const float* x;
  const float* wt;          // [k][ldw]: the filter matrix transposed, rows padded with zeros
  float* out;
  const float* bias;
  const float* res;
  const float* gate;        // [batch][k] factor of each input channel, or null
  int ldw, m, k, hw, n;     // n = batch * hw columns
  long long x_batch, out_batch;
  int ih, iw, ow, kh, kw, sh, sw, dh, dw, pt, pl;
  int act;
  float act_alpha, act_beta;
  int kper;                 // K steps per block of the cluster
  int early;                // the filter is a constant: read ahead of pdl_wait
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// Copies 16 / 4 bytes, or writes zeros when !ok (the source is then not read).
__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, bool ok) {
  const int n = ok ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A thread's TM rows are neighbours (TM 2 or 4): one aligned load.
template <int TM>
__device__ __forceinline__ void load_a(const float* row, int ty, float (&a)[TM]) {
  static_assert(TM == 2 || TM == 4, "rows per thread");
  if (TM == 4) {
    const float4 v = *reinterpret_cast<const float4*>(row + ty * 4);
    a[0] = v.x; a[1] = v.y; a[TM - 2] = v.z; a[TM - 1] = v.w;
  } else {
    const float2 v = *reinterpret_cast<const float2*>(row + ty * 2);
    a[0] = v.x; a[1] = v.y;
  }
}

__device__ __forceinline__ float finish(const ConvDev& p, float v, float bias) {
  if (p.bias) v = __fadd_rn(v, bias);
  if (p.act == ACT_NONE) return v;
  if (p.act == ACT_RELU) return fmaxf(v, 0.f);
  if (p.act == ACT_HARDSWISH) return __fmul_rn(v, hard_sigmoid_ref(v, p.act_alpha, p.act_beta));
  return apply_act(p.act, v, p.act_alpha, p.act_beta);
}

// Four neighbouring columns of one output row.
template <int LOAD>
__device__ __forceinline__ void store_quad(const ConvDev& p, int row, int col, float4 v) {
  if (row >= p.m || col >= p.n) return;
  const float bias = p.bias ? ld_plain(p.bias + row) : 0.f;
  v.x = finish(p, v.x, bias); v.y = finish(p, v.y, bias); v.z = finish(p, v.z, bias); v.w = finish(p, v.w, bias);
  if (LOAD == LOAD_VEC) {   // planes are whole float4s: the four columns lie in one image
    const int b = col / p.hw;
    const long long at = b * p.out_batch + (long long)row * p.hw + (col - b * p.hw);
    if (p.res) {
      const float4 r = *reinterpret_cast<const float4*>(p.res + at);
      v.x = __fadd_rn(v.x, r.x); v.y = __fadd_rn(v.y, r.y); v.z = __fadd_rn(v.z, r.z); v.w = __fadd_rn(v.w, r.w);
    }
    *reinterpret_cast<float4*>(p.out + at) = v;
    return;
  }
  const float e[4] = {v.x, v.y, v.z, v.w};
  int b = col / p.hw, px = col - b * p.hw;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (col + j >= p.n) return;
    const long long at = b * p.out_batch + (long long)row * p.hw + px;
    p.out[at] = p.res ? __fadd_rn(e[j], p.res[at]) : e[j];
    if (++px == p.hw) { px = 0; ++b; }
  }
}

constexpr int TN = 4, WK = 4;
constexpr int BN = 16 * TN, BK = 32, T = GROUP * WK, S = 4;
template <int TM>
struct Cfg {
  static constexpr int BM = 8 * TM;
  static constexpr int STAGE = BK * (BM + BN);                 // floats
  static constexpr int QUADS = TM * TN / 4;                    // float4s of results per thread
  static constexpr int PARTS = WK * GROUP * TM * TN;           // floats of partial sums
  static constexpr int FLOATS = S * STAGE > PARTS ? S * STAGE : PARTS;
};

template <int TM, int LOAD>
__global__ void __launch_bounds__(T) conv_simt_kernel(const ConvDev p) {
  using C = Cfg<TM>;
  constexpr int BM = C::BM, QUADS = C::QUADS;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, g = tid / GROUP, t = tid % GROUP, lane = t & 31, warp = t >> 5;
  // A warp covers 4 x 8 threads of the group's 8 x 16: one wavefront per shared-memory load.
  const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int nkt = (p.k + BK - 1) / BK;
  const int kt0 = blockIdx.z * p.kper, kt1 = min(nkt, kt0 + p.kper), kts = kt1 - kt0;

  // k -> (offset of the tap inside an image, its row and column) for filters with a window.
  int2* tab = reinterpret_cast<int2*>(smem + C::FLOATS);
  if (LOAD == LOAD_WINDOW) {
    const int taps = p.kh * p.kw;
    for (int k = tid; k < p.k; k += T) {
      const int c = k / taps, r = k - c * taps, fy = r / p.kw * p.dh, fx = (r % p.kw) * p.dw;
      tab[k] = make_int2(c * p.ih * p.iw + fy * p.iw + fx, fy << 16 | fx);
    }
    __syncthreads();
  }
  pdl_trigger();

  // The column(s) this thread loads are the same in every K step.
  constexpr int CPR = LOAD == LOAD_VEC ? BN / 4 : BN, RPP = T / CPR, ROWS = BK / RPP;   // columns a row, rows a pass
  static_assert(T % CPR == 0 && BK % RPP == 0, "loader shape");
  const int lc = tid % CPR, lr = tid / CPR;
  const int col = n0 + (LOAD == LOAD_VEC ? 4 * lc : lc);
  const bool col_ok = col < p.n;
  const int cb = col_ok ? col / p.hw : 0, px = col_ok ? col - cb * p.hw : 0;
  const float* xcol = p.x + cb * p.x_batch;
  int iy0 = 0, ix0 = 0;
  if (LOAD == LOAD_WINDOW) {
    const int oy = px / p.ow;
    iy0 = oy * p.sh - p.pt;
    ix0 = (px - oy * p.ow) * p.sw - p.pl;
    xcol += (long long)iy0 * p.iw + ix0;
  } else {
    xcol += px;
  }
  const float* gcol = p.gate ? p.gate + (long long)cb * p.k : nullptr;

  auto load_w = [&](int s, int kt) {
    float* As = smem + s * C::STAGE;
    const int k0 = kt * BK;
#pragma unroll
    for (int i = tid; i < BK * (BM / 4); i += T) {
      const int r = i / (BM / 4), c4 = (i % (BM / 4)) * 4;
      const bool ok = k0 + r < p.k && m0 + c4 < p.ldw;
      cp16(As + r * BM + c4, ok ? p.wt + (long long)(k0 + r) * p.ldw + m0 + c4 : p.wt, ok);
    }
  };
  auto load_x = [&](int s, int kt) {
    float* Bs = smem + s * C::STAGE + BK * BM;
    const int k0 = kt * BK;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int r = lr + i * RPP, k = k0 + r;
      if (LOAD == LOAD_VEC) {
        const bool ok = col_ok && k < p.k;
        cp16(Bs + r * BN + 4 * lc, ok ? xcol + (long long)k * p.hw : p.x, ok);
      } else if (LOAD == LOAD_SCALAR) {
        const bool ok = col_ok && k < p.k;
        cp4(Bs + r * BN + lc, ok ? xcol + (long long)k * p.hw : p.x, ok);
      } else {
        bool ok = col_ok && k < p.k;
        const int2 e = ok ? tab[k] : make_int2(0, 0);
        const int iy = iy0 + (e.y >> 16), ix = ix0 + (e.y & 0xffff);
        ok = ok && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
        cp4(Bs + r * BN + lc, ok ? xcol + e.x : p.x, ok);
      }
    }
  };
  float gv[ROWS];                          // factors of the elements this thread loads next
  auto fetch_gate = [&](int kt) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int k = kt * BK + lr + i * RPP;
      gv[i] = col_ok && k < p.k ? gcol[k] : 0.f;
    }
  };

  if (!p.early) pdl_wait();                // packed by a step in front
#pragma unroll
  for (int s = 0; s < S - 1; ++s)
    if (s < kts) load_w(s, kt0 + s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < S - 1; ++s) {
    if (s < kts) load_x(s, kt0 + s);
    cp_commit();
  }
  if (p.gate && kts > 0) fetch_gate(kt0);

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int it = 0; it < kts; ++it) {
    const int s = it % S;
    cp_wait<S - 2>();
    if (p.gate) {                          // own elements only: visible without a barrier
      float* Bs = smem + s * C::STAGE + BK * BM;
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        float* e = Bs + (lr + i * RPP) * BN + (LOAD == LOAD_VEC ? 4 * lc : lc);
        if (LOAD == LOAD_VEC) {
          float4 v = *reinterpret_cast<float4*>(e);
          v.x = __fmul_rn(v.x, gv[i]); v.y = __fmul_rn(v.y, gv[i]); v.z = __fmul_rn(v.z, gv[i]); v.w = __fmul_rn(v.w, gv[i]);
          *reinterpret_cast<float4*>(e) = v;
        } else {
          *e = __fmul_rn(*e, gv[i]);
        }
      }
      if (it + 1 < kts) fetch_gate(kt0 + it + 1);
    }
    __syncthreads();                       // stage s complete for all; stage of step it - 1 is free
    if (it + S - 1 < kts) {
      load_w((it + S - 1) % S, kt0 + it + S - 1);
      load_x((it + S - 1) % S, kt0 + it + S - 1);
    }
    cp_commit();
    const float* As = smem + s * C::STAGE + g * (BK / WK) * BM;
    const float* Bs = smem + s * C::STAGE + BK * BM + g * (BK / WK) * BN;
#pragma unroll
    for (int kk = 0; kk < BK / WK; ++kk) {
      float a[TM], b[TN];
      load_a<TM>(As + kk * BM, ty, a);
      const float4 v = *reinterpret_cast<const float4*>(Bs + kk * BN + tx * 4);
      b[0] = v.x; b[1] = v.y; b[2] = v.z; b[3] = v.w;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
  }
  cp_wait<0>();

  const int parts = gridDim.z;             // blocks of the cluster
  // Partial sums: row i of thread t of group g at [(g * TM + i) * 128 + t].
  float4* part = reinterpret_cast<float4*>(smem);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
    part[(g * TM + i) * GROUP + t] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  cg::cluster_group cl = cg::this_cluster();
  if (parts > 1) cl.sync();
  else __syncthreads();
  // Each block of the cluster finishes its share of the quads.
  const int share = QUADS * GROUP / parts, base = blockIdx.z * share;
  for (int v = tid; v < share; v += T) {
    const int e = base + v, q = e / GROUP, tt = e % GROUP;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < parts; ++r) {
      const float4* src = parts > 1 ? cl.map_shared_rank(part, r) : part;
#pragma unroll
      for (int w = 0; w < WK; ++w) {
        const float4 u = src[w * QUADS * GROUP + e];
        sum.x = __fadd_rn(sum.x, u.x); sum.y = __fadd_rn(sum.y, u.y);
        sum.z = __fadd_rn(sum.z, u.z); sum.w = __fadd_rn(sum.w, u.w);
      }
    }
    const int ll = tt & 31, ww = tt >> 5;
    const int yy = (ww >> 1) * 4 + (ll >> 3), xx = (ww & 1) * 8 + (ll & 7);
    store_quad<LOAD>(p, m0 + yy * TM + q, n0 + xx * 4, sum);
  }
  if (parts > 1) cl.sync();                // no block leaves while others read its sums
}

template <int TM, int LOAD>
cudaError_t launch_one(const ConvDev& p, int split, cudaStream_t st) {
  using C = Cfg<TM>;
  static unsigned long long done = 0;
  const size_t smem = C::FLOATS * sizeof(float) + (LOAD == LOAD_WINDOW ? (size_t)p.k * sizeof(int2) : 0);
  if (cudaError_t e = ensure_dynamic_smem(conv_simt_kernel<TM, LOAD>, 96 << 10, &done)) return e;
  const dim3 grid((unsigned)((p.n + BN - 1) / BN), (unsigned)((p.m + C::BM - 1) / C::BM), (unsigned)split);
  return launch_pdl(conv_simt_kernel<TM, LOAD>, grid, dim3(T), smem, st, split, p);
}

__global__ void pack_filter_kernel(const float* __restrict__ w, float* __restrict__ wt, int m, int k, int ldw) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)k * ldw) return;
  const int kk = (int)(i / ldw), r = (int)(i % ldw);
  wt[i] = r < m ? w[(long long)r * k + kk] : 0.f;
}

inline bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

cudaError_t launch_pack_filter(const float* w, float* wt, int64_t m, int64_t k, cudaStream_t st) {
  const int64_t ldw = conv_simt_ldw(m), n = k * ldw;
  if (n == 0) return cudaSuccess;
  pack_filter_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w, wt, (int)m, (int)k, (int)ldw);
  return cudaGetLastError();
}

bool conv_simt_supported(const ConvParams& q) {
  const int64_t k = (int64_t)q.c * q.kh * q.kw, cols = (int64_t)q.n * q.oh * q.ow;
  return q.group == 1 && k >= 1 && k <= 4096 && cols < (1ll << 30) && (int64_t)q.c * q.ih * q.iw < (1ll << 30) &&
         q.kh * q.dh < 32768 && q.kw * q.dw < 32768 && q.oc <= 65535 * 16;
}

cudaError_t launch_conv_simt(const ConvParams& q, const float* x, const float* wt, const float* bias, const float* gate,
                             const float* residual, float* out, bool constants, cudaStream_t st) {
  ConvDev p{};
  p.x = x; p.wt = wt; p.out = out; p.bias = bias; p.res = residual; p.gate = gate;
  p.ldw = (int)conv_simt_ldw(q.oc); p.m = q.oc; p.k = q.c * q.kh * q.kw; p.hw = q.oh * q.ow; p.n = q.n * p.hw;
  if (p.m == 0 || p.n == 0) return cudaSuccess;
  p.x_batch = (long long)q.c * q.ih * q.iw; p.out_batch = (long long)p.m * p.hw;
  p.ih = q.ih; p.iw = q.iw; p.ow = q.ow; p.kh = q.kh; p.kw = q.kw; p.sh = q.sh; p.sw = q.sw; p.dh = q.dh; p.dw = q.dw;
  p.pt = q.pad_t; p.pl = q.pad_l;
  p.early = constants;
  p.act = q.act; p.act_alpha = q.act_alpha; p.act_beta = q.act_beta;
  const bool window = q.kh != 1 || q.kw != 1 || q.sh != 1 || q.sw != 1 || q.pad_t || q.pad_l || q.oh != q.ih || q.ow != q.iw;
  if (window && gate) return cudaErrorInvalidValue;
  const bool vec = !window && (p.hw % 4) == 0 && al16(x) && al16(out) && (!residual || al16(residual));
  // Tiles of 32 channels when they already give every SM one; else of 16, and K cut over the
  // blocks of a cluster (at least one K step each) until the SMs have about one block each.
  const int sms = device_sm_count(), nkt = (p.k + BK - 1) / BK;
  auto tiles = [&](int bm) { return (long long)((p.n + BN - 1) / BN) * ((p.m + bm - 1) / bm); };
  const bool tall = tiles(32) >= sms;
  int split = 1;
  while (split < 8 && 2 * split <= nkt && 2 * split * tiles(tall ? 32 : 16) <= sms + sms / 4) split *= 2;
  p.kper = (nkt + split - 1) / split;
  if (tall) {
    if (window) return launch_one<4, LOAD_WINDOW>(p, split, st);
    return vec ? launch_one<4, LOAD_VEC>(p, split, st) : launch_one<4, LOAD_SCALAR>(p, split, st);
  }
  if (window) return launch_one<2, LOAD_WINDOW>(p, split, st);
  return vec ? launch_one<2, LOAD_VEC>(p, split, st) : launch_one<2, LOAD_SCALAR>(p, split, st);
}

}  // namespace ac

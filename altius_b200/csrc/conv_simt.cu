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
// Shape: a tile is 16 output channels x 64 columns. Each of a block's eight warps holds all of it in registers (4 x 8 a
// thread) and takes four rows of every K step of 32, loaded by itself: no barrier between loads and sums. A
// cluster of up to eight blocks shares the tile over ranges of K. Partial sums meet in (distributed)
// shared memory in a fixed order, so results do not depend on timing; the blocks of a cluster send
// theirs with stores that count on the receiver's mbarrier. The filter's part of the first stages is
// requested before the kernel in front has finished.
//
// Measured, per launch in a MobileNetV3-Large at batch one, from the end of the kernel in front: 40 -> 120 at 28 x 28 4.8 us
// -> 3.1; 672 -> 112 at 14 x 14 with a gate 10.7 -> 6.1; 960 -> 160 at 7 x 7 with a gate 12.7 -> 5.2. Before that: four groups of 128
// threads on 2 x 4 results each with a barrier of the block in every K step (1100 clocks a step against 800: shared memory
// hands a warp 128 bytes a clock, so the bytes loaded per product count), planes by 4-byte cp.async, the gate fetched one step
// ahead, remote partial sums read block by block, the residual behind them. (A pass over zeros ahead of the wait, to have the code in
// the instruction cache, gave a MobileNetV3-Large nothing, 312.8 us with it and 312.0 without, and cost 0.5 us of a launch behind
// another of these and 2 us behind a kernel that lets nothing start early.) Beside the kernel before it, which had tiles of 32 channels too:
// over 74 layers of 3000 to 60000 pixels and 3 to 48 channels 0.85 of its time, the worst 1.09 (12 images of 24 x 33 x 33 and 6 channels,
// 5.5 us -> 6.0; nine of 32 x 57 x 57 and 3 9.6 -> 10.0), over 125 of all sizes 0.80.
#include <cooperative_groups.h>

#include "cluster_send.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"

namespace cg = cooperative_groups;

namespace ac {
namespace {

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
  int early;                // the filter and the bias are constants: read ahead of pdl_wait
  int* err;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// Copies 16 bytes, or writes zeros when !ok (the source is then not read).
__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void add4(float4& s, float4 v) {
  s.x = __fadd_rn(s.x, v.x); s.y = __fadd_rn(s.y, v.y); s.z = __fadd_rn(s.z, v.z); s.w = __fadd_rn(s.w, v.w);
}

__device__ __forceinline__ float finish(const ConvDev& p, float v, float bias) {
  if (p.bias) v = __fadd_rn(v, bias);
  if (p.act == ACT_NONE) return v;
  if (p.act == ACT_RELU) return fmaxf(v, 0.f);
  if (p.act == ACT_HARDSWISH) return __fmul_rn(v, hard_sigmoid_ref(v, p.act_alpha, p.act_beta));
  return apply_act(p.act, v, p.act_alpha, p.act_beta);
}

// Four neighbouring columns of one output row: where they lie, and what is added behind the activation.
template <int LOAD>
struct Quad {
  long long at = 0;
  int live = 0;                            // columns that exist; LOAD_VEC: planes are whole float4s, all four or none
  int left = 0;                            // pixels up to the end of the first column's plane
  float res[4] = {0.f, 0.f, 0.f, 0.f};
  float bias = 0.f;

  __device__ __forceinline__ void place(const ConvDev& p, bool mine, int row, int col) {
    if (!mine || row >= p.m || col >= p.n) return;
    const int b = col / p.hw, px = col - b * p.hw;
    at = b * p.out_batch + (long long)row * p.hw + px;
    live = LOAD == LOAD_VEC ? 4 : min(4, p.n - col);
    left = p.hw - px;
    if (p.bias) bias = ld_plain(p.bias + row);
  }
  // The j-th column's element; the last pixel of an image's plane is followed by the next image's first.
  template <typename F>
  __device__ __forceinline__ void each(const ConvDev& p, F f) const {
    long long a = at;
    int l = left;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j < live) f(j, a);
      ++a;
      if (--l == 0) { l = p.hw; a += p.out_batch - p.hw; }
    }
  }
  __device__ __forceinline__ void fetch(const ConvDev& p) {
    if (!p.res) return;
    if (LOAD == LOAD_VEC) {
      if (!live) return;
      const float4 r = *reinterpret_cast<const float4*>(p.res + at);
      res[0] = r.x; res[1] = r.y; res[2] = r.z; res[3] = r.w;
    } else {
      each(p, [&](int j, long long a) { res[j] = p.res[a]; });
    }
  }
  __device__ __forceinline__ void store(const ConvDev& p, float4 v) const {
    float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = finish(p, e[j], bias);
      if (p.res) e[j] = __fadd_rn(e[j], res[j]);
    }
    if (LOAD == LOAD_VEC) {
      if (live) *reinterpret_cast<float4*>(p.out + at) = make_float4(e[0], e[1], e[2], e[3]);
    } else {
      each(p, [&](int j, long long a) { p.out[a] = e[j]; });
    }
  }
};

constexpr int BM = 16, BN = 64, BK = 32, WARPS = 8, T = 32 * WARPS, KW = BK / WARPS, S = 4;
constexpr int SLICE = KW * (BM + BN);                      // floats: a warp's rows of a K step
constexpr int QUADS = BM * BN / 4;                         // float4s of the tile
constexpr int RING = WARPS * S * SLICE, PARTS = WARPS * QUADS * 4;
constexpr int FLOATS = (RING > PARTS ? RING : PARTS) + QUADS * 4;
static_assert(QUADS == T, "a thread adds one float4 of the result up");

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

template <int LOAD>
__global__ void __launch_bounds__(T, 2) conv_simt_kernel(const ConvDev p) {
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) uint64_t sent;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = lane >> 3, tx = lane & 7;          // 4 rows x (2 x 4) columns a thread, the tile a warp
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int nkt = (p.k + BK - 1) / BK;
  const int kt0 = blockIdx.z * p.kper, kt1 = min(nkt, kt0 + p.kper), kts = kt1 - kt0;
  const int parts = gridDim.z, rank = blockIdx.z;   // blocks of the cluster
  const int share = QUADS / parts;                  // float4s of the result that a block finishes

  // k -> (offset of the tap inside an image, its row and column) for filters with a window.
  int2* tab = reinterpret_cast<int2*>(smem + FLOATS);
  if (LOAD == LOAD_WINDOW) {
    const int taps = p.kh * p.kw;
    for (int k = tid; k < p.k; k += T) {
      const int c = k / taps, r = k - c * taps, fy = r / p.kw * p.dh, fx = (r % p.kw) * p.dw;
      tab[k] = make_int2(c * p.ih * p.iw + fy * p.iw + fx, fy << 16 | fx);
    }
  }
  if (tid == 0 && parts > 1) {
    tc::mbar_init(&sent, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_arrive_expect_tx(&sent, (uint32_t)(parts * share * 16));
  }
  __syncthreads();
  pdl_trigger();
  cg::cluster_group cl = cg::this_cluster();
  if (parts > 1) cl.barrier_arrive();

  // The column(s) this lane loads are the same in every row: one float4 of every second row, or columns lane and lane + 32.
  constexpr int COLS = LOAD == LOAD_VEC ? 1 : 2, ROWS = LOAD == LOAD_VEC ? KW / 2 : KW, FL = LOAD == LOAD_VEC ? 4 : 1;
  const int lr = LOAD == LOAD_VEC ? lane >> 4 : 0, lc = LOAD == LOAD_VEC ? (lane & 15) * 4 : lane;
  constexpr int RSTEP = LOAD == LOAD_VEC ? 2 : 1;
  const float *xcol[COLS], *gcol[COLS];
  int iy0[COLS], ix0[COLS];
  bool col_ok[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    const int col = n0 + lc + 32 * c;
    col_ok[c] = col < p.n;
    const int b = col_ok[c] ? col / p.hw : 0, px = col_ok[c] ? col - b * p.hw : 0;
    xcol[c] = p.x + b * p.x_batch;
    iy0[c] = ix0[c] = 0;
    if (LOAD == LOAD_WINDOW) {
      const int oy = px / p.ow;
      iy0[c] = oy * p.sh - p.pt;
      ix0[c] = (px - oy * p.ow) * p.sw - p.pl;
      xcol[c] += (long long)iy0[c] * p.iw + ix0[c];
    } else {
      xcol[c] += px;
    }
    gcol[c] = p.gate ? p.gate + (long long)b * p.k : nullptr;
  }

  // Everything a warp multiplies it has loaded itself: rows [4 warp, 4 warp + 4) of every K step, so no barrier of
  // the block stands between the loads and the sums.
  float* mine = smem + warp * (S * SLICE);
  auto load_w = [&](int s, int kt) {
    const int r = lane >> 2, c4 = (lane & 3) * 4, k = kt * BK + warp * KW + r;
    if (lane < KW * (BM / 4)) {
      const bool ok = k < p.k && m0 + c4 < p.ldw;
      cp16(mine + s * SLICE + r * BM + c4, ok ? p.wt + (long long)k * p.ldw + m0 + c4 : p.wt, ok);
    }
  };
  // The planes' part of a K step goes through registers: a warp's cp.async of 4 bytes a lane took 15 clocks of the SM to
  // issue whatever its width, 24 of them in front of the first step 5600 clocks.
  struct Piece { float x[ROWS][COLS][FL], gate[LOAD == LOAD_WINDOW ? 1 : ROWS][COLS]; };   // no gate with a window
  auto fetch = [&](Piece& u, int kt, bool go) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        const int k = kt * BK + warp * KW + lr + i * RSTEP;
        bool ok = go && col_ok[c] && k < p.k;
        if (LOAD != LOAD_WINDOW) u.gate[i][c] = p.gate && ok ? gcol[c][k] : 1.f;
        if (LOAD == LOAD_VEC) {
          const float4 v = ok ? *reinterpret_cast<const float4*>(xcol[c] + (long long)k * p.hw) : make_float4(0.f, 0.f, 0.f, 0.f);
          u.x[i][c][0] = v.x; u.x[i][c][FL > 1 ? 1 : 0] = v.y; u.x[i][c][FL > 1 ? 2 : 0] = v.z; u.x[i][c][FL > 1 ? 3 : 0] = v.w;
        } else if (LOAD == LOAD_SCALAR) {
          u.x[i][c][0] = ok ? xcol[c][(long long)k * p.hw] : 0.f;
        } else {
          const int2 e = ok ? tab[k] : make_int2(0, 0);
          const int iy = iy0[c] + (e.y >> 16), ix = ix0[c] + (e.y & 0xffff);
          ok = ok && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
          u.x[i][c][0] = ok ? xcol[c][e.x] : 0.f;
        }
      }
  };
  auto put = [&](int s, const Piece& u) {
    float* Bs = mine + s * SLICE + KW * BM;
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        float v[FL];
#pragma unroll
        for (int j = 0; j < FL; ++j)
          v[j] = LOAD != LOAD_WINDOW && p.gate ? __fmul_rn(u.x[i][c][j], u.gate[LOAD == LOAD_WINDOW ? 0 : i][c]) : u.x[i][c][j];
        float* at = Bs + (lr + i * RSTEP) * BN + lc + 32 * c;
        if (LOAD == LOAD_VEC) *reinterpret_cast<float4*>(at) = make_float4(v[0], v[FL > 1 ? 1 : 0], v[FL > 1 ? 2 : 0], v[FL > 1 ? 3 : 0]);
        else *at = v[0];
      }
  };

  // Float4 e of the tile: row (e / 8 % 4) * 4 + e / 64, columns from e / 32 % 2 * 32 + e % 8 * 4.
  Quad<LOAD> quad;                                                 // what this thread finishes
  float4* part = reinterpret_cast<float4*>(smem);                  // [warps][QUADS], over the ring
  float4* recv = reinterpret_cast<float4*>(smem + FLOATS) - QUADS; // [parts][share], written by the cluster's blocks

  if (!p.early) pdl_wait();                // filter or bias come from a step in front
#pragma unroll 1
  for (int s = 0; s < S - 1; ++s)
    if (s < kts) load_w(s, kt0 + s);
  cp_commit();
  {
    const int e = rank * share + tid;
    quad.place(p, tid < share, m0 + (e >> 3 & 3) * 4 + (e >> 6), n0 + (e >> 5 & 1) * 32 + (e & 7) * 4);
  }

  pdl_wait();
  {
    Piece u[S - 1];
#pragma unroll
    for (int s = 0; s < S - 1; ++s)
      if (s < kts) fetch(u[s], kt0 + s, true);
    quad.fetch(p);
#pragma unroll
    for (int s = 0; s < S - 1; ++s)
      if (s < kts) put(s, u[s]);
  }

  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);

  for (int it = 0; it < kts; ++it) {
    const int s = it % S;
    if (it == 0) cp_wait<0>();             // the filter's part of the first stages
    else cp_wait<S - 2>();
    __syncwarp();                          // stage s complete for the warp; stage of step it - 1 is free
    Piece u;
    const bool more = it + S - 1 < kts;
    if (more) load_w((it + S - 1) % S, kt0 + it + S - 1);
    cp_commit();
    fetch(u, kt0 + it + S - 1, more);
    const float* As = mine + s * SLICE;
    const float* Bs = As + KW * BM;
#pragma unroll
    for (int kk = 0; kk < KW; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(As + kk * BM + ty * 4);
      const float4 b0 = *reinterpret_cast<const float4*>(Bs + kk * BN + tx * 4);
      const float4 b1 = *reinterpret_cast<const float4*>(Bs + kk * BN + 32 + tx * 4);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
        acc[i][0] = fma2(aa, make_float2(b0.x, b0.y), acc[i][0]);
        acc[i][1] = fma2(aa, make_float2(b0.z, b0.w), acc[i][1]);
        acc[i][2] = fma2(aa, make_float2(b1.x, b1.y), acc[i][2]);
        acc[i][3] = fma2(aa, make_float2(b1.z, b1.w), acc[i][3]);
      }
    }
    if (more) put((it + S - 1) % S, u);
  }

  // The warps' sums, then the blocks': both in order. A block sends each other one its share.
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      part[warp * QUADS + (2 * i + h) * 32 + lane] = make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
  __syncthreads();
  float4 sum = part[tid];
#pragma unroll
  for (int w = 1; w < WARPS; ++w) add4(sum, part[w * QUADS + tid]);
  if (parts > 1) {
    cl.barrier_wait();                     // every block of the cluster runs and has announced what it waits for
    const int owner = tid / share;
    send4(cluster_addr(recv + rank * share + tid - owner * share, owner), cluster_addr(&sent, owner), sum);
    if (tid < share) {
      if (!wait_sent(&sent, 0)) atomicExch(p.err, 71);
      sum = recv[tid];
      for (int r = 1; r < parts; ++r) add4(sum, recv[r * share + tid]);
    }
  }
  quad.store(p, sum);
}

template <int LOAD>
cudaError_t launch_one(const ConvDev& p, int split, cudaStream_t st) {
  static unsigned long long done = 0;
  const size_t smem = FLOATS * sizeof(float) + (LOAD == LOAD_WINDOW ? (size_t)p.k * sizeof(int2) : 0);
  if (cudaError_t e = ensure_dynamic_smem(conv_simt_kernel<LOAD>, 96 << 10, &done)) return e;
  const dim3 grid((unsigned)((p.n + BN - 1) / BN), (unsigned)((p.m + BM - 1) / BM), (unsigned)split);
  return launch_pdl(conv_simt_kernel<LOAD>, grid, dim3(T), smem, st, split, p);
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
                             const float* residual, float* out, bool constants, int* err_word, cudaStream_t st) {
  ConvDev p{};
  p.x = x; p.wt = wt; p.out = out; p.bias = bias; p.res = residual; p.gate = gate;
  p.ldw = (int)conv_simt_ldw(q.oc); p.m = q.oc; p.k = q.c * q.kh * q.kw; p.hw = q.oh * q.ow; p.n = q.n * p.hw;
  if (p.m == 0 || p.n == 0) return cudaSuccess;
  p.x_batch = (long long)q.c * q.ih * q.iw; p.out_batch = (long long)p.m * p.hw;
  p.ih = q.ih; p.iw = q.iw; p.ow = q.ow; p.kh = q.kh; p.kw = q.kw; p.sh = q.sh; p.sw = q.sw; p.dh = q.dh; p.dw = q.dw;
  p.pt = q.pad_t; p.pl = q.pad_l;
  p.early = constants;
  p.err = err_word;
  p.act = q.act; p.act_alpha = q.act_alpha; p.act_beta = q.act_beta;
  const bool window = q.kh != 1 || q.kw != 1 || q.sh != 1 || q.sw != 1 || q.pad_t || q.pad_l || q.oh != q.ih || q.ow != q.iw;
  if (window && gate) return cudaErrorInvalidValue;
  const bool vec = !window && (p.hw % 4) == 0 && al16(x) && al16(out) && (!residual || al16(residual));
  // K is cut over the blocks of a cluster (at least one K step each) until the SMs have about one block each.
  const int sms = device_sm_count(), nkt = (p.k + BK - 1) / BK;
  const long long tiles = (long long)((p.n + BN - 1) / BN) * ((p.m + BM - 1) / BM);
  int split = 1;
  while (split < 8 && 2 * split <= nkt && 2 * split * tiles <= sms + sms / 4) split *= 2;
  p.kper = (nkt + split - 1) / split;
  if (window) return launch_one<LOAD_WINDOW>(p, split, st);
  return vec ? launch_one<LOAD_VEC>(p, split, st) : launch_one<LOAD_SCALAR>(p, split, st);
}

}  // namespace ac

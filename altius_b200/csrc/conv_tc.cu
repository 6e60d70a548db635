// fp32-level convolutions on the tensor cores (tcgen05, 3xTF32), as implicit products
//   out[b] (oc x pixels) = W (oc x k) * col[b] (k x pixels)
// over the columns of ALL images at once (column = image * pixels + pixel), with bias, activation and
// residual in the epilogue. Restates what the reference does per image with im2col + cblas_sgemm
// (crates/session_interpreter/src/conv2d.rs:81-209).
//
// The PIXELS are the rows (M = 128) of the MMA and the output channels its N (any multiple of 16
// up to 256): a tile is full whatever the channel count, and since tensor memory hands a thread
// one row, a warp holds 32 neighbouring pixels of one channel and stores the NCHW result as
// whole 128-byte lines straight from registers. The planes are read by ordinary loads, 32
// pixels of one channel a warp, split into TF32 hi / lo in registers and written to shared memory as
// K-major tiles; so planes of any size (7 x 7 = 49 floats a row, which TMA cannot address) and
// filters with a window (addresses from a table in shared memory, no column buffer) take the same
// path, and a squeeze-and-excite gate is one multiply in front of the split. The filter arrives
// split, blocked and swizzled (prepared once) with one bulk copy per K step.
//
// What bounds it: the layers of the CNNs have K of 16 to 960 and move 0.5 to 100 FMAs per byte. The
// wide planes are bound by HBM if loads, MMAs and stores of different tiles overlap: two blocks share
// an SM and each walks tiles; the loads of the next tile are in flight, and its MMAs run into a second
// buffer of accumulators where tensor memory has one, while a tile is finished and stored. The narrow planes (7 x 7, 14 x 14) have few tiles
// and a long K and are bound by the K steps of one SM (1500 to 2000 clocks each: loads, split, stores and
// barrier one behind the other): there a cluster of up to eight blocks cuts K and adds its accumulators up through
// distributed shared memory, in rank order.
#include <cooperative_groups.h>

#include <algorithm>

#include "conv_tc_shape.h"
#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace ac {
namespace {

using namespace tc;
using namespace conv_tc;

constexpr int kLoaders = 256, kThreads = kLoaders + 32;

struct ConvTcDev {
  const float* x;
  const float* w;           // [n tile][K step][hi: bn x 32 | lo: bn x 32], rows of 128 bytes, swizzled
  float* out;
  const float* bias;
  const float* res;
  const float* gate;        // [batch][k] factor of each input channel, or null
  int m, k, hw, n;          // n = batch * hw columns
  int bn, stages, kper;     // channels per tile, ring entries, K steps per block of the cluster
  int resident;             // the filter tile stays in shared memory (its K steps behind the ring)
  int set, mains, bufs, cols;   // columns of an accumulator, accumulators of the main terms (0: one for all terms), buffers, columns in all
  long long x_batch, out_batch;
  int ih, iw, ow, kh, kw, sh, sw, dh, dw, pt, pl;
  float act_alpha, act_beta;
  int early;                // filter and bias are constants: read ahead of pdl_wait
  int* err;
};

// Byte offset of 16-byte chunk c of row r in a K-major tile of 128-byte rows with the 128-byte swizzle.
__host__ __device__ __forceinline__ uint32_t sw128(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// ONE: one accumulator for all terms, two buffers (a block that does not walk uses the first).
// ALONE: no second block fits the SM. Then a second set of registers takes the next step's loads while this one is split. Else 96
// registers: a quarter of an SM holds five such warps (16384 registers), so that two blocks of nine fit. With 112 it holds four,
// one block per SM, whatever the shared memory leaves (32 images of 16 x 112 x 112 into 64 channels: 9 warps active, issue 37 %,
// 56 us; MobileNetV3-Large at 32 images 919 us, with two blocks 798).
// CUT: a pointwise product whose K is cut over a cluster, with the exchange unrolled: stores to one owner without a test per value, eight
// channels of the final sum under way at once (one behind the other they took 310 clocks each, and of 37000 clocks of 32 images of
// 672 x 14 x 14 into 112 the exchange had 13000): 18.4 -> 15.4 us, 8 of 512 x 28 x 28 into 128 16.9 -> 13.3, 32 of 960 x 7 x 7 into
// 160 12.9 -> 12.3. A kernel of its own, without the code for a block that cuts nothing (with it 1 us more); unrolled in the others it
// cost those that cut nothing 0.9 us, taken out of them 0.3 to 0.7. Windows keep the plain form.
template <bool WINDOW, int ACT, bool ONE, bool ALONE, bool CUT>
__global__ void __maxnreg__(ALONE ? 112 : 96) conv_tc_kernel(const ConvTcDev p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], w_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ float bias_s[256];                // of this block's channels, so that no store waits for a load of its own
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bn = p.bn, S = p.stages, parts = gridDim.z;
  const int nkb = (p.k + KB - 1) / KB, kb0 = blockIdx.z * p.kper, kbs = min(nkb, kb0 + p.kper) - kb0;
  const int bbytes = bn * KB * 8, stage_bytes = 2 * kABytes + (p.resident ? 0 : bbytes);
  uint8_t* wres = smem + S * stage_bytes;      // the resident filter tile
  float* part = reinterpret_cast<float*>(wres + (p.resident ? p.kper * bbytes : 0));   // [parts][bn / parts][PX] sums of the cluster
  int2* tab = reinterpret_cast<int2*>(part + (CUT || parts > 1 ? bn * PX : 0));
  const int tiles = (p.n + PX - 1) / PX, mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  // Accumulators of a tile: [cross terms | main terms of even | of odd K steps], or one for all.
  const uint32_t set = p.set, cols = p.cols, span = (p.mains + 1) * set;
  const int mains = ONE ? 0 : min(p.mains, kbs);   // in use
  const int two = ONE ? 1 : p.bufs - 1;        // tile i has buffer i & two, for the (i >> two)-th time
  cg::cluster_group cl = cg::this_cluster();
  if (CUT || parts > 1) cl.barrier_arrive();          // answered before the first write to another block's memory

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], kLoaders / 32 + (p.resident ? 0 : 1));   // every loader warp once, and the bulk copy's bytes
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], kLoaders / 32);
    }
    mbar_init(&w_full, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kLoaders / 32) {
    // The launch asks for shared memory in proportion to these columns: whatever blocks share an
    // SM, their columns fit the 512, and the allocation never waits.
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (!p.early) pdl_wait();                    // computed by a step in front
  const int m0 = blockIdx.y * bn, mlast = p.m - 1 - m0;   // first channel; last one that exists, relative to it
  if (tid < bn) bias_s[tid] = p.bias && tid <= mlast ? ld_plain(p.bias + m0 + tid) : 0.f;
  if (WINDOW) {
    // k -> (offset of the tap inside an image, its row and column)
    const int taps = p.kh * p.kw;
    for (int k = tid; k < p.k; k += kThreads) {
      const int c = k / taps, r = k - c * taps, fy = r / p.kw * p.dh, fx = (r % p.kw) * p.dw;
      tab[k] = make_int2(c * p.ih * p.iw + fy * p.iw + fx, fy << 16 | fx);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();

  const float* wsrc = p.w + ((size_t)blockIdx.y * nkb + kb0) * (bbytes / 4);
  auto load_filter = [&](int g) {              // ring entry of running K step g
    const int s = g % S;
    mbar_arrive_expect_tx(&full[s], (uint32_t)bbytes);
    bulk_load(smem + s * stage_bytes + 2 * kABytes, wsrc + (size_t)(g % kbs) * (bbytes / 4), (uint32_t)bbytes, &full[s]);
  };
  if (tid == 0) {                              // ahead of pdl_wait where these are constants
    if (p.resident) {
      mbar_arrive_expect_tx(&w_full, (uint32_t)(kbs * bbytes));
      bulk_load(wres, wsrc, (uint32_t)(kbs * bbytes), &w_full);
    } else {
      for (int g = 0; g < S && g < kbs * mine; ++g) load_filter(g);
    }
  }
  pdl_wait();
  if (CUT || parts > 1) cl.barrier_wait();

  auto finish = [&](float v, float bias) { return apply_act(ACT, __fadd_rn(v, bias), p.act_alpha, p.act_beta); };
  const size_t hw4 = (size_t)p.hw * 4;         // bytes between channels

  if (warp < kLoaders / 32) {
    // Thread t owns pixel t % 128 of a tile: as loader for 16 of the 32 k of a step, in the
    // epilogue for every other group of 16 channels.
    const int row = tid & (PX - 1), kh16 = (tid >> 7) * 16;
    const uint32_t off0 = sw128(row, kh16 / 4);   // chunk q of this half of the row: off0 ^ (q << 4)
    const float* xcol = p.x;                   // this thread's column of the tile being loaded
    const float* gcol = nullptr;
    int iy0 = 0, ix0 = 0;
    auto place = [&](int i) {                  // tile i of this block's
      const int col = ((int)blockIdx.x + i * (int)gridDim.x) * PX + row;
      const bool ok = i < mine && col < p.n;
      const int cb = ok ? col / p.hw : 0, px = ok ? col - cb * p.hw : 0;
      xcol = p.x + cb * p.x_batch;
      if (WINDOW) {
        const int oy = px / p.ow;
        iy0 = oy * p.sh - p.pt;
        ix0 = (px - oy * p.ow) * p.sw - p.pl;
        xcol += (long long)iy0 * p.iw + ix0;
      } else {
        xcol += px;
        if (p.gate) gcol = p.gate + (long long)cb * p.k;
      }
    };
    // Sixteen loads without a branch between them (a conditional load each serialised them at the
    // latency of L2: 4000 clocks a step instead of 1300). What lies outside is read at some valid
    // address and zeroed when it is used: bit j of the result says that value j counts.
    auto fetch = [&](int kb, float (&d)[16]) -> uint32_t {
      const int k0 = (kb0 + kb) * KB + kh16;
      if (!WINDOW && k0 + 16 <= p.k) {
        const char* at = reinterpret_cast<const char*>(xcol) + k0 * hw4;
#pragma unroll
        for (int j = 0; j < 16; ++j) d[j] = *reinterpret_cast<const float*>(at + (uint32_t)j * (uint64_t)hw4);
        return 0xffffu;
      }
      uint32_t use = 0;
      if (k0 >= p.k) return use;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int k = min(k0 + j, p.k - 1);
        bool ok = k0 + j < p.k;
        const float* at;
        if (WINDOW) {
          const int2 e = tab[k];
          ok = ok && (unsigned)(iy0 + (e.y >> 16)) < (unsigned)p.ih && (unsigned)(ix0 + (e.y & 0xffff)) < (unsigned)p.iw;
          at = xcol + e.x;
          at = ok ? at : p.x;
        } else {
          at = xcol + (long long)k * p.hw;
        }
        d[j] = *at;
        use |= (ok ? 1u : 0u) << j;
      }
      return use;
    };
    // The gate multiplies the values just before their split; a warp's pixels lie in one or two
    // images, so these are one or two lines each.
    auto apply_gate = [&](int kb, const float* gc, float (&d)[16]) {
      const int k0 = (kb0 + kb) * KB + kh16;
      float gv[16];
      if ((p.k & 3) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 u = *reinterpret_cast<const float4*>(gc + min(k0 + 4 * q, p.k - 4));
          gv[4 * q] = u.x; gv[4 * q + 1] = u.y; gv[4 * q + 2] = u.z; gv[4 * q + 3] = u.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) gv[j] = gc[min(k0 + j, p.k - 1)];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) d[j] = __fmul_rn(d[j], gv[j]);
    };

    float v[16], ahead_v[ALONE ? 16 : 1];
    uint32_t use = 0;
    int g = 0;                                 // running K step
    bool alive = true;
    // Loads steps [from, to) of tile i (the first of them is already in v) into the ring; leaves the step
    // behind them in v.
    auto fill = [&](int i, int from, int to) {
      for (int kb = from; kb < to && alive; ++kb, ++g) {
        const float* gc = gcol;
        auto next = [&](float (&d)[16]) -> uint32_t {
          if (kb + 1 == kbs) place(i + 1);
          return kb + 1 < kbs || i + 1 < mine ? fetch(kb + 1 < kbs ? kb + 1 : 0, d) : 0u;
        };
        uint32_t ahead_use = 0;
        if constexpr (ALONE) ahead_use = next(ahead_v);
        if (gc) apply_gate(kb, gc, v);
        const int s = g % S;
        if (g >= S) {
          if (!mbar_wait_all(&empty[s], ((g / S) & 1) ^ 1)) { atomicExch(p.err, 31); abort_flag = 1; alive = false; return; }
          if (tid == 0 && !p.resident) load_filter(g);
        }
        uint8_t* hi_t = smem + s * stage_bytes;
        // A half of the step that no MMA reads needs no stores.
        const bool stores = kh16 == 0 || (kb0 + kb) * KB + 16 < p.k;
        if (use != 0xffffu) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = (use >> j) & 1u ? v[j] : 0.f;
        }
        if (stores) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float4 hi, lo;
            tf32_split(make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]), hi, lo);
            uint8_t* at = hi_t + (off0 ^ (uint32_t)(q << 4));
            *reinterpret_cast<float4*>(at) = hi;
            *reinterpret_cast<float4*>(at + kABytes) = lo;
          }
        }
        fence_proxy_async();
        __syncwarp();                          // one arrival per warp: those of 256 threads took their turns at the barrier
        if (lane == 0) mbar_arrive(&full[s]);
        if constexpr (ALONE) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = ahead_v[j];
          use = ahead_use;
        } else {
          use = next(v);                       // under way over the epilogue that may lie in front of the next step
        }
      }
    };

    if (mine > 0) {
      place(0);
      use = fetch(0, v);
      fill(0, 0, kbs);
    }
    // With one buffer the products of tile i + 1 wait for this epilogue: only the ring is filled ahead of it.
    const int ahead = ONE || two ? kbs : min(kbs, S);
    for (int i = 0; i < mine && alive; ++i) {
      if (i + 1 < mine) fill(i + 1, 0, ahead);
      if (!alive) break;
      const int col = ((int)blockIdx.x + i * (int)gridDim.x) * PX + row;
      const bool col_ok = col < p.n;
      const int cc = min(col, p.n - 1), cb = cc / p.hw;
      const long long at = cb * p.out_batch + (cc - cb * p.hw) + (long long)m0 * p.hw;
      if (!mbar_wait_all(&acc_full[i & two], (i >> two) & 1)) { atomicExch(p.err, 33); abort_flag = 1; break; }
      tc_fence_after();
      const int share = bn / parts;
      const uint32_t base = tmem + (i & two) * span + ((uint32_t)((warp & 3) * 32) << 16);
      for (int c = (warp >> 2) * 16; c < bn && c <= mlast; c += 32) {
        uint32_t u[16];
        tc_ld_32x16(base + (uint32_t)c + (mains ? set : 0u), u);
        auto add = [&](uint32_t from) {          // u += an accumulator, once both are there
          uint32_t more[16];
          tc_ld_32x16(base + (uint32_t)c + from, more);
          tc_wait_ld(u, more);
#pragma unroll
          for (int j = 0; j < 16; ++j) u[j] = __float_as_uint(__fadd_rn(__uint_as_float(u[j]), __uint_as_float(more[j])));
        };
        if (CUT || parts > 1) {
          // To the block that finishes these channels; no one waits for a remote load.
          if (mains > 1) add(2 * set);
          if (mains) add(0u);
          else tc_wait_ld(u);
          int owner = c / share, left = share - c % share;
          if (CUT && left >= 16) {
            float* dst = cl.map_shared_rank(part, owner) + ((int)blockIdx.z * share + (share - left)) * PX + row;
#pragma unroll
            for (int e = 0; e < 16; ++e) dst[e * PX] = __uint_as_float(u[e]);
            continue;
          }
          for (int j = 0; j < 16;) {           // uniform: channels per owner are a multiple of two
            float* dst = cl.map_shared_rank(part, owner) + ((int)blockIdx.z * share + (share - left)) * PX + row;
            const int run = min(left, 16 - j);
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (e >= j && e < j + run) dst[(e - j) * PX] = __uint_as_float(u[e]);
            j += run; left = share; ++owner;
          }
          continue;
        }
        char* o = reinterpret_cast<char*>(p.out + at) + c * hw4;
        const char* rs = p.res ? reinterpret_cast<const char*>(p.res + at) + c * hw4 : nullptr;
        float r[16];
        if (rs) {
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = *reinterpret_cast<const float*>(rs + (uint32_t)min(j, mlast - c) * hw4);
        }
        if (mains > 1) add(2 * set);
        if (mains) add(0u);
        else tc_wait_ld(u);
        float y[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 b = *reinterpret_cast<const float4*>(bias_s + c + 4 * q);
          y[4 * q] = finish(__uint_as_float(u[4 * q]), b.x);
          y[4 * q + 1] = finish(__uint_as_float(u[4 * q + 1]), b.y);
          y[4 * q + 2] = finish(__uint_as_float(u[4 * q + 2]), b.z);
          y[4 * q + 3] = finish(__uint_as_float(u[4 * q + 3]), b.w);
        }
        if (rs) {
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] = __fadd_rn(y[j], r[j]);
        }
        if (!col_ok) continue;
        if (c + 15 <= mlast) {
#pragma unroll
          for (int j = 0; j < 16; ++j) *reinterpret_cast<float*>(o + (uint32_t)j * hw4) = y[j];
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j <= mlast) *reinterpret_cast<float*>(o + (uint32_t)j * hw4) = y[j];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[i & two]);
      if (!ONE && i + 1 < mine) fill(i + 1, ahead, kbs);
    }
  } else if (elect_one()) {
    // Both operands TF32 (format 2), K-major, fp32 accumulator.
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(PX >> 4) << 24);
    bool ok = !p.resident || mbar_wait(&w_full, 0);
    if (!ok) { atomicExch(p.err, 34); abort_flag = 1; }
    for (int i = 0, g = 0; i < mine && ok; ++i) {
      if (i > two) {
        ok = mbar_wait(&acc_empty[i & two], ((i >> two) & 1) ^ 1);
        if (!ok) { atomicExch(p.err, 35); abort_flag = 1; break; }
        tc_fence_after();
      }
      const uint32_t d = tmem + (i & two) * span;
      for (int kb = 0; kb < kbs; ++kb, ++g) {
        const int s = g % S;
        ok = mbar_wait(&full[s], (g / S) & 1);
        if (!ok) { atomicExch(p.err, 32); abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t a = smem_u32(smem + s * stage_bytes);
        const uint32_t b = p.resident ? smem_u32(wres + kb * bbytes) : a + 2 * kABytes;
        const uint64_t da = desc_sw128(a), dal = desc_sw128(a + kABytes);
        const uint64_t db = desc_sw128(b), dbl = desc_sw128(b + bbytes / 2);
        const uint32_t dm = mains ? d + (uint32_t)(1 + (mains > 1 ? kb & 1 : 0)) * set : d;
        const int steps = min(4, (p.k - (kb0 + kb) * KB + 7) / 8);
        // The cross terms of a step first: 2^-11 of the result, they are added while its sum may still be small.
        auto cross = [&](int kk) {
          const uint64_t off = (uint64_t)(kk * 32 >> 4);
          tc_mma_tf32(d, dal + off, db + off, idesc, (kb > 0 || kk > 0) ? 1u : 0u);   // a_lo * b_hi
          tc_mma_tf32(d, da + off, dbl + off, idesc, 1u);                             // a_hi * b_lo
        };
        auto main = [&](int kk) {
          const uint64_t off = (uint64_t)(kk * 32 >> 4);
          tc_mma_tf32(dm, da + off, db + off, idesc, (ONE || kb >= mains || kk > 0) ? 1u : 0u);   // a_hi * b_hi
        };
        // Full steps unrolled: issuing an instruction took 113 clocks in a loop of run-time length, 40 to
        // 65 (up to 128 channels) this way.
        if (steps == 4) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) cross(kk);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) main(kk);
        } else {
#pragma unroll 1
          for (int kk = 0; kk < steps; ++kk) cross(kk);
#pragma unroll 1
          for (int kk = 0; kk < steps; ++kk) main(kk);
        }
        tc_commit(&empty[s]);
      }
      if (ok) tc_commit(&acc_full[i & two]);
    }
  }
  __syncwarp();

  if (CUT || parts > 1) {
    // Every block of the cluster finishes its share of the channels of the one tile.
    cl.sync();
    const int share = bn / parts, c0 = blockIdx.z * share, row = tid & (PX - 1), col = blockIdx.x * PX + row;
    if (warp < kLoaders / 32 && col < p.n) {
      const int cb = col / p.hw;
      const long long at = cb * p.out_batch + (col - cb * p.hw) + (long long)m0 * p.hw;
      if constexpr (CUT) {
        constexpr int G = 8;
        char* o = reinterpret_cast<char*>(p.out + at) + c0 * hw4;
        const char* rs = p.res ? reinterpret_cast<const char*>(p.res + at) + c0 * hw4 : nullptr;
        const int last = min(share - 1, mlast - c0);
#pragma unroll 1
        for (int c1 = tid >> 7; c1 <= last; c1 += 2 * G) {
          float r[G], sum[G];
#pragma unroll
          for (int i = 0; i < G; ++i) {
            r[i] = sum[i] = 0.f;
            if (rs) r[i] = *reinterpret_cast<const float*>(rs + (uint32_t)min(c1 + 2 * i, last) * hw4);
          }
          for (int q = 0; q < parts; ++q) {
            const float* from = part + q * share * PX + row;
#pragma unroll
            for (int i = 0; i < G; ++i) sum[i] = __fadd_rn(sum[i], from[min(c1 + 2 * i, last) * PX]);
          }
#pragma unroll
          for (int i = 0; i < G; ++i) {
            const int c = c1 + 2 * i;
            float y = finish(sum[i], bias_s[c0 + min(c, last)]);
            if (rs) y = __fadd_rn(y, r[i]);
            if (c <= last) *reinterpret_cast<float*>(o + (uint32_t)c * hw4) = y;
          }
        }
      } else {
#pragma unroll 2
        for (int c = tid >> 7; c < share; c += 2) {
          if (c0 + c > mlast) break;
          const float r = p.res ? p.res[at + (long long)(c0 + c) * p.hw] : 0.f;
          float sum = 0.f;
          for (int q = 0; q < parts; ++q) sum = __fadd_rn(sum, part[(q * share + c) * PX + row]);
          float y = finish(sum, bias_s[c0 + c]);
          if (p.res) y = __fadd_rn(y, r);
          p.out[at + (long long)(c0 + c) * p.hw] = y;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag != 0 && tid == 0) {           // bounded time for copies still in flight to land
    for (int s = 0; s < S; ++s) {
      (void)mbar_wait(&full[s], 0);
      (void)mbar_wait(&full[s], 1);
    }
    if (p.resident) (void)mbar_wait(&w_full, 0);
  }
  __syncthreads();
  if (warp == kLoaders / 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
  }
}

// One thread per 16-byte chunk of the blocked filter.
__global__ void pack_filter_tc_kernel(const float* __restrict__ w, uint8_t* __restrict__ out, int m, int k, int bn, int tiles) {
  const int nkb = (k + KB - 1) / KB;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)tiles * nkb * bn * 8) return;
  const int c = (int)(i & 7), r = (int)((i >> 3) % bn), kb = (int)((i >> 3) / bn % nkb), tile = (int)((i >> 3) / bn / nkb);
  const int row = tile * bn + r;
  float v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int kk = kb * KB + c * 4 + j;
    v[j] = row < m && kk < k ? w[(long long)row * k + kk] : 0.f;
  }
  float4 hi, lo;
  tf32_split(make_float4(v[0], v[1], v[2], v[3]), hi, lo);
  uint8_t* blk = out + ((size_t)tile * nkb + kb) * bn * KB * 8;
  *reinterpret_cast<float4*>(blk + sw128(r, c)) = hi;
  *reinterpret_cast<float4*>(blk + bn * KB * 4 + sw128(r, c)) = lo;
}

Shape shape_of(const ConvParams& q) {
  return pick_shape(q, {device_sm_count(), cluster_slots(2), cluster_slots(4), cluster_slots(8)});
}

template <bool WINDOW, int ACT, bool ONE, bool ALONE, bool CUT>
cudaError_t launch_form(const ConvTcDev& p, const Shape& sh, cudaStream_t st) {
  static unsigned long long done = 0;
  if (cudaError_t e = ensure_dynamic_smem(conv_tc_kernel<WINDOW, ACT, ONE, ALONE, CUT>, (int)kSmemMax, &done)) return e;
  const dim3 grid((unsigned)sh.ctas, (unsigned)sh.tiles, (unsigned)sh.split);
  return launch_pdl(conv_tc_kernel<WINDOW, ACT, ONE, ALONE, CUT>, grid, dim3(kThreads), sh.smem, st, sh.split, p);
}

template <bool WINDOW, int ACT>
cudaError_t launch_act(const ConvTcDev& p, const Shape& sh, bool walks, cudaStream_t st) {
  // Walking blocks of more than half of an SM's shared memory (calls of 32 x 117 x 57 x 57 into 216: with the second set 94 us,
  // without 101; 13 x 326 x 57 x 57 into 170: 79 and 78). Blocks of that size with a tile each lose by it (MobileNetV3-Large, 56
  // images of 192 x 192: 925 us, without 912); where only the grid is too small for two on an SM, and with a window, it gains on
  // some shapes what it loses on others.
  const bool alone = sh.smem > kSmemSm / 2 - kSmemBeside && walks;
  if constexpr (!WINDOW) {
    if (alone) return sh.mains == 0 ? launch_form<WINDOW, ACT, true, true, false>(p, sh, st) : launch_form<WINDOW, ACT, false, true, false>(p, sh, st);
    if (sh.split > 1)
      return sh.mains == 0 ? launch_form<WINDOW, ACT, true, false, true>(p, sh, st) : launch_form<WINDOW, ACT, false, false, true>(p, sh, st);
  }
  return sh.mains == 0 ? launch_form<WINDOW, ACT, true, false, false>(p, sh, st) : launch_form<WINDOW, ACT, false, false, false>(p, sh, st);
}

template <bool WINDOW>
cudaError_t launch_one(const ConvTcDev& p, const Shape& sh, bool walks, int act, cudaStream_t st) {
  switch (act) {
    case ACT_NONE: return launch_act<WINDOW, ACT_NONE>(p, sh, walks, st);
    case ACT_RELU: return launch_act<WINDOW, ACT_RELU>(p, sh, walks, st);
    case ACT_HARDSWISH: return launch_act<WINDOW, ACT_HARDSWISH>(p, sh, walks, st);
    case ACT_HARDSIGMOID: return launch_act<WINDOW, ACT_HARDSIGMOID>(p, sh, walks, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool conv_tc_supported(const ConvParams& q) {
  const int64_t k = (int64_t)q.c * q.kh * q.kw, cols = (int64_t)q.n * q.oh * q.ow;
  return q.group == 1 && k >= 1 && k <= 4096 && cols >= 1 && cols < (1ll << 30) && (int64_t)q.c * q.ih * q.iw < (1ll << 30) &&
         q.kh * q.dh < 32768 && q.kw * q.dw < 32768 && q.oc >= 1 && q.oc <= 16384 && q.act != ACT_GELU && shape_of(q).bn > 0;
}

double conv_tc_rounds(const ConvParams& q) { return shape_of(q).rounds; }

int64_t conv_tc_filter_elems(const ConvParams& q) {
  const Shape sh = shape_of(q);
  const int64_t nkb = ((int64_t)q.c * q.kh * q.kw + KB - 1) / KB;
  return (int64_t)sh.tiles * nkb * sh.bn * KB * 2;
}

cudaError_t launch_pack_filter_tc(const ConvParams& q, const float* w, float* packed, cudaStream_t st) {
  const Shape sh = shape_of(q);
  const int k = q.c * q.kh * q.kw;
  const long long chunks = (long long)sh.tiles * ((k + KB - 1) / KB) * sh.bn * 8;
  pack_filter_tc_kernel<<<(unsigned)((chunks + 255) / 256), 256, 0, st>>>(w, reinterpret_cast<uint8_t*>(packed), q.oc, k, sh.bn,
                                                                       sh.tiles);
  return cudaGetLastError();
}

cudaError_t launch_conv_tc(const ConvParams& q, int images, const float* x, const float* packed, const float* bias, const float* gate,
                           const float* residual, float* out, bool constants, int* err_word, cudaStream_t st) {
  Shape sh = shape_of(q);
  ConvTcDev p{};
  p.x = x; p.w = packed; p.out = out; p.bias = bias; p.res = residual; p.gate = gate;
  p.m = q.oc; p.k = q.c * q.kh * q.kw; p.hw = q.oh * q.ow; p.n = images * p.hw;
  if (p.m == 0 || p.n == 0) return cudaSuccess;
  const bool walks = sh.ctas < (q.n * p.hw + PX - 1) / PX;   // in the whole batch: a part takes the whole's kernel
  sh.ctas = std::min(sh.ctas, (p.n + PX - 1) / PX);
  p.bn = sh.bn; p.stages = sh.stages; p.kper = sh.kper; p.resident = sh.resident;
  p.set = sh.set; p.mains = sh.mains; p.bufs = sh.bufs; p.cols = sh.cols;
  p.x_batch = (long long)q.c * q.ih * q.iw; p.out_batch = (long long)p.m * p.hw;
  p.ih = q.ih; p.iw = q.iw; p.ow = q.ow; p.kh = q.kh; p.kw = q.kw; p.sh = q.sh; p.sw = q.sw; p.dh = q.dh; p.dw = q.dw;
  p.pt = q.pad_t; p.pl = q.pad_l;
  p.act_alpha = q.act_alpha; p.act_beta = q.act_beta;
  p.early = constants;
  p.err = err_word;
  const bool window = q.kh != 1 || q.kw != 1 || q.sh != 1 || q.sw != 1 || q.pad_t || q.pad_l || q.oh != q.ih || q.ow != q.iw;
  if (window && gate) return cudaErrorInvalidValue;
  return window ? launch_one<true>(p, sh, walks, q.act, st) : launch_one<false>(p, sh, walks, q.act, st);
}

}  // namespace ac

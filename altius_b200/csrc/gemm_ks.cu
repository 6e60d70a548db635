// fp16-split GEMM for few rows (a small batch of a transformer): C = epilogue(A * B^T) with both operands
// as fp16 halves by TMA (A on the fixed scale, written by the kernel in front; B prepared once), three
// kind::f16 MMAs per product -- the operand formats of the CTA-pair kernel (gemm_tc.cu), which takes
// the larger problems. The tensor core truncates its sum at every instruction, an error that grows with the
// number of instructions behind one another on an accumulator of full size; so the cross terms
// (2^-11 of the result) have an accumulator of their own and the others are dealt to as many as
// tensor memory holds beside it, K-block by K-block in turn
// (197 x 768 x 2304: relative error against 64 bits 9.8e-7 in one accumulator, 1.2e-7 this way; the pair kernel 3.5e-7).
//
// What bounds it: 197 rows against 768 x 2304 are 2.1 GFLOP and 7 MB of weights, 1.2 us of either, so what
// counts is latency. On 256 x 256 tiles such a product has 9 tiles for 74 pairs; cut along K its
// partial sums went through memory to a second kernel, 20 us in all. Here a cluster of S blocks
// shares one 128 x BN tile: each takes a range of K (two to eight K-blocks), and the accumulators
// meet in distributed shared memory: every block sends each peer that peer's columns of its
// accumulator, and after one cluster barrier finishes its own BN / S columns (sum in rank order, so
// the result does not depend on timing; bias, activation, residual; whole-line stores). The weights
// of the first stages are requested while the kernel in front still runs.
//
// Per block: warps 0-15 move the accumulator and run the epilogue, warp 16 issues TMA, warp 17 MMAs.
//
// The full-range products (3xTF32) of few rows run here too, from fp32 operands (WIDE): one kernel without K-slices through
// memory (a second kernel of 6 us behind each product), cross terms apart, so errors against 64 bits two to five times
// smaller: 1386 x 384 x 1152 21.2 -> 14.1 us, 4.9e-7 -> 1.2e-7; 12 layers of DeiT-S at 7 images 1186 -> 972 us.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "gemm_ks_shape.h"
#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"
#include "tc_common.cuh"
#include "tensor_map.h"

namespace cg = cooperative_groups;

namespace ac {
namespace {

using namespace tc;
using namespace gemm_ks;

constexpr int kEpiThreads = 512, kTmaWarp = 16, kMmaWarp = 17, kThreads = 576;

struct KsDev {
  int m, n, k;
  int bn, stages, kper;                       // columns of a tile, ring entries, K-blocks per block of the cluster
  int inv;                                    // ceil(2^20 / quads), quads = float4s per row of a block's share: e / quads = e * inv >> 20
  float* c; long long ldc;                    // may be null when c16_hi / c16_lo are given
  uint2* c16_hi; uint2* c16_lo; long long ldc16;
  const float* bias; const float* res; long long ldres;
  const float* acc_scale;                     // device scalar or null
  int* err;
};

// Eight 32-bit columns of the warp's 32 lanes.
__device__ __forceinline__ void st8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(__float_as_uint(v[0])),
               "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])),
               "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
}
// A in tensor memory: row r in lane r, eight values of K in eight columns.
__device__ __forceinline__ void mma_tf32_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// WIDE: fp32 operands of any range as 3xTF32, K-blocks of 32 floats. B comes prepared; A arrives as it is, and the sixteen warps split it
// into tensor memory, from where the products take it (written back beside it in shared memory the halves cost 7 % more).
template <int ACT, bool WIDE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_ks_kernel(const __grid_constant__ CUtensorMap ta_hi, const __grid_constant__ CUtensorMap ta_lo,
               const __grid_constant__ CUtensorMap tb_hi, const __grid_constant__ CUtensorMap tb_lo, const KsDev p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kMaxStages], ready[kMaxStages], empty[kMaxStages], acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ unsigned seen;                   // what the block has seen of the values it split
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bn = p.bn, S = p.stages, parts = gridDim.z, share = bn / parts, rank = blockIdx.z;
  const int bhalf = bn * KB * 2;
  constexpr int kABytes = WIDE ? kAHalf : 2 * kAHalf;
  const int stage_bytes = kABytes + 2 * bhalf;
  // [parts][quads][BM + 1]: behind the ring, or over it where no other block writes there.
  float4* part = reinterpret_cast<float4*>(smem + (parts > 1 ? S * stage_bytes : 0));
  constexpr int kStep = WIDE ? KB / 2 : KB;   // of K in a block
  const int nkb = (p.k + kStep - 1) / kStep, kb0 = rank * p.kper, kbs = min(nkb, kb0 + p.kper) - kb0;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * bn;
  // Accumulators of bn columns: the cross terms have the first, the products of the high halves the others. (Three
  // at most, for any width, left 394 x 384 x 1152 at 1.66e-7 where the kernel it replaces has 1.42e-7.)
  // Wide: behind them two buffers for A's hi and lo halves of a K-block, 32 columns each. (Three or four gave nothing: 1190 clocks
  // a K-block whatever the columns up to 96, which is the issue of its twelve products.)
  constexpr int kACols = WIDE ? 128 : 0;
  const int mains = min((512 - kACols) / bn - 1, kbs), used = bn * (mains + 1) + kACols;
  const uint32_t cols = used <= 64 ? 64 : used <= 128 ? 128 : used <= 256 ? 256 : 512;
  cg::cluster_group cl = cg::this_cluster();
  if (parts > 1) cl.barrier_arrive();         // answered before the first write to another block's memory
  if (tid == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&ready[s], kEpiThreads / 32); mbar_init(&empty[s], 1); }
    mbar_init(&acc_full, 1);
    seen = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  auto load_b = [&](int it) {
    uint8_t* b = smem + (it % S) * stage_bytes + kABytes;
    mbar_arrive_expect_tx(&full[it % S], (uint32_t)stage_bytes);
    tma_load_3d(b, &tb_hi, &full[it % S], (kb0 + it) * kStep, n0, 0);
    tma_load_3d(b + bhalf, &tb_lo, &full[it % S], (kb0 + it) * kStep, n0, 0);
  };
  auto load_a = [&](int it) {
    uint8_t* a = smem + (it % S) * stage_bytes;
    tma_load_3d(a, &ta_hi, &full[it % S], (kb0 + it) * kStep, m0, 0);
    if (!WIDE) tma_load_3d(a + kAHalf, &ta_lo, &full[it % S], (kb0 + it) * kStep, m0, 0);
  };
  if (warp == kTmaWarp && lane == 0)
    for (int it = 0; it < S && it < kbs; ++it) load_b(it);   // constants: ahead of pdl_wait
  __syncwarp();
  // ---- accumulator -> the blocks that finish its columns -> this block's columns of the tile ----
  // Columns are handled in float4s: `quads` of them per row and block, float4 q of row r of rank s at
  // [(s * quads + q) * (BM + 1) + r]: a warp's rows are neighbours when they are sent (512 bytes a
  // store) and its columns lie in different banks when they are read.
  const int quads = share / 4, total = BM * quads;
  int live = 0;                                // of them this thread's block has to finish: none in the first pass
  constexpr int CH = 3;                        // float4s a thread has in work at once
  float4 rs[CH], bi[CH];
#pragma unroll
  for (int i = 0; i < CH; ++i) rs[i] = bi[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  auto place = [&](int e, int* row, int* q) {
    *row = (int)(((unsigned)e * (unsigned)p.inv) >> 20);
    *q = e - *row * quads;
    return e < live && m0 + *row < p.m && n0 + rank * share + 4 * *q < p.n;   // n % 4 == 0: the four columns exist together
  };
  auto fetch = [&](int e0) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      int row, q;
      rs[i] = bi[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!place(e0 + i * kEpiThreads, &row, &q)) continue;
      const int col = n0 + rank * share + 4 * q;
      if (p.res) rs[i] = *reinterpret_cast<const float4*>(p.res + (long long)(m0 + row) * p.ldres + col);
      if (p.bias) bi[i] = ld_plain(reinterpret_cast<const float4*>(p.bias + col));
    }
  };
  const float sc = WIDE ? 1.f : p.acc_scale ? __fmul_rn(ld_plain(p.acc_scale), kFixedUnscale) : kFixedUnscale;   // prepared with B: a constant
  auto finish = [&] {
    float most = 0.f;
    for (int e0 = tid; e0 < max(live, kEpiThreads); e0 += CH * kEpiThreads) {
      if (e0 != tid) fetch(e0);
      float4 x[CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int e = e0 + i * kEpiThreads;
        int row, q;
        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!place(e, &row, &q)) continue;
        const float4* src = part + q * (BM + 1) + row;
        x[i] = src[0];
        for (int s = 1; s < parts; ++s) {
          const float4 u = src[s * quads * (BM + 1)];
          x[i].x = __fadd_rn(x[i].x, u.x); x[i].y = __fadd_rn(x[i].y, u.y); x[i].z = __fadd_rn(x[i].z, u.z); x[i].w = __fadd_rn(x[i].w, u.w);
        }
      }
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const float4 b = bi[i], r = rs[i];
        float4 y = x[i];
        if (!WIDE) { y.x = __fmul_rn(y.x, sc); y.y = __fmul_rn(y.y, sc); y.z = __fmul_rn(y.z, sc); y.w = __fmul_rn(y.w, sc); }
        if (p.bias) { y.x = __fadd_rn(y.x, b.x); y.y = __fadd_rn(y.y, b.y); y.z = __fadd_rn(y.z, b.z); y.w = __fadd_rn(y.w, b.w); }
        if (ACT == ACT_GELU) {
          const float2 lo = gelu_ref2(make_float2(y.x, y.y)), hi = gelu_ref2(make_float2(y.z, y.w));
          y = make_float4(lo.x, lo.y, hi.x, hi.y);
        } else if (ACT == ACT_RELU) {
          y.x = fmaxf(y.x, 0.f); y.y = fmaxf(y.y, 0.f); y.z = fmaxf(y.z, 0.f); y.w = fmaxf(y.w, 0.f);
        }
        if (p.res) { y.x = __fadd_rn(y.x, r.x); y.y = __fadd_rn(y.y, r.y); y.z = __fadd_rn(y.z, r.z); y.w = __fadd_rn(y.w, r.w); }
        x[i] = y;
      }
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        int row, q;
        if (!place(e0 + i * kEpiThreads, &row, &q)) continue;
        const long long r = m0 + row;
        const int col = n0 + rank * share + 4 * q;
        if (p.c) *reinterpret_cast<float4*>(p.c + r * p.ldc + col) = x[i];
        if (!WIDE && p.c16_hi) {
          uint2 h, l;
          f16_split_fixed(x[i], h, l);
          const long long at = (r * p.ldc16 + col) >> 2;
          p.c16_hi[at] = h;
          p.c16_lo[at] = l;
          most = split_track(most, x[i]);
        }
      }
    }
    if (!WIDE && p.c16_hi && live > 0) {
      const unsigned all = __reduce_or_sync(0xffffffffu, split_seen_fixed_of_max(most));
      if (lane == 0) atomicOr(&seen, all);
    }
  };
  uint32_t tmem = 0;
  auto produce = [&] {
    pdl_wait();
    if (parts > 1) cl.barrier_wait();           // every block of the cluster runs
    // Tensor memory only now: taken earlier, it would wait for the blocks of the kernel in front that share the SM;
    // and the next kernel may start only behind it, or its allocation could come first.
    if (warp == kTmaWarp && lane == 0)
      for (int it = 0; it < S && it < kbs; ++it) load_a(it);
    __syncwarp();
    if (warp == kMmaWarp) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(cols));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = tmem_slot;
    pdl_trigger();

    if (warp == kTmaWarp) {
      if (lane == 0) {
        for (int it = S; it < kbs; ++it) {
          {
            if (!mbar_wait(&empty[it % S], (uint32_t)((it / S) & 1) ^ 1)) {
              atomicExch(p.err, 61);
              for (int s = 0; s < S; ++s) (void)mbar_wait(&full[s], (uint32_t)((it - 1) / S) & 1);   // copies in flight land
              break;
            }
            load_b(it);
          }
          load_a(it);
        }
      }
    } else if (warp == kMmaWarp) {
      if (elect_one()) {
        constexpr uint32_t kFmt = WIDE ? 2u : 0u;   // TF32 or fp16
        const uint32_t idesc = (1u << 4) | (kFmt << 7) | (kFmt << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        for (int it = 0; it < kbs; ++it) {
          const int s = it % S;
          if (!mbar_wait(WIDE ? &ready[s] : &full[s], (uint32_t)(it / S) & 1)) {
            atomicExch(p.err, 62);
            for (int w = it; w < kbs && w < it + S; ++w) (void)mbar_wait(&full[w % S], (uint32_t)(w / S) & 1);   // copies in flight land
            break;
          }
          tc_fence_after();
          const uint32_t a = smem_u32(smem + s * stage_bytes);
          const uint64_t da = desc_sw128(a), dal = desc_sw128(a + kAHalf);
          const uint64_t db = desc_sw128(a + kABytes), dbl = desc_sw128(a + kABytes + bhalf);
          const uint32_t ta = tmem + (uint32_t)(bn * (mains + 1) + (it & 1) * 64);   // wide: A's halves
          // Always four steps (what lies beyond K arrives as zeros): with a run-time count an instruction
          // took 113 clocks to issue, unrolled 57 (96 columns).
          const uint32_t cross = tmem, main = tmem + (uint32_t)((1 + it % mains) * bn);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint64_t off = (uint64_t)(kk * 32 >> 4);
            auto mma = [&](uint32_t d, bool lo, uint64_t b, uint32_t accumulate) {
              if (WIDE) mma_tf32_ta(d, ta + (uint32_t)(8 * kk + (lo ? 32 : 0)), b + off, idesc, accumulate);
              else tc_mma_f16(d, (lo ? dal : da) + off, b + off, idesc, accumulate);
            };
            mma(main, false, db, (it >= mains || kk > 0) ? 1u : 0u);        // a_hi * b_hi
            mma(cross, true, db, (it > 0 || kk > 0) ? 1u : 0u);   // a_lo * b_hi
            mma(cross, false, dbl, 1u);                           // a_hi * b_lo
          }
          tc_commit(&empty[s]);
        }
        tc_commit(&acc_full);
      }
    }
    if (warp < kEpiThreads / 32) {
      fetch(tid);                                // under the products
      if (WIDE) {
        for (int it = 0; it < kbs; ++it) {
          const int s = it % S;
          if (!mbar_wait_all(&full[s], (uint32_t)(it / S) & 1)) { atomicExch(p.err, 65); break; }
          // This warp's 32 rows, 8 of their 32 values: two 16-byte chunks, which the swizzle spreads over the banks.
          const int row = (warp & 3) * 32 + lane, part8 = warp >> 2;
          const uint8_t* at = smem + s * stage_bytes + row * 128;
          float h[8], l[8];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float4 hi, lo;
            tf32_split(*reinterpret_cast<const float4*>(at + (((2 * part8 + c) ^ (row & 7)) << 4)), hi, lo);
            h[4 * c] = hi.x; h[4 * c + 1] = hi.y; h[4 * c + 2] = hi.z; h[4 * c + 3] = hi.w;
            l[4 * c] = lo.x; l[4 * c + 1] = lo.y; l[4 * c + 2] = lo.z; l[4 * c + 3] = lo.w;
          }
          // The products that took the buffer's last contents are complete (with a ring of two or fewer the entry could not
          // have been loaded before).
          if (S > 2 && it >= 2 && !mbar_wait_all(&empty[(it - 2) % S], (uint32_t)((it - 2) / S) & 1)) { atomicExch(p.err, 66); break; }
          tc_fence_after();
          const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(bn * (mains + 1) + (it & 1) * 64 + 8 * part8);
          st8(ta, h);
          st8(ta + 32u, l);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ready[s]);
        }
      }
      if (!warp_mbar_wait(&acc_full, 0, lane)) atomicExch(p.err, 63);
      tc_fence_after();
      const int row = (warp & 3) * 32 + lane;
      const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
      for (int c = (warp >> 2) * 16; c < bn; c += 64) {
        const uint32_t at = base + (uint32_t)c;
        uint32_t u[16], x[16], y[16];
        auto plus = [](uint32_t (&a)[16], const uint32_t (&b)[16]) {
#pragma unroll
          for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__fadd_rn(__uint_as_float(a[i]), __uint_as_float(b[i])));
        };
        tc_ld_32x16(at + (uint32_t)bn, u);
        for (int a = 2; a <= mains; a += 2) {       // two accumulators on their way at once, added in order
          tc_ld_32x16(at + (uint32_t)(a * bn), x);
          if (a < mains) tc_ld_32x16(at + (uint32_t)((a + 1) * bn), y);
          tc_wait_ld(u, x);
          plus(u, x);
          if (a < mains) {
            tc_landed(y);
            plus(u, y);
          }
        }
        tc_ld_32x16(at, x);
        tc_wait_ld(u, x);
        plus(u, x);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int cq = c / 4 + i, owner = (int)(((unsigned)cq * (unsigned)p.inv) >> 20);
          float4* dst = part + ((rank * quads + cq - owner * quads) * (BM + 1) + row);
          if (parts > 1) dst = cl.map_shared_rank(dst, owner);
          *dst = make_float4(__uint_as_float(u[4 * i]), __uint_as_float(u[4 * i + 1]), __uint_as_float(u[4 * i + 2]),
                             __uint_as_float(u[4 * i + 3]));
        }
      }
      tc_fence_before();
    }
    __syncwarp();
    if (parts > 1) cl.sync();
    else __syncthreads();
  };
  // The first pass has nothing to finish: it brings the epilogue's code into the instruction cache while
  // the kernel in front still runs (over cold code it took 5600 clocks for 1500 of work).
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) {
      live = total;
      produce();
    }
    if (warp < kEpiThreads / 32) finish();
  }
  __syncthreads();
  // Out of range, or nothing but tiny values in this block's 128 x share results.
  if (tid == 0 && ((seen & 1u) || ((seen & 4u) && !(seen & 2u)))) atomicCAS(p.err, 0, kRangeCode);
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
  }
}

}  // namespace

// The parts of the chip that hold a cluster have 14 to 18 SMs each, so fewer blocks run at once than there
// are SMs: 36 clusters of four took two rounds (18 us for 197 x 768 x 2304), 24 one.
int cluster_slots(int split) {
  if (split <= 1) return device_sm_count();
  static std::atomic<int> known[64][4];
  const int at = split <= 2 ? 1 : split <= 4 ? 2 : 3;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (const int v = known[dev][at].load(std::memory_order_relaxed)) return v;
  static unsigned long long done = 0;
  int slots = 0;
  if (ensure_dynamic_smem(gemm_ks_kernel<ACT_NONE, false>, (int)kSmemMax, &done) == cudaSuccess) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1, (unsigned)device_sm_count(), (unsigned)split);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = (unsigned)split;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&slots, gemm_ks_kernel<ACT_NONE, false>, &cfg) != cudaSuccess) slots = 0;
  }
  (void)cudaGetLastError();
  if (slots <= 0) {            // no device: the counts of a B200
    static const int b200[4] = {148, 74, 33, 15};
    slots = b200[at];
  }
  known[dev][at].store(slots, std::memory_order_relaxed);
  return slots;
}

namespace {

Shape shape_of(int64_t m, int64_t n, int64_t k, bool wide) {
  return pick_shape(m, n, k, wide, [](int split) { return cluster_slots(split); });
}

template <int ACT, bool WIDE>
cudaError_t launch_act(const CUtensorMap& ah, const CUtensorMap& al, const CUtensorMap& bh, const CUtensorMap& bl,
                       const KsDev& d, const Shape& sh, cudaStream_t st) {
  // The kernel takes its addresses in shared memory, its cluster's included, from these numbers without a check of its own.
  Shape whole;
  if (!make_shape(sh.bn, sh.split, d.k, WIDE, &whole) || d.bn != sh.bn || d.kper != whole.kper || d.stages != whole.stages || d.inv != whole.inv ||
      sh.smem != whole.smem)
    return cudaErrorInvalidValue;
  static unsigned long long done = 0;
  if (cudaError_t e = ensure_dynamic_smem(gemm_ks_kernel<ACT, WIDE>, (int)kSmemMax, &done)) return e;
  const dim3 grid((unsigned)((d.n + sh.bn - 1) / sh.bn), (unsigned)((d.m + BM - 1) / BM), (unsigned)sh.split);
  return launch_pdl(gemm_ks_kernel<ACT, WIDE>, grid, dim3(kThreads), sh.smem, st, sh.split, ah, al, bh, bl, d);
}
template <bool WIDE>
cudaError_t launch_any(int act, const CUtensorMap& ah, const CUtensorMap& al, const CUtensorMap& bh, const CUtensorMap& bl, const KsDev& d,
                       const Shape& sh, cudaStream_t st) {
  if (act == ACT_GELU) return launch_act<ACT_GELU, WIDE>(ah, al, bh, bl, d, sh, st);
  if (act == ACT_RELU) return launch_act<ACT_RELU, WIDE>(ah, al, bh, bl, d, sh, st);
  return launch_act<ACT_NONE, WIDE>(ah, al, bh, bl, d, sh, st);
}

inline bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

KsDev device_params(const GemmParams& q, const Shape& sh, int* err_word) {
  KsDev d{};
  d.m = (int)q.m; d.n = (int)q.n; d.k = (int)q.k;
  d.bn = sh.bn; d.stages = sh.stages; d.kper = sh.kper; d.inv = sh.inv;
  d.c = q.c; d.ldc = q.ldc;
  d.bias = q.bias_n; d.res = q.residual; d.ldres = q.ld_res;
  d.err = err_word;
  return d;
}

}  // namespace

// Products that this kernel has more tiles than SMs for go to CTA pairs with short accumulators where these are faster; fitted in
// this kernel's clocks, launch and ends included as in pick_shape (us with a LayerNormalization in front, here -> there: 3152 x
// 768 x 768 31.6 -> 23.2, 12672 x 384 x 384 37.3 -> 30.4, 788 x 768 x 3072 30.6 -> 22.7; but 2885 x 768 x 768 20.5 -> 23.0, 1576 x
// 512 x 512 14.2 -> 18.4). Relative error against 64 bits there 1.6e-7, to K = 576 1.2e-7; here 2.1e-7 at K = 768, 1.5e-7 at 384.
// Tiles of 128 columns fill the pairs in one round where 192 leave a third of them idle (us, m x k x n with a quarter of the product
// that makes the operand, here -> 128 | 192: 2885 x 3072 x 768 50.6 -> 46.2 | 53.9, 1576 x 3072 x 768 42.5 -> 39.0 | 46.6,
// 1182 x 4096 x 1024 51.8 -> 48.0 | 57.0, 4000 x 2048 x 512 41.0 -> 37.4 | 43.2; two rounds: 9838 x 384 x 384 24.1 -> 18.6 | 21.6,
// 3152 x 3072 x 768 77.9 -> 71.8 | 55.3; few rows: 788 x 3072 x 768 26.7 -> 36.1 | 43.6). From K = 1024 on this kernel takes a
// tenth longer than its estimate, and its error grows (5.8e-7 at 3072).
PairSums gemm_ks_pairs(int64_t m, int64_t n, int64_t k) {
  const double here = gemm_ks_clocks(m, n, k);
  double there;
  const PairSums t = gemm_pair_sums_tiles(m, n, k, &there);
  return here >= gemm_tc_pair_clocks(m, n, k) || there < here * (k >= 1024 ? 1.08 : 0.97) ? t : PairSums{};
}

bool gemm_ks_wins(int64_t m, int64_t n, int64_t k) {
  const double here = gemm_ks_clocks(m, n, k);
  return here < gemm_tc_pair_clocks(m, n, k) || (here < 1e30 && gemm_pair_sums_wins(m, n, k));
}

double gemm_ks_clocks(int64_t m, int64_t n, int64_t k) {
  if (m < 1 || n < 4 || (n % 4) || k < 64 || (k % 8) || m > (1 << 20) || n > (1 << 20)) return 1e30;
  return shape_of(m, n, k, false).clocks;
}

bool gemm_ks_epilogue_ok(int act, bool bias_m, bool c_in, float alpha, float bias_scale) {
  return (act == ACT_NONE || act == ACT_GELU || act == ACT_RELU) && !bias_m && !c_in && alpha == 1.f && bias_scale == 1.f;
}

cudaError_t launch_gemm_ks(const GemmParams& q, PairSums pairs, int* err_word, cudaStream_t st) {
  if (!q.a16_hi || !q.a16_lo || !q.b16_hi || !q.b16_lo || !q.a16_fixed || !q.b16_plain || q.batch != 1 || (q.n % 4) ||
      (q.k % 8) || (q.lda16 % 8) || (q.ldb16 % 8) || !al16(q.a16_hi) || !al16(q.a16_lo) || !al16(q.b16_hi) || !al16(q.b16_lo) ||
      (q.c && (!al16(q.c) || (q.ldc % 4))) || (q.residual && (!al16(q.residual) || (q.ld_res % 4))) || (q.bias_n && !al16(q.bias_n)) ||
      (q.c16_hi && (q.ldc16 % 4)) || !gemm_ks_epilogue_ok(q.act, q.bias_m != nullptr, q.beta != 0.f && q.c_in, q.alpha, q.bias_scale))
    return cudaErrorInvalidValue;
  if (pairs.run) {
    if (q.c16_hi && ((q.n % 8) || (q.ldc16 % 8) || !al16(q.c16_hi) || !al16(q.c16_lo))) return cudaErrorInvalidValue;   // 16 bytes of a row at once
    return launch_gemm_pair_sums(q, pairs, err_word, st);
  }
  const Shape sh = shape_of(q.m, q.n, q.k, false);
  if (!sh.bn) return cudaErrorInvalidValue;
  KsDev d = device_params(q, sh, err_word);
  d.c16_hi = static_cast<uint2*>(q.c16_hi); d.c16_lo = static_cast<uint2*>(q.c16_lo); d.ldc16 = q.ldc16;
  d.acc_scale = q.b16_inv_scale;
  CUtensorMap ah, al, bh, bl;
  if (!make_map16(&ah, q.a16_hi, q.k, q.m, 1, q.lda16, q.m * q.lda16, BM) || !make_map16(&al, q.a16_lo, q.k, q.m, 1, q.lda16, q.m * q.lda16, BM) ||
      !make_map16(&bh, q.b16_hi, q.k, q.n, 1, q.ldb16, q.n * q.ldb16, sh.bn) || !make_map16(&bl, q.b16_lo, q.k, q.n, 1, q.ldb16, q.n * q.ldb16, sh.bn))
    return cudaErrorInvalidValue;
  return launch_any<false>(q.act, ah, al, bh, bl, d, sh, st);
}

double gemm_ks_wide_clocks(int64_t m, int64_t n, int64_t k) {
  if (m < 1 || n < 4 || (n % 4) || k < 32 || (k % 4) || m > (1 << 20) || n > (1 << 20)) return 1e30;
  // Long K: the other kernel's slices fill the SMs better than either estimate says (1386 x 3072 x 768 38.4 us, here 42.4; 394 x 2048 x 512
  // 15.5, 15.9; but 198 x 3072 x 768 17.0, 16.0).
  return shape_of(m, n, k, true).clocks * (k > 1536 ? 1.15 : 1.0);
}

cudaError_t launch_gemm_ks_wide(const GemmParams& q, int* err_word, cudaStream_t st) {
  if (!q.a || !q.b || !q.b_lo || !q.c || !q.trans_b || q.trans_a || q.batch != 1 || q.c16_hi || gemm_ks_wide_clocks(q.m, q.n, q.k) >= 1e30 ||
      (q.lda % 4) || (q.ldb % 4) || (q.ldc % 4) || !al16(q.a) || !al16(q.b) || !al16(q.b_lo) || !al16(q.c) ||
      (q.residual && (!al16(q.residual) || (q.ld_res % 4))) || (q.bias_n && !al16(q.bias_n)) ||
      !gemm_ks_epilogue_ok(q.act, q.bias_m != nullptr, q.beta != 0.f && q.c_in, q.alpha, q.bias_scale))
    return cudaErrorInvalidValue;
  const Shape sh = shape_of(q.m, q.n, q.k, true);
  const KsDev d = device_params(q, sh, err_word);
  CUtensorMap a, bh, bl;
  if (!make_map128(&a, q.a, 4, q.k, q.m, 1, q.lda, q.m * q.lda, BM) || !make_map128(&bh, q.b, 4, q.k, q.n, 1, q.ldb, q.n * q.ldb, sh.bn) ||
      !make_map128(&bl, q.b_lo, 4, q.k, q.n, 1, q.ldb, q.n * q.ldb, sh.bn))
    return cudaErrorInvalidValue;
  return launch_any<true>(q.act, a, a, bh, bl, d, sh, st);
}

}  // namespace ac

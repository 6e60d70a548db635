// Fused multi-head attention core for sequences of any length, fed by TMA from the fixed-scale fp16
// halves of the projection (the operator chain and the number format of attention_tc16.cu): the keys
// are taken in blocks of 128 with a running row maximum, so neither the scores nor the
// probabilities of a long sequence exist outside tensor memory. As separate operators (two batched
// products, the softmax, transposes and splits) 577 tokens of 60 heads took 590 us and moved 240 MB.
//
// An item is one (image, head, tile of 128 query rows); it belongs to one of the two softmax groups
// of a block, and the groups work on different items, so that the tensor core computes for one
// while the other is in its softmax.
//
//   warp 17       TMA: K and V of a block of keys into the group's buffer as soon as the products
//                 that read the previous block are complete; Q with the first block of an item.
//   warp 16       allocates tensor memory; one thread issues, for whichever group is ready, either
//                 S = Q K^T (12 MMAs: four K steps, three partial products) or O += P V.
//   warps 0-7     softmax group 0, warps 8-15 group 1: two threads per row, 64 columns each, in
//                 registers: block maximum (exchanged by the two), then P = 2^(t - m + 9) split
//                 into fp16 hi / lo over the scores it came from.
//
// An accumulator takes the products of two blocks of keys; then the softmax threads add it, in fp32, to sums
// of their own in memory (32 KB per group, in L2) and the next block starts it again: with all blocks of
// 577 tokens on one the result was off by 8.8e-7 of it (fp32 products: 7.5e-7), this way by 4.9e-7.
//
// The rows' reference m follows the maximum lazily: as long as no row of a warp has exceeded its m by
// more than 4 (in powers of two) nothing is rescaled and P stays below 2^13; otherwise the warp
// waits for the last product and multiplies its part of O by 2^(m - m').
//
// P V as two instructions per 16 keys instead of three: V hi and V lo are neighbours along N, so
// P_hi * [V_hi | V_lo] goes to 128 accumulator columns in one MMA and P_lo * V_hi adds to the last 64;
// the two halves are added when O is read. The tensor core truncates its sum at every instruction by
// up to an ulp of the sum, so what is small is added where or while the sum is small: the cross terms of
// P V have those 64 columns to themselves, and those of Q K^T come before its main terms.
//
// Measured: 577 tokens, 12 heads, five images 49.5 us, of which the 28 MMAs of a block of keys account for 11 at the rate that large
// products sustain. As in attention_tc16.cu the softmax group's cycle is the bound, not the count of instructions (40 to 65
// clocks each to issue when unrolled). 1.3 of these us are the wait between the products that read P and the scores that overwrite it.
//
// Tensor memory: S / P of group g in columns [128 g, 128 g + 128), O in [256 + 128 g, ...). Every wait
// is bounded; on expiry the kernel records a code in the error word and runs to its end.
#include <cuda.h>

#include <algorithm>

#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"
#include "tc_common.cuh"
#include "tensor_map.h"

namespace ac {
namespace {

using namespace tc;

constexpr int HD = 64, QM = 128, KV = 128;      // head dimension, query rows of an item, keys of a block
constexpr int kMmaWarp = 16, kTmaWarp = 17, kLaunch = 18 * 32;
constexpr int kTile = 128 * 128;                // bytes of one operand's hi (or lo): 128 rows of 128 bytes
constexpr int kGroupBytes = 6 * kTile;          // Q, K, V, each hi and lo
constexpr uint32_t kOCol = 256;
constexpr int kRun = 2;                         // blocks of keys whose products share an accumulator
constexpr uint32_t kPollLimit = 1u << 26;

struct FlashDev {
  float* out; long long out_row_stride, out_batch_stride;   // may be null when o16_hi / o16_lo are given
  uint2* o16_hi; uint2* o16_lo;
  int heads, tokens, tiles, items;
  int q_col, k_col, v_col;
  const float* scale; int scale_mode;
  float* sums;                                  // [grid][group][64 columns][128 rows], with more than kRun blocks of keys
  int* err;
};

// MN-major: 8 k-rows of 64 columns 1024 bytes apart, the next 64 columns (the lo tile) kTile further on.
__device__ __forceinline__ uint64_t desc_mn128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(kTile >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}
__device__ __forceinline__ void mma_f16_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
      "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
      "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The two warps of group g that share tensor-memory lane quarter q.
__device__ __forceinline__ void pair_sync(int g, int q) { asm volatile("bar.sync %0, 64;" ::"r"(1 + 4 * g + q) : "memory"); }

struct Bars {
  uint64_t q_full[2], k_full[2], v_full[2];     // TMA
  uint64_t s_full[2];                           // scores of a block complete (and K, and the last time Q, free)
  uint64_t p_ready[2];                          // P of a block written (8 warps)
  uint64_t pv_done[2];                          // O includes the block (and V is free)
};

template <int SMODE>
__global__ void __launch_bounds__(kLaunch, 1)
attention_flash16_kernel(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo, const FlashDev p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) Bars bar;
  __shared__ uint32_t tmem_slot;
  __shared__ float xch_all[2][2][QM];           // [group][column half][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = p.tokens, blocks = (T + KV - 1) / KV;
  const int slots = 2 * (int)gridDim.x;
  // Items of group g: g * grid + block, then every slots-th.
  auto items_of = [&](int g) {
    const int first = g * (int)gridDim.x + (int)blockIdx.x;
    return first < p.items ? (p.items - first + slots - 1) / slots : 0;
  };
  auto place = [&](int g, int k, int* tile, int* h, int* b) {
    const int item = g * (int)gridDim.x + (int)blockIdx.x + k * slots;
    *tile = item % p.tiles;
    const int unit = item / p.tiles;
    *h = unit % p.heads;
    *b = unit / p.heads;
  };

  if (tid == 0) {
    for (int g = 0; g < 2; ++g) {
      mbar_init(&bar.q_full[g], 1); mbar_init(&bar.k_full[g], 1); mbar_init(&bar.v_full[g], 1);
      mbar_init(&bar.s_full[g], 1); mbar_init(&bar.p_ready[g], 8); mbar_init(&bar.pv_done[g], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();
  pdl_wait();

  if (warp == kTmaWarp) {
    if (lane == 0) {
      int kn[2] = {0, 0}, vn[2] = {0, 0};
      const int n[2] = {items_of(0) * blocks, items_of(1) * blocks};
      uint32_t idle = 0;
      while (vn[0] < n[0] || vn[1] < n[1]) {
        bool did = false;
        for (int g = 0; g < 2; ++g) {
          uint8_t* base = smem + g * kGroupBytes;
          int tile, h, b;
          if (kn[g] < n[g] && (kn[g] == 0 || mbar_test(&bar.s_full[g], (uint32_t)((kn[g] - 1) & 1)))) {
            const int k = kn[g] / blocks, j = kn[g] - k * blocks;
            place(g, k, &tile, &h, &b);
            if (j == 0) {
              mbar_arrive_expect_tx(&bar.q_full[g], 2 * kTile);
              tma_load_3d(base, &tm_hi, &bar.q_full[g], p.q_col + h * HD, tile * QM, b);
              tma_load_3d(base + kTile, &tm_lo, &bar.q_full[g], p.q_col + h * HD, tile * QM, b);
            }
            mbar_arrive_expect_tx(&bar.k_full[g], 2 * kTile);
            tma_load_3d(base + 2 * kTile, &tm_hi, &bar.k_full[g], p.k_col + h * HD, j * KV, b);
            tma_load_3d(base + 3 * kTile, &tm_lo, &bar.k_full[g], p.k_col + h * HD, j * KV, b);
            ++kn[g];
            did = true;
          }
          if (vn[g] < n[g] && vn[g] < kn[g] && (vn[g] == 0 || mbar_test(&bar.pv_done[g], (uint32_t)((vn[g] - 1) & 1)))) {
            const int k = vn[g] / blocks, j = vn[g] - k * blocks;
            place(g, k, &tile, &h, &b);
            mbar_arrive_expect_tx(&bar.v_full[g], 2 * kTile);
            tma_load_3d(base + 4 * kTile, &tm_hi, &bar.v_full[g], p.v_col + h * HD, j * KV, b);
            tma_load_3d(base + 5 * kTile, &tm_lo, &bar.v_full[g], p.v_col + h * HD, j * KV, b);
            ++vn[g];
            did = true;
          }
        }
        idle = did ? 0 : idle + 1;
        if (idle > kPollLimit) {
          atomicExch(p.err, 51);
          for (int g = 0; g < 2; ++g) {         // copies in flight land
            if (kn[g] > 0) (void)mbar_wait(&bar.k_full[g], (uint32_t)((kn[g] - 1) & 1));
            if (vn[g] > 0) (void)mbar_wait(&bar.v_full[g], (uint32_t)((vn[g] - 1) & 1));
          }
          break;
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (elect_one()) {
      int sn[2] = {0, 0}, pn[2] = {0, 0};       // blocks whose scores / products have been issued
      const int n[2] = {items_of(0) * blocks, items_of(1) * blocks};
      uint32_t idle = 0;
      while (pn[0] < n[0] || pn[1] < n[1]) {
        bool did = false;
        for (int g = 0; g < 2; ++g) {
          const uint32_t base = smem_u32(smem + g * kGroupBytes), s_col = tmem + (uint32_t)(g * 128), o_col = tmem + kOCol + (uint32_t)(g * 128);
          // P V of block pn, once P is written (the scores of the block have been issued before).
          if (pn[g] < sn[g] && mbar_test(&bar.p_ready[g], (uint32_t)(pn[g] & 1)) && mbar_test(&bar.v_full[g], (uint32_t)(pn[g] & 1))) {
            tc_fence_after();
            const int j = pn[g] % blocks, chunks = (min(KV, T - j * KV) + 15) / 16;
            const uint32_t id128 = (1u << 4) | (1u << 16) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(QM >> 4) << 24);   // B MN-major
            const uint32_t id64 = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(QM >> 4) << 24);
            const uint64_t v = desc_mn128(base + 4 * kTile);
            auto hi = [&](int c) {              // P_hi * [V_hi | V_lo]
              mma_f16_ta(o_col, s_col + (uint32_t)(16 * c), v + (uint64_t)(c * 128), id128, (j % kRun > 0 || c > 0) ? 1u : 0u);
            };
            auto lo = [&](int c) {              // P_lo * V_hi, beside the other cross terms
              mma_f16_ta(o_col + (uint32_t)HD, s_col + (uint32_t)(16 * c + 8), v + (uint64_t)(c * 128), id64, 1u);
            };
            if (chunks == KV / 16) {            // unrolled: half the time to issue an instruction
#pragma unroll
              for (int c = 0; c < KV / 16; ++c) hi(c);
#pragma unroll
              for (int c = 0; c < KV / 16; ++c) lo(c);
            } else {
#pragma unroll 1
              for (int c = 0; c < chunks; ++c) hi(c);
#pragma unroll 1
              for (int c = 0; c < chunks; ++c) lo(c);
            }
            tc_commit(&bar.pv_done[g]);
            ++pn[g];
            did = true;
          }
          // Scores of block sn over the P of the block before, whose products must be complete (MMAs of another shape and
          // accumulator are not among those that PTX keeps in order).
          if (sn[g] < n[g] && sn[g] == pn[g] && mbar_test(&bar.k_full[g], (uint32_t)(sn[g] & 1)) &&
              (sn[g] == 0 || mbar_test(&bar.pv_done[g], (uint32_t)((sn[g] - 1) & 1))) &&
              (sn[g] % blocks != 0 || mbar_test(&bar.q_full[g], (uint32_t)((sn[g] / blocks) & 1)))) {
            tc_fence_after();
            const int j = sn[g] % blocks, ns = (min(KV, T - j * KV) + 15) / 16 * 16;
            const uint32_t idesc = (1u << 4) | ((uint32_t)(ns >> 3) << 17) | ((uint32_t)(QM >> 4) << 24);
            const uint64_t q_hi = desc_sw128(base), q_lo = desc_sw128(base + kTile);
            const uint64_t k_hi = desc_sw128(base + 2 * kTile), k_lo = desc_sw128(base + 3 * kTile);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {   // the cross terms, 2^-11 of the scores, while the sum is small
              const uint64_t off = (uint64_t)(kk * 32 >> 4);
              tc_mma_f16(s_col, q_lo + off, k_hi + off, idesc, kk ? 1u : 0u);
              tc_mma_f16(s_col, q_hi + off, k_lo + off, idesc, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint64_t off = (uint64_t)(kk * 32 >> 4);
              tc_mma_f16(s_col, q_hi + off, k_hi + off, idesc, 1u);
            }
            tc_commit(&bar.s_full[g]);
            ++sn[g];
            did = true;
          }
        }
        idle = did ? 0 : idle + 1;
        if (idle > kPollLimit) { atomicExch(p.err, 52); break; }
      }
      // No arrival of a commit is still on its way to this block's barriers at exit.
      for (int g = 0; g < 2; ++g)
        if (pn[g] > 0 && !mbar_wait(&bar.pv_done[g], (uint32_t)((pn[g] - 1) & 1))) atomicExch(p.err, 53);
    }
  } else {
    const int g = warp >> 3, q = warp & 3, hf = (warp >> 2) & 1;
    const int row = q * 32 + lane;
    float(*xch)[QM] = xch_all[g];
    const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
    float* sums = p.sums + ((size_t)(2 * blockIdx.x + g) * HD + hf * 32) * QM + row;   // [column][row], written and read by this thread only
    const uint32_t scol = trow + (uint32_t)(g * 128 + hf * 64), ocol = trow + kOCol + (uint32_t)(g * 128 + hf * 32);
    // Scores arrive as (q * 2^8) . (k * 2^8); t = acc * c1 with c1 = 2^-16 * log2(e) (* | /) scale.
    const float kLog2e = 1.44269504088896341f;
    const float sc = SMODE ? ld_plain(p.scale) : 1.f;
    const float c1 = __fmul_rn(SMODE == 1 ? __fmul_rn(sc, kLog2e) : (SMODE == 2 ? __fdiv_rn(kLog2e, sc) : kLog2e),
                               kFixedUnscale * kFixedUnscale);
    float seen_max = 0.f;
    bool ok = true;
    int nb = 0;                                 // running block of this group
    const int my_items = items_of(g);
#pragma unroll 1
    for (int k = 0; k < my_items; ++k) {
      float ref = 0.f, sum = 0.f, since = 1.f;  // since: factor of the moves of ref since `sums` was written
#pragma unroll 1
      for (int j = 0; j < blocks; ++j, ++nb) {
        const int left = T - j * KV - hf * 64;  // keys of this thread's half that exist
        if (ok && !warp_mbar_wait(&bar.s_full[g], (uint32_t)(nb & 1), lane)) { atomicExch(p.err, 54); ok = false; }
        tc_fence_after();
        uint32_t s[64];
#pragma unroll
        for (int c = 0; c < 4; ++c) tc_ld_32x16(scol + (uint32_t)(16 * c), *reinterpret_cast<uint32_t(*)[16]>(&s[16 * c]));
        tc_wait_ld(s);
        float m = -CUDART_INF_F;
        if (left >= 64) {
          float m4[4] = {m, m, m, m};
#pragma unroll
          for (int e = 0; e < 64; e += 2)
            m4[e / 2 & 3] = fmax3(m4[e / 2 & 3], __fmul_rn(__uint_as_float(s[e]), c1), __fmul_rn(__uint_as_float(s[e + 1]), c1));
          m = fmaxf(fmax3(m4[0], m4[1], m4[2]), m4[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (e < left) m = fmaxf(m, __fmul_rn(__uint_as_float(s[e]), c1));
        }
        xch[hf][row] = m;
        pair_sync(g, q);
        m = fmaxf(xch[0][row], xch[1][row]);
        pair_sync(g, q);
        const bool move = j > 0 && __any_sync(0xffffffffu, m > ref + 4.f);   // the same rows, so the same vote, in both warps
        const bool flush = j > 0 && j % kRun == 0;             // this block's products start the accumulator again
        if (j == 0) ref = m;
        if (flush || move) {
          // Free: the scores that have just been read were issued when these products were complete.
          if (ok && !warp_mbar_wait(&bar.pv_done[g], (uint32_t)((nb - 1) & 1), lane)) { atomicExch(p.err, 55); ok = false; }
          tc_fence_after();
        }
        if (flush) {
#pragma unroll
          for (int part = 0; part < 2; ++part) {   // this warp's 32 columns
            uint32_t o[16], ol[16];
            tc_ld_32x16(ocol + (uint32_t)(part * 16), o);
            tc_ld_32x16(ocol + (uint32_t)(HD + part * 16), ol);
            tc_wait_ld(o, ol);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float* at = sums + (part * 16 + e) * QM;
              const float x = __fadd_rn(__uint_as_float(o[e]), __uint_as_float(ol[e]));
              *at = j == kRun ? x : fmaf(*at, since, x);
            }
          }
          since = 1.f;
        }
        if (move) {
          const float next = fmaxf(ref, m), f = ex2(__fsub_rn(ref, next));
          ref = next;
          sum = __fmul_rn(sum, f);
          since = __fmul_rn(since, f);
          if (!flush) {
#pragma unroll
            for (int part = 0; part < 4; ++part) {   // this warp's 32 columns of both halves of O
              const uint32_t at = ocol + (uint32_t)((part >> 1) * 64 + (part & 1) * 16);
              uint32_t o[16];
              tc_ld_32x16(at, o);
              tc_wait_ld(o);
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__fmul_rn(__uint_as_float(o[e]), f));
              st16(at, o);
            }
          }
        }
        const float off = __fsub_rn(ref, 9.f);
        float part_sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (16 * c >= left) break;            // uniform
          uint32_t w[16];                       // columns 0-7: hi of keys 2e, 2e + 1; columns 8-15: lo
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float e[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int col = 16 * c + 4 * i + x;
              e[x] = ex2(fmaf(__uint_as_float(s[col]), c1, -off));
              if (left < 64 && col >= left) e[x] = 0.f;
              part_sum[x] = __fadd_rn(part_sum[x], e[x]);
            }
            uint2 h2, l2;
            f16_split_plain(make_float4(e[0], e[1], e[2], e[3]), h2, l2);
            w[2 * i] = h2.x; w[2 * i + 1] = h2.y;
            w[8 + 2 * i] = l2.x; w[8 + 2 * i + 1] = l2.y;
          }
          st16(scol + (uint32_t)(16 * c), w);
        }
        sum = __fadd_rn(sum, __fadd_rn(__fadd_rn(part_sum[0], part_sum[1]), __fadd_rn(part_sum[2], part_sum[3])));
        wait_st();
        tc_fence_before();
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&bar.p_ready[g]);
      }
      xch[hf][row] = sum;
      pair_sync(g, q);
      sum = __fadd_rn(xch[0][row], xch[1][row]);
      pair_sync(g, q);
      if (ok && !warp_mbar_wait(&bar.pv_done[g], (uint32_t)((nb - 1) & 1), lane)) { atomicExch(p.err, 56); ok = false; }
      tc_fence_after();
      int tile, h, b;
      place(g, k, &tile, &h, &b);
      const float recip = __fmul_rn(__fdiv_rn(1.f, sum), kFixedUnscale);
      const int r = tile * QM + row;
      const bool mine = ok && r < T;
      const long long ob = (long long)b * p.out_batch_stride + h * HD + hf * 32;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t o[16], ol[16];
        tc_ld_32x16(ocol + (uint32_t)(half * 16), o);
        tc_ld_32x16(ocol + (uint32_t)(64 + half * 16), ol);
        tc_wait_ld(o, ol);
        uint4 yh[2], yl[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            y[e] = __fadd_rn(__uint_as_float(o[8 * i + e]), __uint_as_float(ol[8 * i + e]));
            if (blocks > kRun) y[e] = fmaf(sums[(half * 16 + 8 * i + e) * QM], since, y[e]);
            y[e] = __fmul_rn(y[e], recip);
          }
          const float4 y0 = make_float4(y[0], y[1], y[2], y[3]), y1 = make_float4(y[4], y[5], y[6], y[7]);
          if (p.out && mine) {
            float* at = p.out + ob + (long long)r * p.out_row_stride + half * 16 + 8 * i;
            *reinterpret_cast<float4*>(at) = y0;
            *reinterpret_cast<float4*>(at + 4) = y1;
          }
          uint2 h0, l0, h1, l1;
          f16_split_fixed(y0, h0, l0);
          f16_split_fixed(y1, h1, l1);
          yh[i] = make_uint4(h0.x, h0.y, h1.x, h1.y);
          yl[i] = make_uint4(l0.x, l0.y, l1.x, l1.y);
          if (mine) seen_max = split_track(split_track(seen_max, y0), y1);
        }
        if (p.o16_hi) {   // two lanes write 32 bytes of one row and then of the other: whole sectors
          lane_swap(yh[0], yh[1], lane & 1, 1);
          lane_swap(yl[0], yl[1], lane & 1, 1);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int ri = tile * QM + q * 32 + (lane & ~1) + i;
            if (!ok || ri >= T) continue;
            const long long at = (ob + (long long)ri * p.out_row_stride + half * 16 + 8 * (lane & 1)) >> 2;
            *reinterpret_cast<uint4*>(p.o16_hi + at) = yh[i];
            *reinterpret_cast<uint4*>(p.o16_lo + at) = yl[i];
          }
        }
      }
      tc_fence_before();   // the reads of O lie before the next item's arrival on p_ready
    }
    if (p.o16_hi) split_report_warp(split_seen_fixed_of_max(seen_max), p.err);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

template <int SMODE>
cudaError_t launch_mode(const Attention16Params& p, const FlashDev& d, cudaStream_t st) {
  constexpr int kDyn = 2 * kGroupBytes + 1024;
  static unsigned long long done = 0;
  if (cudaError_t e = ensure_dynamic_smem(attention_flash16_kernel<SMODE>, kDyn, &done)) return e;
  CUtensorMap hi, lo;
  if (!make_map16(&hi, p.qkv16_hi, p.ld16, p.tokens, p.batch, p.ld16, (int64_t)p.tokens * p.ld16, 128) ||
      !make_map16(&lo, p.qkv16_lo, p.ld16, p.tokens, p.batch, p.ld16, (int64_t)p.tokens * p.ld16, 128))
    return cudaErrorInvalidValue;
  const int grid = std::min(d.items, device_sm_count());
  return launch_pdl(attention_flash16_kernel<SMODE>, dim3((unsigned)grid), dim3(kLaunch), kDyn, st, 1, hi, lo, d);
}

}  // namespace

bool attention_flash16_shape_ok(int head_dim, int tokens, int64_t ld16, int64_t q_col, int64_t k_col, int64_t v_col,
                                int64_t out_row_stride, int64_t out_batch_stride) {
  return head_dim == HD && tokens >= 1 && tokens <= (1 << 20) && ld16 > 0 && (ld16 % 8) == 0 && (q_col % 8) == 0 &&
         (k_col % 8) == 0 && (v_col % 8) == 0 && q_col >= 0 && k_col >= 0 && v_col >= 0 &&
         (out_row_stride % 8) == 0 && (out_batch_stride % 8) == 0;
}

int64_t attention_flash16_workspace(int64_t batch, int64_t heads, int64_t tokens) {
  const int64_t items = batch * heads * ((tokens + QM - 1) / QM);
  return tokens > kRun * KV ? std::min<int64_t>(items, device_sm_count()) * 2 * HD * QM : 0;
}

cudaError_t launch_attention_flash16(const Attention16Params& p, cudaStream_t st) {
  auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!attention_flash16_shape_ok(p.head_dim, p.tokens, p.ld16, p.q_col, p.k_col, p.v_col, p.out_row_stride, p.out_batch_stride) ||
      p.batch < 1 || p.heads < 1 || !p.qkv16_hi || !p.qkv16_lo || !al(p.qkv16_hi) || !al(p.qkv16_lo) || !al(p.out) ||
      !al(p.out16_hi) || !al(p.out16_lo) || (!p.out && !(p.out16_hi && p.out16_lo)) ||
      (p.out16_hi == nullptr) != (p.out16_lo == nullptr) || !p.err_word ||
      std::max(std::max(p.q_col, p.k_col), p.v_col) + (int64_t)p.heads * HD > p.ld16)
    return cudaErrorInvalidValue;
  FlashDev d;
  d.out = p.out; d.out_row_stride = p.out_row_stride; d.out_batch_stride = p.out_batch_stride;
  d.o16_hi = static_cast<uint2*>(p.out16_hi); d.o16_lo = static_cast<uint2*>(p.out16_lo);
  d.heads = p.heads; d.tokens = p.tokens; d.tiles = (p.tokens + QM - 1) / QM; d.items = p.batch * p.heads * d.tiles;
  d.q_col = (int)p.q_col; d.k_col = (int)p.k_col; d.v_col = (int)p.v_col;
  d.scale = p.scale; d.scale_mode = p.scale ? p.scale_mode : 0;
  d.err = p.err_word;
  d.sums = p.workspace;
  if (p.tokens > kRun * KV && !p.workspace) return cudaErrorInvalidValue;
  if (d.scale_mode == 1) return launch_mode<1>(p, d, st);
  if (d.scale_mode == 2) return launch_mode<2>(p, d, st);
  return launch_mode<0>(p, d, st);
}

}  // namespace ac

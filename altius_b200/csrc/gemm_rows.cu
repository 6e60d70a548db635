// Products of a few rows with a [N, K] operand (classifier heads at small batches; reference:
// crates/session_interpreter/src/gemm.rs:36-110, session.rs:684-734):
//   C[m, n] = act(alpha * A[m, :] . B[n, :] + beta * Cin[m, n] + bias[n]) + residual[m, n]
// in fp32. Bound by reading B once (1000 x 768 floats: 3 MB, 0.5 us of HBM) and by latency: one warp
// per one or two columns n, its lanes along K with 16-byte loads, up to eight rows of A per warp (all
// warps of a block read the same ones: from L1, eight rows of more than 256 floats from shared memory). A tile kernel gives such a product 8 to 16 blocks
// with a split of the operands and a second pass behind it: 15 us for one row of 768 into 1000
// columns, here 3.
#include "kernels.h"
#include "pdl.cuh"
#include "ref_math.cuh"

namespace ac {
namespace {

constexpr int kWarps = 8, KC = 1024;

// Eight rows of A are more than a lane can have under way beside B: the block brings them to shared memory, KC
// floats of K at a time, while each lane already loads its part of B for the next four steps. 80 registers, so that
// three blocks share an SM. (Rows from L1, two steps at a time, two blocks: 16.8 of 20 issue slots waited for a load;
// 32 x 960 x 1280 19 us.)
__device__ __forceinline__ void cp16(float4* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int MT, int NW>
__device__ __forceinline__ void staged_products(const float* const (&a)[MT], const float* const (&b)[NW], int K, int lane, float (&acc)[NW][MT]) {
  __shared__ float4 as[MT * (KC / 4)];
  for (int kc = 0; kc < K; kc += KC) {
    const int kn = min(KC, K - kc), quads = kn / 4;
    if (kc) __syncthreads();                   // everybody is through with the part before
    for (int i = threadIdx.x; i < MT * (KC / 4); i += kWarps * 32) {
      const int r = i / (KC / 4), q = i % (KC / 4);
      const float* row = a[0];
#pragma unroll
      for (int e = 1; e < MT; ++e) row = r == e ? a[e] : row;
      if (q < quads) cp16(&as[i], row + kc + 4 * q);
    }
    float4 bv[4][NW];
    auto request = [&](int u, int k) {
#pragma unroll
      for (int j = 0; j < NW; ++j)
        bv[u][j] = k < kn ? ld_plain(reinterpret_cast<const float4*>(b[j] + kc + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
#pragma unroll
    for (int u = 0; u < 4; ++u) request(u, lane * 4 + 128 * u);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int k0 = lane * 4; k0 < kn; k0 += 512) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + 128 * u;
        if (k < kn) {
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            const float4 av = as[i * (KC / 4) + k / 4];
#pragma unroll
            for (int j = 0; j < NW; ++j)
              acc[j][i] = fmaf(av.x, bv[u][j].x, fmaf(av.y, bv[u][j].y, fmaf(av.z, bv[u][j].z, fmaf(av.w, bv[u][j].w, acc[j][i]))));
          }
        }
        request(u, k + 512);
      }
    }
  }
}

template <int MT, int NW, bool STAGED>
__global__ void __launch_bounds__(kWarps * 32, STAGED ? 3 : 1) gemm_rows_kernel(const GemmParams p) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = (blockIdx.x * kWarps + warp) * NW, m0 = blockIdx.y * MT;
  const int N = (int)p.n, M = (int)p.m, K = (int)p.k;
  pdl_trigger();
  pdl_wait();
  if (!STAGED && n0 >= N) return;
  const float* a[MT];
  const float* b[NW];
#pragma unroll
  for (int i = 0; i < MT; ++i) a[i] = p.a + (long long)min(m0 + i, M - 1) * p.lda;
#pragma unroll
  for (int j = 0; j < NW; ++j) b[j] = p.b + (long long)min(n0 + j, N - 1) * p.ldb;
  float acc[NW][MT];
#pragma unroll
  for (int j = 0; j < NW; ++j)
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[j][i] = 0.f;
  if (STAGED) staged_products<MT, NW>(a, b, K, lane, acc);
  else
#pragma unroll (MT <= 2 ? 4 : 2)
  for (int k = lane * 4; k < K; k += 128) {
    float4 bv[NW];
#pragma unroll
    for (int j = 0; j < NW; ++j) bv[j] = ld_plain(reinterpret_cast<const float4*>(b[j] + k));
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const float4 av = *reinterpret_cast<const float4*>(a[i] + k);
#pragma unroll
      for (int j = 0; j < NW; ++j)
        acc[j][i] = fmaf(av.x, bv[j].x, fmaf(av.y, bv[j].y, fmaf(av.z, bv[j].z, fmaf(av.w, bv[j].w, acc[j][i]))));
    }
  }
  // Lane j * MT + i keeps result (i, j): the epilogue's code exists once.
  float v = 0.f;
#pragma unroll
  for (int j = 0; j < NW; ++j)
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      float u = acc[j][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) u = __fadd_rn(u, __shfl_xor_sync(0xffffffffu, u, o));
      if (lane == j * MT + i) v = u;
    }
  const int m = m0 + lane % MT, n = n0 + lane / MT;
  if (lane >= NW * MT || m >= M || n >= N) return;
  if (p.alpha != 1.f) v = __fmul_rn(p.alpha, v);
  if (p.c_in && p.beta != 0.f) {
    const float cv = p.c_in[(long long)m * p.ldc_in + n];
    v = __fadd_rn(p.beta == 1.f ? cv : __fmul_rn(p.beta, cv), v);
  }
  if (p.bias_n) v = __fadd_rn(v, p.bias_scale == 1.f ? p.bias_n[n] : __fmul_rn(p.bias_scale, p.bias_n[n]));
  v = apply_act(p.act, v, p.act_alpha, p.act_beta);
  if (p.residual) v = __fadd_rn(v, p.residual[(long long)m * p.ld_res + n]);
  p.c[(long long)m * p.ldc + n] = v;
}

template <int MT, int NW, bool STAGED = false>
cudaError_t launch_t(const GemmParams& p, cudaStream_t st) {
  const dim3 grid((unsigned)((p.n + kWarps * NW - 1) / (kWarps * NW)), (unsigned)((p.m + MT - 1) / MT));
  return launch_pdl(gemm_rows_kernel<MT, NW, STAGED>, grid, dim3(kWarps * 32), 0, st, 1, p);
}

inline bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

bool gemm_rows_supported(const GemmParams& p) {
  return p.batch == 1 && !p.trans_a && p.trans_b && p.m >= 1 && p.m <= kGemmRowsMax && p.n >= 1 && p.n < (1ll << 30) &&
         p.k >= 4 && (p.k % 4) == 0 && (p.lda % 4) == 0 && (p.ldb % 4) == 0 && al16(p.a) && al16(p.b) && !p.bias_m &&
         !p.c16_hi && !p.b_row_scale && p.c;
}

cudaError_t launch_gemm_rows(const GemmParams& p, cudaStream_t st) {
  if (p.m == 1) return launch_t<1, 1>(p, st);
  if (p.m == 2) return launch_t<2, 1>(p, st);
  if (p.m <= 4) return launch_t<4, 2>(p, st);
  // A lane's two steps of K are under way at once without a detour: with them alone, shared memory only costs its barrier (5 to 32
  // rows, 40 and 1000 columns, call times: K = 32 to 128 0.7 us longer, 192 and 256 the same, 320 to 768 0.2 to 1.7 us shorter).
  return p.k > 256 ? launch_t<8, 2, true>(p, st) : launch_t<8, 2>(p, st);
}

}  // namespace ac

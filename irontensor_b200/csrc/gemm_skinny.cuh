// Projections of a handful of tokens: y[n, out] = x[n, in] W[out, in]^T with n <= 32, what a generation step and the shortest
// prompts need, with the QKV + rotary epilogue of gemm_sm100.cuh as an option.
//
// Bound: reading W once.  The 128 x 256 tiles of the tcgen05 kernel would put 12 CTAs on a 2048 -> 3072 projection (15 us; 12.6 MB
// of weights are 2 us at the HBM rate), so here every SM streams weights: a CTA owns 16 rows of W, its eight warps split
// the K range, and each lane reads 16 contiguous bytes of a row at a time with all the loads of a chunk in flight.  The products
// run on mma.sync m16n8k16: at two FLOPs per weight and token the tensor rate does not matter, and fragments loaded straight
// from global memory avoid shared memory, barriers and tensor memory set-up, which a 5 us kernel has no time for.  A quad's four
// lanes hold 8 consecutive k each; as A (weights) and B (tokens) use the same order of k, any order is a valid one.
// Partial sums of the eight warps meet in shared memory; the rotation evaluates its few sines itself (no table launch).
// Every CTA also reads all tokens of its K range from L2, n / 16 times the weights' bytes: that is what ends this kernel's
// range (L2 delivers about 7 TB/s in all).  2048 -> 3072: 4.2 us up to 8 tokens, 5.4 at 16, 7.3 at 32 (tcgen05 tiles of 64
// columns: 7.7); 4096 -> 12288: 20 us at 8 tokens, 30 at 16 (tcgen05 tiles of 128 columns: 22).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

#include "rope.cuh"
#include "sm100_ptx.cuh"

namespace it {

struct SkinnyParams {
  const __nv_bfloat16* x;   // [n, K]
  const __nv_bfloat16* w;   // [N, K]
  __nv_bfloat16* y;         // [n, N]; null: the QKV epilogue
  int n, K, N;
  // QKV epilogue (see GemmParams)
  __nv_bfloat16 *q, *k, *v;
  int seq, heads, kv_heads, head_dim;
  long long ld_q, ld_kv;
};

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of 8 tokens.
template <int NT>
__global__ void __launch_bounds__(256)
gemm_skinny_kernel(const SkinnyParams p, const __grid_constant__ RopeFreqs freqs) {
  constexpr int WARPS = 8, U = NT <= 2 ? 4 : 2;    // U: steps of 32 k whose loads are in flight together
  constexpr int TOK = NT * 8, ROWS = 16;
  __shared__ float part[WARPS][ROWS][TOK + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * ROWS;
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  // chunks of U steps of 32 k go to the warps in turn: a row of a chunk is U * 64 contiguous bytes
  const int steps = (p.K + 31) >> 5;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int s0 = warp * U; s0 < steps; s0 += WARPS * U) {
    uint4 a[U][2], b[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (s0 + u) * 32 + t * 8;
      const bool ok = k < p.K;    // K is a multiple of 8
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = r0 + h * 8 + g;
        a[u][h] = (ok && row < p.N) ? __ldg(reinterpret_cast<const uint4*>(p.w + static_cast<size_t>(row) * p.K + k)) : zero;
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int tok = j * 8 + g;
        b[u][j] = (ok && tok < p.n) ? *reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(tok) * p.K + k) : zero;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_bf16_16816(acc[j], a[u][0].x, a[u][1].x, a[u][0].y, a[u][1].y, b[u][j].x, b[u][j].y);
        mma_bf16_16816(acc[j], a[u][0].z, a[u][1].z, a[u][0].w, a[u][1].w, b[u][j].z, b[u][j].w);
      }
  }
  // c0, c1: row g, tokens 2t, 2t + 1; c2, c3: row g + 8
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][(e >> 1) * 8 + g][j * 8 + t * 2 + (e & 1)] = acc[j][e];
  __syncthreads();
  // a thread finishes pairs of neighbouring columns of y: a rotation pair
  for (int idx = threadIdx.x; idx < TOK * (ROWS / 2); idx += 256) {
    const int tok = idx / (ROWS / 2), pr = idx - tok * (ROWS / 2);
    const int col = r0 + 2 * pr;
    if (tok >= p.n || col >= p.N) continue;
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      v0 += part[w][2 * pr][tok];
      v1 += part[w][2 * pr + 1][tok];
    }
    __nv_bfloat16* dst;
    if (p.y != nullptr) {
      dst = p.y + static_cast<size_t>(tok) * p.N + col;
    } else {
      const int hd = p.heads * p.head_dim, kv = p.kv_heads * p.head_dim;
      const bool is_q = col < hd, is_v = col >= hd + kv;
      const int cc = is_q ? col : is_v ? col - hd - kv : col - hd;
      dst = (is_q ? p.q : is_v ? p.v : p.k) + static_cast<long long>(tok) * (is_q ? p.ld_q : p.ld_kv) + cc;
      if (freqs.enabled && !is_v) {
        float c, s;
        rope_sincos(freqs, tok % p.seq + freqs.position_offset, (cc % p.head_dim) >> 1, &c, &s);
        const float x0 = v0;
        v0 = x0 * c - v1 * s;
        v1 = x0 * s + v1 * c;
      }
    }
    *reinterpret_cast<uint32_t*>(dst) = ptx::pack_bf16(v0, v1);
  }
}

}  // namespace it

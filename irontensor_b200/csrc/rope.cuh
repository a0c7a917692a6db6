// Rotary position embedding on [batch, seq, heads, head_dim] tensors, and its inverse.
//
// Follows the reference's rope_f32 / rope_backward_f32 (src/shaders/rope.metal:22-61,
// src/shaders/backward/rope.metal:25-62): for position p and dimension pair i,
//   theta_i = 1 / base^(2i / head_dim),  angle = float(p) * theta_i,
//   forward  (x0, x1) -> (x0 cos - x1 sin,  x0 sin + x1 cos)
//   backward (g0, g1) -> (g0 cos + g1 sin, -g0 sin + g1 cos)      (the transpose of the rotation).
// The reference runs the forward once for Q and once for K, and the backward once for dQ and once
// for dK.  Here Q and K are rotated by ONE launch (rope_qk_kernel), and the backward rotation is not
// a pass at all: the attention backward applies it where dQ and dK leave the chip (the fp32 -> bf16
// finish pass of dQ, the dK epilogue), see fa_bwd_sm100.cuh and fa_generic.cuh.
// Rotating K "on load" inside the attention kernels was rejected: every K tile is loaded once per
// query tile (S/128 times), every Q tile once per key tile in the backward, so the rotation would be
// redone that many times on shared-memory tiles of kernels that are shared-memory bound.
// theta_i comes from the host as a table computed in fp32 exactly as the shader does (powf, then one
// division), so that a CPU check multiplies the position by bit-identical frequencies.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

#include "sm100_ptx.cuh"

namespace it {

struct RopeFreqs {
  float inv_freq[64];   // theta_i for i < head_dim / 2 (head_dim <= 128)
  int enabled;          // 0: no rotation
  int position_offset;  // position of sequence index 0 (KV-cache continuation, rope.metal:16)
};

__device__ __forceinline__ void rope_sincos(const RopeFreqs& f, int position, int pair, float* c, float* s) {
  const float angle = static_cast<float>(position) * f.inv_freq[pair];
  *c = cosf(angle);
  *s = sinf(angle);
}

__device__ __forceinline__ float rope_ld(const float* p) { return *p; }
__device__ __forceinline__ float rope_ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void rope_st(float* p, float v) { *p = v; }
__device__ __forceinline__ void rope_st(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// One CTA per (batch, position); thread t owns dimension pair t % (D/2) and walks the heads of Q
// and then of K (which may have fewer heads) with stride blockDim / (D/2), so each thread computes
// its sine and cosine once.  INVERSE applies the backward rotation.  In place is fine.
template <typename ST, bool INVERSE>
__global__ void __launch_bounds__(256)
rope_qk_kernel(const ST* __restrict__ q_in, const ST* __restrict__ k_in, ST* __restrict__ q_out, ST* __restrict__ k_out,
               int S, int H, int Hkv, int D, const __grid_constant__ RopeFreqs freqs) {
  const int half = D >> 1;
  const int pair = threadIdx.x % half;
  const int lane_head = threadIdx.x / half;
  const int heads_per_pass = blockDim.x / half;
  const long long bs = blockIdx.x;                 // batch * S + position
  const int pos = static_cast<int>(bs % S) + freqs.position_offset;
  float c, s;
  rope_sincos(freqs, pos, pair, &c, &s);
  if (INVERSE) s = -s;
  const int n_heads = H + (k_in != nullptr ? Hkv : 0);
  for (int hh = lane_head; hh < n_heads; hh += heads_per_pass) {
    const bool is_q = hh < H;
    const ST* src = is_q ? q_in + (bs * H + hh) * D : k_in + (bs * Hkv + (hh - H)) * D;
    ST* dst = is_q ? q_out + (bs * H + hh) * D : k_out + (bs * Hkv + (hh - H)) * D;
    const float x0 = rope_ld(src + 2 * pair), x1 = rope_ld(src + 2 * pair + 1);
    rope_st(dst + 2 * pair, x0 * c - x1 * s);
    rope_st(dst + 2 * pair + 1, x0 * s + x1 * c);
  }
}

// The same for rows of whole 16-byte chunks (head_dim a multiple of 8 in bf16, of 4 in fp32): a CTA owns `n_pos` positions,
// evaluates their sines and cosines once, at most one per thread, into shared memory, and streams the heads of Q and K in
// 16-byte chunks, four loads of a thread in flight and issued in front of the sines.  The kernel above evaluates them in
// every thread and moves 4 bytes per thread and head.  Bound: memory latency at the sizes of one layer (2 x 1003 positions, 16 + 4
// heads of 96 columns, bf16, inside a training step of attention: 118.5 -> 116.0 us for the step).
template <typename ST, bool INVERSE>
__global__ void __launch_bounds__(256)
rope_qk_chunks_kernel(const ST* q_in, const ST* k_in, ST* q_out, ST* k_out, long long rows, int n_pos, int S, int H, int Hkv, int D,
                      const __grid_constant__ RopeFreqs freqs) {
  constexpr int VEC = 16 / sizeof(ST);
  __shared__ float2 tab[256];
  const int half = D >> 1, per_head = D / VEC;
  const int n_heads = H + Hkv;
  const long long row0 = static_cast<long long>(blockIdx.x) * n_pos;
  const int n_rows = static_cast<int>(min(static_cast<long long>(n_pos), rows - row0));
  const int n_chunks = n_rows * n_heads * per_head;
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  // chunk index -> element offset in Q (or, past H heads, in K), local row and first column
  auto locate = [&](int i, bool* is_q, long long* off, int* r, int* d) {
    const int head_row = i / per_head;
    *d = (i - head_row * per_head) * VEC;
    *r = head_row / n_heads;
    const int hh = head_row - *r * n_heads;
    *is_q = hh < H;
    *off = (*is_q ? (row0 + *r) * H + hh : (row0 + *r) * Hkv + (hh - H)) * D + *d;
  };
  bool first = true;
  for (int base = static_cast<int>(threadIdx.x); first || base < n_chunks; base += 4 * 256) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * 256;
      if (i < n_chunks) {
        bool is_q;
        long long off;
        int r, d;
        locate(i, &is_q, &off, &r, &d);
        x[u] = *reinterpret_cast<const uint4*>((is_q ? q_in : k_in) + off);
      }
    }
    if (first) {   // every thread passes here once
      for (int t = static_cast<int>(threadIdx.x); t < n_rows * half; t += 256) {
        const int r = t / half;
        float c, s;
        rope_sincos(freqs, static_cast<int>((row0 + r) % S) + freqs.position_offset, t - r * half, &c, &s);
        tab[t] = make_float2(c, INVERSE ? -s : s);
      }
      __syncthreads();
      first = false;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * 256;
      if (i >= n_chunks) break;
      bool is_q;
      long long off;
      int r, d;
      locate(i, &is_q, &off, &r, &d);
      const float2* cs = &tab[r * half + (d >> 1)];
      ST* e = reinterpret_cast<ST*>(&x[u]);
#pragma unroll
      for (int p = 0; p < VEC / 2; ++p) {
        const float x0 = rope_ld(e + 2 * p), x1 = rope_ld(e + 2 * p + 1);
        rope_st(e + 2 * p, x0 * cs[p].x - x1 * cs[p].y);
        rope_st(e + 2 * p + 1, x0 * cs[p].y + x1 * cs[p].x);
      }
      *reinterpret_cast<uint4*>((is_q ? q_out : k_out) + off) = x[u];
    }
  }
}

// (cos, sin) of every (sequence index, dimension pair): [S][D/2] float2.  Built once per call for kernels that would
// otherwise evaluate the same sine and cosine once per head (the attention backward) or per column tile (the fused QKV
// projection).  `first` and `stride` number the threads that share the work.
__device__ __forceinline__ void rope_fill_table(float2* table, int S, int half, const RopeFreqs& freqs, long long first, long long stride) {
  const long long n = static_cast<long long>(S) * half;
  for (long long i = first; i < n; i += stride) {
    const int pos = static_cast<int>(i / half), pair = static_cast<int>(i - static_cast<long long>(pos) * half);
    float c, s;
    rope_sincos(freqs, pos + freqs.position_offset, pair, &c, &s);
    table[i] = make_float2(c, s);
  }
}
__global__ void rope_table_kernel(float2* __restrict__ table, int S, int half, const __grid_constant__ RopeFreqs freqs) {
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  rope_fill_table(table, S, half, freqs, static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x,
                  static_cast<long long>(gridDim.x) * blockDim.x);
}

}  // namespace it

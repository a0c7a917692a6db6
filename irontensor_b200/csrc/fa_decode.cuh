// Attention for one new token per sequence against a key/value cache ("decode"): q [batch, heads, D],
// caches [batch, max_len, kv_heads, D], the first kv_len positions valid.
//
// The reference has no key/value cache: its generator re-runs the whole forward for every token
// (src/inference/generator.rs:146-200) and lists the cache as future work (docs/PRESENTATION.md:576).
// The result here equals the last row of its causal attention over the kv_len tokens
// (src/shaders/flash_attention.metal:167-223 with q = kv_len - 1), computed from the cache alone.
//
// The op is bound by reading the cache once (2 * kv_len * kv_heads * D elements per batch entry) and, for short caches, by
// the chain launch -> load -> softmax -> merge.  So:
//   * a CTA serves the query heads of one K/V head together (grouped-query attention: the cache rows are read once
//     per group, not once per query head), in chunks of at most 8 heads;
//   * cache rows go straight from global memory to registers, 16 bytes per lane: LK lanes share a key, a warp works on
//     32 / LK keys at a time and U such groups of keys (and as many of values) are in flight per warp.  No shared memory and
//     no barrier until the end; each group of LK lanes keeps its own running (max, sum, output) of the online softmax
//     (the recurrence of flash_attention.metal:27-41), merged once: lanes, then warps, then CTAs;
//   * the keys are split over CTAs when batch * kv_heads alone cannot fill the GPU (split-KV).  Up to 8 splits form a
//     thread-block cluster and merge through distributed shared memory in the same launch; more leave partial results for
//     fa_decode_merge_kernel.
// fp32 math in the exp2 domain; bf16 or fp32 storage; D a multiple of 8, at most 128.
// Long bf16 caches with head_dim 64 or 128 go through the tensor-core pipeline instead (fa_fwd_pp_sm100.cuh, DECODE), which
// streams the cache by TMA; both leave the same partial results for fa_decode_merge_kernel.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <cstdint>

#include "sm100_ptx.cuh"

namespace it {

constexpr int DEC_WARPS = 8;
constexpr int DEC_MAX_CLUSTER = 8;   // the portable limit

template <typename ST> struct DecVec;   // 16 bytes of storage as floats
template <> struct DecVec<float> {
  static constexpr int N = 4;
  __device__ static void unpack(const uint4& v, float (&f)[4]) {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
  }
};
template <> struct DecVec<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void unpack(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
};
__device__ __forceinline__ void dec_st(float* p, float v) { *p = v; }
__device__ __forceinline__ void dec_st(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

struct DecodeParams {
  int H, Hkv, D;
  int kv_len;          // valid cache positions
  long long cache_batch_stride;   // elements between batch entries of a cache (max_len * Hkv * D)
  int n_splits;        // key ranges; grid.x
  int split_len;       // keys per range
  int clustered;       // the ranges of a (batch, K/V head) are one cluster
  float scale_log2;    // 1/sqrt(D) * log2(e)
};

// grid: (n_splits, batch * Hkv, head chunks of the group).  LK: lanes per key, the power of two that covers D.  GC: query
// heads per CTA.
template <typename ST, int LK, int GC>
__global__ void __launch_bounds__(32 * DEC_WARPS, GC <= 4 ? 2 : 1)
fa_decode_kernel(const ST* __restrict__ q, const ST* __restrict__ k_cache, const ST* __restrict__ v_cache, ST* __restrict__ o,
                 float* __restrict__ lse, float* __restrict__ part_o, float* __restrict__ part_ml, const DecodeParams prm) {
  constexpr int VN = DecVec<ST>::N, KPW = 32 / LK, U = GC >= 4 ? 2 : 4;
  constexpr int DP = LK * VN;                          // D rounded up
  __shared__ float s_acc[DEC_WARPS][GC][DP];           // each warp's output, relative to its maximum
  __shared__ float s_ml[DEC_WARPS][GC][2];
  __shared__ float c_acc[GC][DP];                      // the CTA's output and (maximum, sum): what the other CTAs of a cluster read
  __shared__ float c_ml[GC][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane % LK, grp = lane / LK;
  const int D = prm.D, G = prm.H / prm.Hkv;
  const int b = static_cast<int>(blockIdx.y) / prm.Hkv, hk = static_cast<int>(blockIdx.y) % prm.Hkv;
  const int g0 = static_cast<int>(blockIdx.z) * GC;    // first head of this chunk within the group
  const int gc = min(GC, G - g0);
  const size_t bh0 = static_cast<size_t>(b) * prm.H + hk * G + g0;   // first (batch, query head)
  const int sp = blockIdx.x;
  const int k_begin = sp * prm.split_len, k_end = min(prm.kv_len, k_begin + prm.split_len);
  const bool col_ok = sub * VN < D;
  const size_t row_stride = static_cast<size_t>(prm.Hkv) * D;
  const size_t base = static_cast<size_t>(b) * prm.cache_batch_stride + static_cast<size_t>(hk) * D + sub * VN;
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();

  float qf[GC][VN], acc[GC][VN], m[GC], l[GC];
#pragma unroll
  for (int g = 0; g < GC; ++g) {
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (g < gc && col_ok) w = *reinterpret_cast<const uint4*>(q + (bh0 + g) * D + sub * VN);
    DecVec<ST>::unpack(w, qf[g]);
#pragma unroll
    for (int e = 0; e < VN; ++e) {
      qf[g][e] *= prm.scale_log2;
      acc[g][e] = 0.f;
    }
    m[g] = -INFINITY;
    l[g] = 0.f;
  }
  for (int k0 = k_begin + warp * (U * KPW); k0 < k_end; k0 += DEC_WARPS * U * KPW) {
    uint4 kr[U], vr[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int key = k0 + u * KPW + grp;
      kr[u] = vr[u] = make_uint4(0u, 0u, 0u, 0u);
      if (key < k_end && col_ok) kr[u] = __ldg(reinterpret_cast<const uint4*>(k_cache + base + static_cast<size_t>(key) * row_stride));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int key = k0 + u * KPW + grp;
      if (key < k_end && col_ok) vr[u] = __ldg(reinterpret_cast<const uint4*>(v_cache + base + static_cast<size_t>(key) * row_stride));
    }
    float s[U][GC];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[VN];
      DecVec<ST>::unpack(kr[u], f);
#pragma unroll
      for (int g = 0; g < GC; ++g) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < VN; ++e) a = fmaf(f[e], qf[g][e], a);
        s[u][g] = a;
      }
    }
#pragma unroll
    for (int off = LK / 2; off > 0; off >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int g = 0; g < GC; ++g) s[u][g] += __shfl_xor_sync(0xffffffffu, s[u][g], off);
#pragma unroll
    for (int g = 0; g < GC; ++g) {
      float mx = m[g];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + u * KPW + grp >= k_end) s[u][g] = -INFINITY;
        mx = fmaxf(mx, s[u][g]);
      }
      const float m_ref = (mx == -INFINITY) ? 0.f : mx;   // no key seen yet by these lanes: stay at (-inf, 0)
      const float corr = ptx::ex2(m[g] - m_ref);
      m[g] = mx;
      l[g] *= corr;
#pragma unroll
      for (int e = 0; e < VN; ++e) acc[g][e] *= corr;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        s[u][g] = ptx::ex2(s[u][g] - m_ref);
        l[g] += s[u][g];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[VN];
      DecVec<ST>::unpack(vr[u], f);
#pragma unroll
      for (int g = 0; g < GC; ++g)
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[g][e] = fmaf(s[u][g], f[e], acc[g][e]);
    }
  }
  // lanes: the key groups of a warp
#pragma unroll
  for (int g = 0; g < GC; ++g) {
    float mx = m[g];
#pragma unroll
    for (int off = LK; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float f = (m[g] == -INFINITY) ? 0.f : ptx::ex2(m[g] - mx);
    l[g] *= f;
#pragma unroll
    for (int e = 0; e < VN; ++e) acc[g][e] *= f;
#pragma unroll
    for (int off = LK; off < 32; off <<= 1) {
      l[g] += __shfl_xor_sync(0xffffffffu, l[g], off);
#pragma unroll
      for (int e = 0; e < VN; ++e) acc[g][e] += __shfl_xor_sync(0xffffffffu, acc[g][e], off);
    }
    if (grp == 0) {
#pragma unroll
      for (int e = 0; e < VN; ++e) s_acc[warp][g][sub * VN + e] = acc[g][e];
      if (sub == 0) {
        s_ml[warp][g][0] = mx;
        s_ml[warp][g][1] = l[g];
      }
    }
  }
  __syncthreads();
  // warps: a CTA has at least one key, so the maximum is finite
  for (int i = threadIdx.x; i < gc * DP; i += 32 * DEC_WARPS) {
    const int g = i / DP, d = i % DP;
    float mx = s_ml[0][g][0];
#pragma unroll
    for (int w = 1; w < DEC_WARPS; ++w) mx = fmaxf(mx, s_ml[w][g][0]);
    float a = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float f = (s_ml[w][g][0] == -INFINITY) ? 0.f : ptx::ex2(s_ml[w][g][0] - mx);
      a = fmaf(f, s_acc[w][g][d], a);
      sum = fmaf(f, s_ml[w][g][1], sum);
    }
    if (prm.n_splits == 1) {
      if (d < D) dec_st(o + (bh0 + g) * D + d, a / sum);
      if (d == 0 && lse != nullptr) lse[bh0 + g] = (mx + log2f(sum)) * 0.6931471805599453f;
    } else if (!prm.clustered) {
      const size_t ps = (bh0 + g) * prm.n_splits + sp;
      if (d < D) part_o[ps * D + d] = a;
      if (d == 0) {
        part_ml[ps * 2] = mx;
        part_ml[ps * 2 + 1] = sum;
      }
    } else {
      c_acc[g][d] = a;
      if (d == 0) {
        c_ml[g][0] = mx;
        c_ml[g][1] = sum;
      }
    }
  }
  if (!prm.clustered) return;
  // CTAs of the cluster: CTA r finishes every n_splits-th output element
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int n = prm.n_splits;
  for (int i = sp + static_cast<int>(threadIdx.x) * n; i < gc * DP; i += 32 * DEC_WARPS * n) {
    const int g = i / DP, d = i % DP;
    float ms[DEC_MAX_CLUSTER], ls[DEC_MAX_CLUSTER], as[DEC_MAX_CLUSTER], mx = -INFINITY;
#pragma unroll
    for (int r = 0; r < DEC_MAX_CLUSTER; ++r) {
      ms[r] = -INFINITY;
      if (r < n) {
        const float* ml = cluster.map_shared_rank(&c_ml[g][0], r);
        ms[r] = ml[0];
        ls[r] = ml[1];
        as[r] = *cluster.map_shared_rank(&c_acc[g][d], r);
      }
    }
#pragma unroll
    for (int r = 0; r < DEC_MAX_CLUSTER; ++r) mx = fmaxf(mx, ms[r]);
    float a = 0.f, sum = 0.f;
#pragma unroll
    for (int r = 0; r < DEC_MAX_CLUSTER; ++r)
      if (r < n) {
        const float f = ptx::ex2(ms[r] - mx);
        a = fmaf(f, as[r], a);
        sum = fmaf(f, ls[r], sum);
      }
    if (d < D) dec_st(o + (bh0 + g) * D + d, a / sum);
    if (d == 0 && lse != nullptr) lse[bh0 + g] = (mx + log2f(sum)) * 0.6931471805599453f;
  }
  cluster.sync();   // nobody's shared memory goes away while it is read
}

// One CTA of 128 threads per (batch, head): merges the splits' partial results.  The first 64 threads turn the splits' maxima
// into weights, then every dimension is a sum of independent loads.  A split past kv_len has (m, l) = (-inf, 0).
constexpr int DEC_MAX_SPLITS = 64;
template <typename ST>
__global__ void __launch_bounds__(128)
fa_decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                       ST* __restrict__ o, float* __restrict__ lse, int n_splits, int D) {
  __shared__ float s_w[DEC_MAX_SPLITS], s_mx[2], s_sum[2];
  const size_t bh = blockIdx.x;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  ptx::grid_dep_wait();     // the partial results come from the kernel in front
  ptx::grid_dep_launch();
  float m = -INFINITY, l = 0.f;
  if (t < n_splits) {
    const float2 ml = *reinterpret_cast<const float2*>(part_ml + (bh * n_splits + t) * 2);
    m = ml.x;
    l = ml.y;
  }
  float mx = m;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if (warp < 2 && lane == 0) s_mx[warp] = mx;
  __syncthreads();
  mx = fmaxf(s_mx[0], s_mx[1]);
  const float w = (m == -INFINITY) ? 0.f : ptx::ex2(m - mx);
  if (t < DEC_MAX_SPLITS) s_w[t] = w;
  float sum = l * w;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if (warp < 2 && lane == 0) s_sum[warp] = sum;
  __syncthreads();
  sum = s_sum[0] + s_sum[1];
  if (t < D) {
    float acc = 0.f;
    const float* p = part_o + bh * n_splits * D + t;
#pragma unroll 8
    for (int s = 0; s < n_splits; ++s)
      if (s_w[s] != 0.f) acc = fmaf(p[static_cast<size_t>(s) * D], s_w[s], acc);
    dec_st(o + bh * D + t, acc / sum);
  }
  if (t == 0 && lse != nullptr) lse[bh] = (mx + log2f(sum)) * 0.6931471805599453f;
}

}  // namespace it

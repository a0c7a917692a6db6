// Rows of causal attention and its gradients over the visible (query, key) pairs alone, on CUDA cores.
//
// A tensor-core tile on the diagonal multiplies its masked probabilities, which are 0, by whole operand tiles, and 0 times an
// infinity or a NaN is NaN: one non-finite row of V (forward), of K or V (dQ) or of Q or dO (dK, dV) would reach every row of
// its diagonal tile, rows that do not see it included.  The kernels that took shapes over from CUDA-core kernels, which walk
// visible pairs only, therefore look at the finished rows and have one that is not finite computed again here (a row that sees
// the non-finite one comes out non-finite again).  Finite rows pay for the look, one FMA per value.  The look is taken behind
// the loops over tiles: a call inside them cost the registers of its arguments all the time (B2 S1003 H16 Hkv4 D96, backward
// with its forward: 111 -> 137 us).
// A thread computes four columns at a time from global memory, so a tensor full of NaN is slow, but no slower than it was.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

#include "layout.cuh"
#include "sm100_ptx.cuh"

namespace it {

// Operands of one launch: q and dO laid out by `st`, k and v by `st_kv` (whose slice() takes a query slice).
template <typename ST>
struct VisiblePairs {
  const ST *q, *k, *v, *d_o;
  TensorStrides st, st_kv;
  int D;
  float scale_log2;   // 1/sqrt(D) * log2(e)
  __device__ const ST* row_of(const ST* p, const TensorStrides& s, int bh, int i) const {
    return p + s.slice(bh) + static_cast<long long>(i) * s.row;
  }
};

__device__ __forceinline__ float4 vp_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 vp_ld4(const __nv_bfloat16* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u), __uint_as_float(w.y << 16),
                     __uint_as_float(w.y & 0xFFFF0000u));
}
template <typename ST>
__device__ __forceinline__ float vp_dot(const ST* a, const ST* b, int D) {
  float s = 0.f;
  for (int d = 0; d < D; d += 4) {
    const float4 x = vp_ld4(a + d), y = vp_ld4(b + d);
    s = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, s))));
  }
  return s;
}
__device__ __forceinline__ void vp_add(float4* acc, float w, const float4& x) {
  acc->x = fmaf(w, x.x, acc->x);
  acc->y = fmaf(w, x.y, acc->y);
  acc->z = fmaf(w, x.z, acc->z);
  acc->w = fmaf(w, x.w, acc->w);
}
// Nothing that follows changes it.
__device__ __forceinline__ bool vp_all_nan(const float4& a) { return a.x != a.x && a.y != a.y && a.z != a.z && a.w != a.w; }

// NaN if one of the values is an infinity or a NaN, 0 otherwise; chain over several.
__device__ __forceinline__ float nonfinite(float z, float x) { return fmaf(x, 0.f, z); }
__device__ __forceinline__ bool any_nonfinite(const float4& v) {
  return nonfinite(nonfinite(nonfinite(nonfinite(0.f, v.x), v.y), v.z), v.w) != 0.f;
}

// O[i][col .. col+3] = sum over keys [0, i] of 2^(s * scale_log2 - m) * inv_l * V.
template <typename ST>
__device__ __noinline__ float4 visible_o(const VisiblePairs<ST>& t, int bh, int i, int col, float m, float inv_l) {
  const ST* qi = t.row_of(t.q, t.st, bh, i);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = 0; j <= i && !vp_all_nan(acc); ++j) {
    const float p = ptx::ex2(fmaf(vp_dot(qi, t.row_of(t.k, t.st_kv, bh, j), t.D), t.scale_log2, -m));
    vp_add(&acc, p, vp_ld4(t.row_of(t.v, t.st_kv, bh, j) + col));
  }
  return make_float4(acc.x * inv_l, acc.y * inv_l, acc.z * inv_l, acc.w * inv_l);
}

// dQ[i][col .. col+3] from keys [0, k_hi), without the factor 1/sqrt(D).
template <typename ST>
__device__ __noinline__ float4 visible_dq(const VisiblePairs<ST>& t, int bh, int i, int k_hi, int col, float lse2, float delta) {
  const ST *qi = t.row_of(t.q, t.st, bh, i), *di = t.row_of(t.d_o, t.st, bh, i);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = 0; j < k_hi && !vp_all_nan(acc); ++j) {
    const ST* kj = t.row_of(t.k, t.st_kv, bh, j);
    const float p = ptx::ex2(fmaf(vp_dot(qi, kj, t.D), t.scale_log2, -lse2));
    vp_add(&acc, p * (vp_dot(di, t.row_of(t.v, t.st_kv, bh, j), t.D) - delta), vp_ld4(kj + col));
  }
  return acc;
}

// Queries [j_lo, j_hi) of slice bh: their part of dK[i] (without 1/sqrt(D)) or dV[i], columns col .. col+3, added to `acc`.
// lse and delta: those of query 0 of the slice; lse_scale turns lse into base-2 logarithms.
template <typename ST>
__device__ __noinline__ float4 visible_dkv(const VisiblePairs<ST>& t, bool is_dk, int bh, int i, int j_lo, int j_hi, int col, const float* lse,
                                           float lse_scale, const float* delta, float4 acc) {
  const ST *ki = t.row_of(t.k, t.st_kv, bh, i), *vi = t.row_of(t.v, t.st_kv, bh, i);
  for (int j = j_lo; j < j_hi && !vp_all_nan(acc); ++j) {
    const ST *qj = t.row_of(t.q, t.st, bh, j), *dj = t.row_of(t.d_o, t.st, bh, j);
    const float p = ptx::ex2(fmaf(vp_dot(qj, ki, t.D), t.scale_log2, -lse[j] * lse_scale));
    if (is_dk)
      vp_add(&acc, p * (vp_dot(dj, vi, t.D) - delta[j]), vp_ld4(qj + col));
    else
      vp_add(&acc, p, vp_ld4(dj + col));
  }
  return acc;
}

// Through the inverse rotary rotation: cs = (cos, sin) of the two pairs.
__device__ __forceinline__ float4 rotate_back(const float4& g, const float4& cs) {
  return make_float4(g.x * cs.x + g.y * cs.y, g.y * cs.x - g.x * cs.y, g.z * cs.z + g.w * cs.w, g.w * cs.z - g.z * cs.w);
}

}  // namespace it

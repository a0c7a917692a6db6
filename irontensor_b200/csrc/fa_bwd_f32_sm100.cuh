// Attention backward (dQ, dK, dV from Q, K, V, O, dO, LSE) for FP32 tensors on the sm_100a tensor cores.
//
// The reference trains in fp32 (src/train/helpers.rs:142-182).  As in the fp32 forward (fa_fwd_f32_sm100.cuh) every operand
// is split into three bf16 terms (24 mantissa bits) and a product of two split operands is the six term products of order
// above 2^-24, accumulated in fp32 in tensor memory.
//
// Two kinds of CTA in one launch, so that nothing is summed across CTAs and results are bit-reproducible:
//   dQ CTA (one 128-row query tile)      : stationary X0 = Q, X1 = dO;  streamed Y0 = K, Y1 = V
//   dK/dV CTA (one 128-row key tile)     : stationary X0 = K, X1 = V;   streamed Y0 = Q, Y1 = dO
// With T0 = X0 Y0^T (the scores, or their transpose) and T1 = X1 Y1^T (dP, or its transpose) both kinds do the same:
//   P = 2^(T0 c - LSE log2e),  dS = P o (T1 - delta),  acc0 = dS Y0  (dQ, or dK),  acc1 = P Y1  (dV; dK/dV CTA only).
// The accumulators are those of one tile; the math warps add them up in the output rows (see `drain`).
// The scores are computed twice, seven contractions in place of five; in exchange dS is only ever an A operand in the
// orientation it is produced in, so it goes registers -> tensor memory -> MMA and never through shared memory (which the
// twelve operand planes fill), and dQ needs neither an fp32 accumulator in memory nor its clearing and read-back.
//
// Roles: warps 0-3 and 4-7 math (a thread owns one row and one half of the 128 columns), warps 8-11 loaders (fp32 rows ->
// registers -> three swizzled bf16 planes), warp 12 tensor-memory allocation and the MMA-issuing thread.  Per tile the
// tensor core sees T0, T1, acc1, acc0: P is computed under T1, dS under acc1, Y1 is replaced under acc0; the exposed part
// of a tile is the store of Y0 (shared memory has room for one Y0) and, in a dQ CTA, dS.
// Tensor memory: T0 [0,128) + [128,192), T1 [192,320) + [320,384), acc0 [384,448), acc1 [448,512).  A math group writes the
// three planes of its 64 columns of P (96 columns of packed bf16) over its own 64 columns of T0, which it has read, and 32
// of the extra ones; dS over T1 likewise.
//
// Bound: the MMAs.  24 + 24 + 48 + 48 instructions of 64 or 32 cycles per 128 x 128 tile and head: 4600 cycles (dQ) and
// 6100 cycles (dK/dV).  Before this kernel the fp32 backward ran on CUDA cores, a warp per row: B16 H4 S256 D64 551 us,
// B8 H12 S512 D64 2865 us.
// head_dim <= 64, a multiple of 4; any sequence length (rows past it are zero planes and masked scores).
#pragma once
#include "fa_fwd_f32_sm100.cuh"
#include "rope.cuh"
#include "sm100_ptx.cuh"
#include "visible_pairs.cuh"

namespace it {

struct BwdF32Traits {
  static constexpr int BM = 128, DP = 64;
  static constexpr int PLANE_BYTES = 128 * 128;          // [128 rows][64 bf16], 128-byte swizzle
  static constexpr int SMEM_X0 = 0;                      // three planes each
  static constexpr int SMEM_X1 = SMEM_X0 + 3 * PLANE_BYTES;
  static constexpr int SMEM_Y0 = SMEM_X1 + 3 * PLANE_BYTES;
  static constexpr int SMEM_Y1 = SMEM_Y0 + 3 * PLANE_BYTES;
  static constexpr int SMEM_ROW = SMEM_Y1 + 3 * PLANE_BYTES;   // [2 tiles][128] -LSE*log2e, [2 tiles][128] -delta of the streamed rows
  static constexpr int SMEM_BAR = SMEM_ROW + 4 * 512;
  static constexpr int NUM_BARS = 11;
  static constexpr int SMEM_MISC = SMEM_BAR + NUM_BARS * 8;
  static constexpr int SMEM_BYTES = SMEM_MISC + 16;
  static constexpr int THREADS = 416;
  static constexpr uint32_t TMEM_COLS = 512;
  static constexpr uint32_t COL_T0 = 0, COL_E0 = 128, COL_T1 = 192, COL_E1 = 320, COL_ACC0 = 384, COL_ACC1 = 448;
};

struct BwdF32Params {
  const float* q;
  const float* k;
  const float* v;
  const float* d_o;
  const float* lse;           // [BH, S]
  const float* delta;         // [BH, S] rowsum(dO * O)
  float* dq;
  float* dk;
  float* dv;
  const float2* rope_table;   // [S][D/2] (cos, sin): dQ and dK leave through the inverse rotation; null: no rotation
  ptx::TensorStrides st;      // q, dO, dq
  ptx::TensorStrides st_kv;   // k, v, dk, dv
  int* status;
  int S, D, BH, causal;
  float scale;                // 1/sqrt(D)
  float scale_log2;           // scale * log2(e)
};

// delta[bh, s] = sum_d dO * O, and the rotary table when one is wanted.  A row is read by 16 lanes of 16 bytes; a warp
// covers eight rows with all its loads in flight before the first use.
__global__ void __launch_bounds__(256)
fa_bwd_f32_prepare_kernel(const float* __restrict__ o, const float* __restrict__ d_o, float* __restrict__ delta, long long rows, int S,
                          int D, ptx::TensorStrides st, float2* __restrict__ rope_table, const __grid_constant__ RopeFreqs freqs) {
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const int lane = threadIdx.x & 31, sub = lane & 15, half = lane >> 4;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long row0 = (tid >> 5) * 8;
  if (rope_table != nullptr) rope_fill_table(rope_table, S, D >> 1, freqs, tid, static_cast<long long>(gridDim.x) * blockDim.x);
  if (row0 >= rows) return;
  float4 a[4], b[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const long long row = row0 + 2 * r + half;
    a[r] = b[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows && sub * 4 < D) {
      const int bh = static_cast<int>(row / S);
      const long long off = st.slice(bh) + (row - static_cast<long long>(bh) * S) * st.row;
      a[r] = reinterpret_cast<const float4*>(o + off)[sub];
      b[r] = reinterpret_cast<const float4*>(d_o + off)[sub];
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float acc = fmaf(a[r].x, b[r].x, fmaf(a[r].y, b[r].y, fmaf(a[r].z, b[r].z, a[r].w * b[r].w)));
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    const long long row = row0 + 2 * r + half;
    if (sub == 0 && row < rows) delta[row] = acc;
  }
}

// The fp32 rows [128 * tile, 128 * tile + 128) of one slice, in the registers of 128 threads: thread t holds float4 column
// t & 15 of rows (t >> 4) + 8 i.  Rows past S and columns past D read as zero.
__device__ __forceinline__ void f32_tile_fetch(const float* base, long long row_stride, int tile, int S, int D, int t, float4 (&r)[16]) {
  const int c4 = t & 15, r0 = t >> 4;
  const bool col_ok = 4 * c4 < D;
  const int s0 = tile * 128 + r0;
  const float* p = base + static_cast<long long>(s0) * row_stride + 4 * c4;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (col_ok && s0 + 8 * i < S) r[i] = __ldg(reinterpret_cast<const float4*>(p + static_cast<long long>(8 * i) * row_stride));
  }
}
// ... split into three bf16 planes in the swizzled layout the MMA descriptors read.
__device__ __forceinline__ void f32_tile_store(uint8_t* planes, int t, const float4 (&r)[16]) {
  constexpr int PB = BwdF32Traits::PLANE_BYTES;
  const int c4 = t & 15, r0 = t >> 4;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    uint32_t h0, m0, l0, h1, m1, l1;
    split3_bf16x2(r[i].x, r[i].y, &h0, &m0, &l0);
    split3_bf16x2(r[i].z, r[i].w, &h1, &m1, &l1);
    const uint32_t off = ptx::swz128_offset(r0 + 8 * i, c4 * 4);
    *reinterpret_cast<uint2*>(planes + off) = make_uint2(h0, h1);
    *reinterpret_cast<uint2*>(planes + PB + off) = make_uint2(m0, m1);
    *reinterpret_cast<uint2*>(planes + 2 * PB + off) = make_uint2(l0, l1);
  }
  ptx::fence_proxy_async_smem();
}

// `width` columns of the finished row x_idx of dQ (KV: of dK or dV) from column `col` on, over the visible pairs alone and in fp32
// throughout.  For rows that are not finite; see visible_pairs.cuh.  Without the causal mask these too: a finite value above bf16's
// largest (3.39e38, as in masks of the lowest fp32 value) has no three bf16 terms, and infinities become NaN there.  `bh`: the row's query slice (KV: the first of the group).
template <bool KV>
__device__ __noinline__ void fa_bwd_f32_visible(const BwdF32Params& prm, int bh, int x_idx, bool is_dv, int col, int width, float* out) {
  const VisiblePairs<float> t{prm.q, prm.k, prm.v, prm.d_o, prm.st, prm.st_kv, prm.D, prm.scale_log2};
  constexpr float LOG2E = 1.4426950408889634f;
  for (int i = 0; i < width; i += 4) {
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h = 0; h < (KV ? prm.st_kv.group : 1); ++h) {
      const size_t r = static_cast<size_t>(bh + h) * prm.S;
      w = KV ? visible_dkv(t, !is_dv, bh + h, x_idx, prm.causal ? x_idx : 0, prm.S, col + i, prm.lse + r, LOG2E, prm.delta + r, w)
             : visible_dq(t, bh, x_idx, prm.causal ? x_idx + 1 : prm.S, col + i, prm.lse[r + x_idx] * LOG2E, prm.delta[r + x_idx]);
    }
    if (!is_dv) {
      w = make_float4(w.x * prm.scale, w.y * prm.scale, w.z * prm.scale, w.w * prm.scale);
      if (prm.rope_table != nullptr)
        w = rotate_back(w, *reinterpret_cast<const float4*>(prm.rope_table + static_cast<size_t>(x_idx) * (prm.D >> 1) + ((col + i) >> 1)));
    }
    *reinterpret_cast<float4*>(out + i) = w;
  }
}

// KV = true: dK/dV CTA; false: dQ CTA.  `tile` is the CTA's stationary tile, `slice` the query slice (dQ) or
// batch * kv_heads + kv_head (dK/dV).
template <bool KV>
__device__ __forceinline__ void fa_bwd_f32_body(const BwdF32Params& prm, uint8_t* smem, int slice, int tile) {
  using T = BwdF32Traits;
  using namespace ptx;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::SMEM_BAR);
  uint64_t* x0_full = bars + 0;    // 128 math arrivals
  uint64_t* x1_full = bars + 1;    // 128 math arrivals
  uint64_t* y0_full = bars + 2;    // 128 loader arrivals
  uint64_t* y1_full = bars + 3;    // 128 loader arrivals (with the streamed rows' LSE and delta)
  uint64_t* y0_free = bars + 4;    // MMA commit: acc0 done, Y0 may be rewritten
  uint64_t* y1_free = bars + 5;    // MMA commit: last read of Y1
  uint64_t* t0_full = bars + 6;    // MMA commit
  uint64_t* t1_full = bars + 7;    // MMA commit
  uint64_t* p_full = bars + 8;     // 256 math arrivals: T0 read (and P written, dK/dV)
  uint64_t* ds_full = bars + 9;    // 256 math arrivals: dS written
  uint64_t* row_full = bars + 10;  // 128 loader arrivals: the streamed rows' LSE and delta (dK/dV)
  const uint32_t tmem_base = *reinterpret_cast<uint32_t*>(smem + T::SMEM_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + T::SMEM_MISC + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = prm.S, D = prm.D;
  const int n_tiles = (S + T::BM - 1) / T::BM;
  const int G = KV ? prm.st_kv.group : 1;
  const int kv_heads = prm.st.heads / prm.st_kv.group;
  const int bh0 = KV ? (slice / kv_heads) * prm.st.heads + (slice % kv_heads) * prm.st_kv.group : slice;   // first query slice
  const int j_lo = (KV && prm.causal) ? tile : 0;                     // streamed tiles [j_lo, j_hi) of each query head
  const int j_hi = (!KV && prm.causal) ? tile + 1 : n_tiles;
  const int per_head = j_hi - j_lo;
  const int n_iter = per_head * G;
  const float* x0 = (KV ? prm.k : prm.q) + (KV ? prm.st_kv.slice(bh0) : prm.st.slice(bh0));
  const float* x1 = (KV ? prm.v : prm.d_o) + (KV ? prm.st_kv.slice(bh0) : prm.st.slice(bh0));
  const long long x_row = KV ? prm.st_kv.row : prm.st.row, y_row = KV ? prm.st.row : prm.st_kv.row;

  if (warp >= 8 && warp < 12) {
    // ------------------------------------------------------------ loaders
    // One tile's worth of registers: while the tensor core works on tile n the loaders hold Y1(n+1) until acc1(n) has
    // let go of Y1's planes, then fetch Y0(n+1) under acc0(n) and store it behind it.
    const int t = threadIdx.x - 256;
    float4 r[16];
    float lse2 = -INFINITY, dl = 0.f;   // negated, as the packed operations of the math warps want them
    auto y0_of = [&](int n) { return (KV ? prm.q + prm.st.slice(bh0 + n / per_head) : prm.k + prm.st_kv.slice(bh0)); };
    auto y1_of = [&](int n) { return (KV ? prm.d_o + prm.st.slice(bh0 + n / per_head) : prm.v + prm.st_kv.slice(bh0)); };
    auto tile_of = [&](int n) { return j_lo + n % per_head; };
    auto fetch_rows = [&](int n) {   // LSE and delta of streamed row t; rows past S never contribute (P = 2^-inf)
      const int s = tile_of(n) * T::BM + t;
      lse2 = -INFINITY;
      dl = 0.f;
      if (s < S) {
        const size_t i = static_cast<size_t>(bh0 + n / per_head) * S + s;
        lse2 = prm.lse[i] * -1.4426950408889634f;
        dl = -prm.delta[i];
      }
    };
    auto store_rows = [&](int n) {   // two buffers: read by the math groups of tile n, rewritten for n + 2
      float* rows = reinterpret_cast<float*>(smem + T::SMEM_ROW) + (n & 1) * 128;
      rows[t] = lse2;
      rows[256 + t] = dl;
      mbar_arrive(row_full);
    };
    bool ok = true;
    f32_tile_fetch(y0_of(0), y_row, tile_of(0), S, D, t, r);
    if (KV) {
      fetch_rows(0);
      store_rows(0);
    }
    f32_tile_store(smem + T::SMEM_Y0, t, r);
    mbar_arrive(y0_full);
    f32_tile_fetch(y1_of(0), y_row, tile_of(0), S, D, t, r);
    f32_tile_store(smem + T::SMEM_Y1, t, r);
    mbar_arrive(y1_full);
    for (int n = 1; n < n_iter && ok; ++n) {
      f32_tile_fetch(y1_of(n), y_row, tile_of(n), S, D, t, r);
      if (KV) fetch_rows(n);
      ok = mbar_wait(y1_free, (n - 1) & 1, abort_flag, prm.status, DEV_ERR_TIMEOUT_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      f32_tile_store(smem + T::SMEM_Y1, t, r);
      mbar_arrive(y1_full);
      f32_tile_fetch(y0_of(n), y_row, tile_of(n), S, D, t, r);
      ok = mbar_wait(y0_free, (n - 1) & 1, abort_flag, prm.status, DEV_ERR_TIMEOUT_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (KV) store_rows(n);   // acc0(n-1) is done, so the math groups are through with tile n - 1 and, long before, n - 2
      f32_tile_store(smem + T::SMEM_Y0, t, r);
      mbar_arrive(y0_full);
    }
  } else if (warp == 12) {
    // ------------------------------------------------------------ MMA issuer (one thread)
    if (elect_one()) {
      const int d_steps = (D + 15) >> 4;
      constexpr uint32_t IDESC_T = make_idesc(128, 128, false, false);
      const uint32_t IDESC_ACC = make_idesc(128, d_steps * 16, false, true);
      const uint32_t x0_a = smem_addr(smem + T::SMEM_X0), x1_a = smem_addr(smem + T::SMEM_X1), y0_a = smem_addr(smem + T::SMEM_Y0),
                     y1_a = smem_addr(smem + T::SMEM_Y1);
      // term pairs (a plane, b plane) of order above 2^-24, smallest first: lo hi, mid mid, hi lo, mid hi, hi mid, hi hi
      constexpr int TA[6] = {2, 1, 0, 1, 0, 0};
      constexpr int TB[6] = {0, 1, 2, 0, 1, 0};
      auto issue_t = [&](uint32_t xa, uint32_t ya, uint32_t col) {   // T = X Y^T
#pragma unroll
        for (int term = 0; term < 6; ++term) {
          const uint64_t da = make_sdesc(xa + TA[term] * T::PLANE_BYTES, 16, 1024);
          const uint64_t db = make_sdesc(ya + TB[term] * T::PLANE_BYTES, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < T::DP / 16; ++kk)
            if (kk < d_steps)
              umma_ss(tmem_base + col, sdesc_advance(da, kk * 32), sdesc_advance(db, kk * 32), IDESC_T, (term > 0 || kk > 0) ? 1u : 0u);
        }
      };
      auto issue_acc = [&](uint32_t t_col, uint32_t e_col, uint32_t ya, uint32_t acc) {   // acc = (P or dS) Y
#pragma unroll
        for (int term = 0; term < 6; ++term) {
          const uint64_t db = make_sdesc(ya + TB[term] * T::PLANE_BYTES, T::PLANE_BYTES, 1024);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {   // 16 columns of the streamed tile each: math group kk >> 2
            const uint32_t a = (TA[term] == 2 ? e_col + (kk >> 2) * 32 : t_col + (kk >> 2) * 64 + TA[term] * 32) + (kk & 3) * 8;
            umma_ts(tmem_base + acc, tmem_base + a, sdesc_advance(db, kk * 2048), IDESC_ACC, (term > 0 || kk > 0) ? 1u : 0u);
          }
        }
      };
      bool ok = mbar_wait(x0_full, 0, abort_flag, prm.status, DEV_ERR_TIMEOUT_LOAD);
      for (int n = 0; n < n_iter && ok; ++n) {
        const uint32_t par = n & 1;
        ok = mbar_wait(y0_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_LOAD);
        if (!ok) break;
        tc_fence_after();
        issue_t(x0_a, y0_a, T::COL_T0);
        umma_commit(t0_full);
        if (n == 0) ok = mbar_wait(x1_full, 0, abort_flag, prm.status, DEV_ERR_TIMEOUT_LOAD);
        if (ok) ok = mbar_wait(y1_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_LOAD);
        if (!ok) break;
        tc_fence_after();
        issue_t(x1_a, y1_a, T::COL_T1);
        umma_commit(t1_full);
        if (!KV) umma_commit(y1_free);
        ok = mbar_wait(p_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_SOFTMAX);
        if (!ok) break;
        if (KV) {
          tc_fence_after();
          issue_acc(T::COL_T0, T::COL_E0, y1_a, T::COL_ACC1);
          umma_commit(y1_free);
        }
        ok = mbar_wait(ds_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_SOFTMAX);
        if (!ok) break;
        tc_fence_after();
        issue_acc(T::COL_T1, T::COL_E1, y0_a, T::COL_ACC0);
        umma_commit(y0_free);
      }
    }
  } else {
    // ------------------------------------------------------------ math (warps 0-7)
    const int g = warp >> 2;                    // which 64 of the 128 columns
    const int lane_base = (warp & 3) * 32;
    const int row = lane_base + lane;           // row of the stationary tile
    const int x_idx = tile * T::BM + row;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(lane_base) << 16);
    const float sl2 = prm.scale_log2;
    {
      float4 x[16];
      f32_tile_fetch(g ? x1 : x0, x_row, tile, S, D, threadIdx.x & 127, x);
      f32_tile_store(smem + (g ? T::SMEM_X1 : T::SMEM_X0), threadIdx.x & 127, x);
      mbar_arrive(g ? x1_full : x0_full);
    }
    float row_lse2 = -INFINITY, row_dl = 0.f;    // dQ: this thread's query row, negated
    if (!KV && x_idx < S) {
      row_lse2 = prm.lse[static_cast<size_t>(bh0) * S + x_idx] * -1.4426950408889634f;
      row_dl = -prm.delta[static_cast<size_t>(bh0) * S + x_idx];
    }
    bool ok = true;
    uint32_t p[64];   // this thread's T0, then P, then dS (fp32 bits)
    // the three planes of 64 values: 32 columns each of packed bf16
    auto put_planes = [&](uint32_t t_col, uint32_t e_col) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], mi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          split3_bf16x2(__uint_as_float(p[c * 32 + 2 * i]), __uint_as_float(p[c * 32 + 2 * i + 1]), &hi[i], &mi[i], &lo[i]);
        tmem_st_x16(t_lane + t_col + g * 64 + c * 16, hi);
        tmem_st_x16(t_lane + t_col + g * 64 + 32 + c * 16, mi);
        tmem_st_x16(t_lane + e_col + g * 32 + c * 16, lo);
      }
      tmem_wait_st();
    };
    // The tile's accumulators into the output rows (group 0 its row of dK, group 1 of dV; dQ: a half of the row each), which
    // hold the sum of the tiles before; with the last tile's go scale and rotation.  The tensor core truncates when it adds
    // into fp32, so a sum left in tensor memory over all tiles drifts with their number: dK of 1024 rows was 7.0e-6 off 64
    // bits (the CUDA-core kernel 1.3e-6); added up here, rounding to nearest, it is 0.8e-6 at any length.  Runs while Y0 is
    // replaced and the next T0 computed.
    auto drain = [&](int n, bool last) -> bool {
      constexpr int NC = KV ? 2 : 1;
      float* out = KV ? (g ? prm.dv : prm.dk) + prm.st_kv.slice(bh0) + static_cast<long long>(x_idx) * prm.st_kv.row
                      : prm.dq + prm.st.slice(bh0) + static_cast<long long>(x_idx) * prm.st.row + g * 32;
      const int width = KV ? D : D - g * 32;   // columns of this thread's part (may be <= 0)
      float4 prev[NC * 8];
#pragma unroll
      for (int i = 0; i < NC * 8; ++i) {
        prev[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n > 0 && x_idx < S && 4 * i < width) prev[i] = reinterpret_cast<const float4*>(out)[i];
      }
      float z = 0.f;   // NaN: the row is not finite
      bool got = mbar_wait(y0_free, n & 1, abort_flag, prm.status, DEV_ERR_TIMEOUT_MMA);   // the tile's MMAs are complete
      got = __all_sync(0xffffffffu, got);
      if (!got) return false;
      tc_fence_after();
      const float f = !last || (KV && g) ? 1.0f : prm.scale;
      const bool rotate = last && prm.rope_table != nullptr && !(KV && g);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        uint32_t a[32];
        tmem_ld_x32(t_lane + ((KV && g) ? T::COL_ACC1 : T::COL_ACC0) + (KV ? c * 32 : g * 32), a);
        tmem_wait_ld();
        if (x_idx < S) {
          const float2* tab = prm.rope_table + static_cast<size_t>(x_idx) * (D >> 1) + (KV ? c * 16 : g * 16);
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            if (c * 32 + i >= width) break;
            const float4 pv = prev[c * 8 + (i >> 2)];
            float4 w = make_float4((__uint_as_float(a[i]) + pv.x) * f, (__uint_as_float(a[i + 1]) + pv.y) * f,
                                   (__uint_as_float(a[i + 2]) + pv.z) * f, (__uint_as_float(a[i + 3]) + pv.w) * f);
            if (rotate) w = rotate_back(w, *reinterpret_cast<const float4*>(tab + (i >> 1)));   // (cos, sin) of two pairs
            if (last) z = nonfinite(nonfinite(nonfinite(nonfinite(z, w.x), w.y), w.z), w.w);
            *reinterpret_cast<float4*>(out + c * 32 + i) = w;
          }
        }
      }
      if (last && z != 0.f) fa_bwd_f32_visible<KV>(prm, bh0, x_idx, KV && g, KV ? 0 : g * 32, KV ? D : min(32, width), out);
      return true;
    };
    for (int n = 0; n < n_iter; ++n) {
      if (n > 0 && !(ok = drain(n - 1, false))) break;
      const uint32_t par = n & 1;
      const int jt = j_lo + n % per_head;
      const float* rows = reinterpret_cast<const float*>(smem + T::SMEM_ROW) + (n & 1) * 128 + g * 64;
      if (KV) ok = mbar_wait(row_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_LOAD);
      if (ok) ok = mbar_wait(t0_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_MMA);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      tmem_ld_x32(t_lane + T::COL_T0 + g * 64, *reinterpret_cast<uint32_t(*)[32]>(&p[0]));
      tmem_ld_x32(t_lane + T::COL_T0 + g * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&p[32]));
      tmem_wait_ld();
      // column i of this thread is streamed row jt * 128 + g * 64 + i
      const int c0 = jt * T::BM + g * 64;
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        float4 l4 = make_float4(row_lse2, row_lse2, row_lse2, row_lse2);
        if (KV) l4 = *reinterpret_cast<const float4*>(rows + i);
        const float2 x01 = fma2(bits2(p[i + 0], p[i + 1]), make_float2(sl2, sl2), make_float2(l4.x, l4.y));
        const float2 x23 = fma2(bits2(p[i + 2], p[i + 3]), make_float2(sl2, sl2), make_float2(l4.z, l4.w));
        p[i + 0] = __float_as_uint(ex2(x01.x));
        p[i + 1] = __float_as_uint(ex2(x01.y));
        p[i + 2] = __float_as_uint(ex2(x23.x));
        p[i + 3] = __float_as_uint(ex2(x23.y));
      }
      if (prm.causal && jt == tile) {   // the diagonal tile: keys after the query are masked
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (KV ? (x_idx > c0 + i) : (c0 + i > x_idx)) p[i] = 0u;
      }
      if (!KV && (jt + 1) * T::BM > S) {   // keys past the sequence (queries past it have P = 2^-inf)
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (c0 + i >= S) p[i] = 0u;
      }
      if (KV) put_planes(T::COL_T0, T::COL_E0);
      tc_fence_before();
      mbar_arrive(p_full);
      ok = mbar_wait(t1_full, par, abort_flag, prm.status, DEV_ERR_TIMEOUT_MMA);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[32];
        tmem_ld_x32(t_lane + T::COL_T1 + g * 64 + c * 32, d);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float4 d4 = make_float4(row_dl, row_dl, row_dl, row_dl);
          if (KV) d4 = *reinterpret_cast<const float4*>(rows + 256 + c * 32 + i);
          uint32_t* pp = &p[c * 32 + i];
          const float2 s01 = mul2(bits2(pp[0], pp[1]), add2(bits2(d[i + 0], d[i + 1]), make_float2(d4.x, d4.y)));
          const float2 s23 = mul2(bits2(pp[2], pp[3]), add2(bits2(d[i + 2], d[i + 3]), make_float2(d4.z, d4.w)));
          pp[0] = __float_as_uint(s01.x);
          pp[1] = __float_as_uint(s01.y);
          pp[2] = __float_as_uint(s23.x);
          pp[3] = __float_as_uint(s23.y);
        }
      }
      put_planes(T::COL_T1, T::COL_E1);
      tc_fence_before();
      mbar_arrive(ds_full);
    }
    if (ok) drain(n_iter - 1, true);
  }
}

// Grid: for each rank (0 = most streamed tiles under the causal mask) the dK/dV CTAs of every K/V slice, then the dQ CTAs
// of every query slice: the longest CTAs start first.
__global__ void __launch_bounds__(416, 1) fa_bwd_f32_sm100_kernel(const __grid_constant__ BwdF32Params prm) {
  using T = BwdF32Traits;
  using namespace ptx;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::SMEM_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + T::SMEM_MISC + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + T::SMEM_MISC);
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    if (smem_addr(smem) & 1023u) {
      *abort_flag = 1;
      atomicCAS(prm.status, 0, DEV_ERR_SMEM_ALIGN);
    }
    if (*reinterpret_cast<volatile int*>(prm.status) != 0) *abort_flag = 1;
    const uint32_t counts[T::NUM_BARS] = {128, 128, 128, 128, 1, 1, 1, 1, 256, 256, 128};
    for (int i = 0; i < T::NUM_BARS; ++i) mbar_init(&bars[i], counts[i]);
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 12) {
    tmem_alloc(tmem_slot, T::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dep_wait();   // O, LSE and dO may come from the kernels in front, delta from the prepare pass
  grid_dep_launch();
  if (*abort_flag == 0) {
    const int n_kv = prm.BH / prm.st_kv.group;
    const int rank = static_cast<int>(blockIdx.x) / (n_kv + prm.BH), i = static_cast<int>(blockIdx.x) % (n_kv + prm.BH);
    if (i < n_kv)
      fa_bwd_f32_body<true>(prm, smem, i, rank);
    else
      fa_bwd_f32_body<false>(prm, smem, i - n_kv, (prm.S + T::BM - 1) / T::BM - 1 - rank);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    if (*abort_flag)
      for (int i = 0; i < 50; ++i) __nanosleep(20000);
    tc_fence_after();
    tmem_dealloc(*tmem_slot, T::TMEM_COLS);
  }
}

}  // namespace it

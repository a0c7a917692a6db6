"""GPU parity at the edges of what each kernel is dispatched for: head dims that the tensor-core tiles are padded for,
sequences shorter than a tile, remainders of tiles.  Same oracle and bounds as test_gpu_attention.py."""
import math

import numpy as np
import pytest

import gpu_util as gu
import oracle_lib as ol
from irontensor_b200 import _lib, synth
from test_gpu_attention import BF16_REL_L2, seeded

pytestmark = pytest.mark.gpu


def check_bf16(got, want, name, rel_scale=1.0):
    """The bounds of test_gpu_attention.check_bf16, with one difference: an element may be off by 2e-2 (what the kernels add)
    plus 2^-9 of its own magnitude, which is what storing it as bf16 costs.  The fixed 2e-2 of that file holds for values
    below about 4; the gradients of the first causal rows, which few keys share, are larger at head dims near 96."""
    kind = name.split()[-1]
    assert not np.isnan(got).any(), f"{name}: NaN in output"
    over = np.abs(got.astype(np.float64) - want) - (2e-2 + 2.0 ** -9 * np.abs(want))
    assert over.max() <= 0, f"{name}: max-abs bound exceeded by {over.max():.2e}"
    rel = gu.err_stats(got, want)[1]
    assert rel <= BF16_REL_L2[kind] * rel_scale, f"{name}: rel-L2 {rel:.3e} > {BF16_REL_L2[kind] * rel_scale:.2e}"


# H is chosen so that a tensor has at least 4000 elements: the relative-L2 bounds of check_bf16 lie 10 % above the worst
# figure of large tensors, and the relative error of an L2 norm estimated from N values is 1 / sqrt(2 N) = 1.1 %.
@pytest.mark.parametrize("S,H,D,causal", [
    (2, 256, 8, True), (31, 16, 16, True), (64, 160, 16, True), (50, 150, 16, False), (65, 8, 40, False), (127, 8, 64, True), (127, 4, 128, False),   # shorter than a tile
    (128, 4, 32, True), (129, 4, 8, True), (300, 3, 24, True), (257, 2, 56, False),                        # padded to 64 columns
    (130, 4, 72, True), (300, 3, 80, False), (1003, 2, 96, True), (256, 2, 120, True), (385, 2, 104, False),   # padded to 128
])
def test_bf16_any_head_dim_and_length(it_ctx, S, H, D, causal):
    q, k, v, d_o = seeded(900 + S + D, 1, H, S, D, bf16=True)
    o, lse, dq, dk, dv = gu.run_fwd_bwd(it_ctx, q, k, v, d_o, causal, bf16=True)
    ro, rlse = ol.fwd(q, k, v, causal)
    rdq, rdk, rdv = ol.bwd(q, k, v, d_o, causal)
    assert np.abs(lse - rlse).max() <= 1e-4
    # Two keys: dQ = dS_0 (K_0 - K_1) with dS_0 = p (1 - p) (dP_0 - dP_1), and an error e of delta = dO . O (O is stored as bf16)
    # moves dQ by e (p K_0 + (1 - p) K_1).  At D = 8: e = sqrt(8) * 0.7 * 1.6e-3, |p K_0 + (1 - p) K_1| about half of |K_0 - K_1|,
    # p (1 - p) (dP_0 - dP_1) about 0.2 * 4: 2e-3 of dQ (dK alike) on top of the bound's own 3.4e-3, and sums of two terms
    # average nothing out: 1.5 times the bound.
    rel_scale = 1.5 if S == 2 else 1.0
    for got, want, name in ((o, ro, "O"), (dq, rdq, "dQ"), (dk, rdk, "dK"), (dv, rdv, "dV")):
        check_bf16(got, want, f"{(S, H, D)} causal={causal} {name}", rel_scale)


def test_bf16_one_key(it_ctx):
    """One key: the softmax is exactly 1, so O = V and dV = dO bit for bit; dS is a difference of two equal sums."""
    q, k, v, d_o = seeded(77, 2, 3, 1, 96, bf16=True)
    o, lse, dq, dk, dv = gu.run_fwd_bwd(it_ctx, q, k, v, d_o, True, bf16=True)
    assert np.array_equal(o, v) and np.array_equal(dv, d_o)
    assert np.abs(dq).max() <= 1e-4 and np.abs(dk).max() <= 1e-4


@pytest.mark.parametrize("B,S,H,Hkv,D,rope", [(2, 100, 8, 2, 96, True), (1, 333, 4, 1, 80, True), (2, 260, 6, 3, 32, False)])
def test_bf16_grouped_heads_at_padded_head_dims(it_ctx, B, S, H, Hkv, D, rope):
    from irontensor_b200 import Tensor, attention_gqa, attention_gqa_backward
    q, _, _, d_o = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(910 + D, B, H, S, D, bf16=True)]
    _, k, v, _ = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(911 + D, B, Hkv, S, D, bf16=True)]
    tq, tk, tv, tdo = (Tensor.from_f32_as_bf16(t.reshape(-1), list(t.shape)) for t in (q, k, v, d_o))
    o = attention_gqa(tq, tk, tv, True)
    dq, dk, dv = attention_gqa_backward(tdo, tq, tk, tv, o, True, rope_base=10000.0 if rope else None, position_offset=5)
    assert it_ctx.poll_status() == 0
    ro, rlse = ol.gqa_fwd(q, k, v, True)
    rdq, rdk, rdv = ol.gqa_bwd(q, k, v, d_o, True)
    if rope:
        rdq, rdk = ol.rope(rdq, 10000.0, 5, inverse=True), ol.rope(rdk, 10000.0, 5, inverse=True)
    assert np.abs(o.lse.to_f32_host() - rlse).max() <= 1e-4
    for got, want, name in ((o, ro, "O"), (dq, rdq, "dQ"), (dk, rdk, "dK"), (dv, rdv, "dV")):
        scale = math.sqrt(H // Hkv) if name in ("dK", "dV") else 1.0   # sums over the group's heads
        check_bf16(got.to_f32_host() / scale, want / scale, f"{(B, S, H, Hkv, D)} {name}")


def test_noalloc_backward_of_a_padded_shape_beyond_the_scratch(it_ctx):
    """A padded shape whose dQ accumulator exceeds the built-in scratch still runs without one (CUDA-core kernels)."""
    import torch
    B, H, S, D = 2, 33, 1024, 32
    assert B * H * S * D * 4 > _lib.IT_NOALLOC_SCRATCH_BYTES
    q, k, v, d_o = [gu.to_dev(t.reshape(B, H, S, D), True) for t in synth.attention_inputs(78, B, H, S, D, bf16=True)]
    from irontensor_b200 import raw
    o, lse = torch.empty_like(q), torch.empty((B, H, S), dtype=torch.float32, device="cuda")
    raw.fwd(_lib.IT_BF16, B, H, S, D, True, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), ctx=it_ctx)
    g = [torch.full_like(q, float("nan")) for _ in range(3)]
    _lib.check(it_ctx.lib.it_flash_attention_bwd_noalloc(
        it_ctx.handle, it_ctx.stream(), _lib.IT_BF16, B, H, S, D, 1, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
        d_o.data_ptr(), lse.data_ptr(), g[0].data_ptr(), g[1].data_ptr(), g[2].data_ptr()))
    assert it_ctx.poll_status() == 0
    sl = (slice(1, 2), slice(32, 33))
    want = ol.bwd(*[gu.to_host(t[sl].contiguous()) for t in (q, k, v, d_o)], True)
    for got, w, name in zip(g, want, ("dQ", "dK", "dV")):
        check_bf16(gu.to_host(got[sl].contiguous()), w, name)


@pytest.mark.parametrize("B,S,H,Hkv,D,causal,rope", [
    (2, 32, 4, 4, 64, True, False), (1, 33, 3, 3, 20, False, False), (1, 127, 2, 2, 64, True, True), (2, 128, 4, 2, 32, True, False),
    (1, 129, 4, 4, 64, False, True), (1, 257, 6, 2, 60, True, True), (1, 400, 2, 1, 4, False, False), (1, 640, 4, 4, 64, True, False),
])
def test_fp32_backward_on_the_tensor_cores(it_ctx, B, S, H, Hkv, D, causal, rope):
    """The split-operand fp32 backward at the edges of its tiles.  Tolerance: the path's 1e-4; the operands carry 24 bits and
    the sums are fp32, so the error is that of fp32 sums of a few hundred terms of order one (1e-6 to 1e-5)."""
    from irontensor_b200 import Tensor, attention_gqa, attention_gqa_backward
    q, _, _, d_o = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(940 + S, B, H, S, D)]
    _, k, v, _ = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(941 + S, B, Hkv, S, D)]
    tq, tk, tv, tdo = (Tensor.from_f32_slice(t.reshape(-1), list(t.shape)) for t in (q, k, v, d_o))
    o = attention_gqa(tq, tk, tv, causal)
    dq, dk, dv = attention_gqa_backward(tdo, tq, tk, tv, o, causal, rope_base=10000.0 if rope else None, position_offset=7)
    assert it_ctx.poll_status() == 0
    rdq, rdk, rdv = ol.gqa_bwd(q, k, v, d_o, causal)
    if rope:
        rdq, rdk = ol.rope(rdq, 10000.0, 7, inverse=True), ol.rope(rdk, 10000.0, 7, inverse=True)
    for got, want, name in ((dq, rdq, "dQ"), (dk, rdk, "dK"), (dv, rdv, "dV")):
        g = got.to_f32_host()
        assert not np.isnan(g).any()
        assert np.abs(g - want).max() <= 1e-4, f"{name}: {np.abs(g - want).max():.2e}"
        assert np.linalg.norm(g - want) <= 1e-5 * np.linalg.norm(want), name


# The skinny kernel's token groups of 8, its 16-row tiles and 32-wide K steps, and the three tile widths of the tcgen05 GEMM
# (chosen by how many tiles the product has), each with remainders in every dimension.
@pytest.mark.parametrize("n,k,out", [(1, 8, 8), (3, 40, 24), (8, 264, 120), (9, 2048, 200), (16, 72, 1000), (17, 520, 40), (32, 2048, 3064),
                                     (33, 136, 200), (64, 4104, 520), (130, 264, 9480), (700, 200, 5000), (2500, 136, 3080)])
def test_projection_of_any_number_of_tokens(it_ctx, n, k, out):
    """linear_forward against an fp32 product of the same bf16 operands: error of the bf16 result, 2^-9 / sqrt(3) relative per
    element plus fp32 sums (1.7e-3 in L2)."""
    from irontensor_b200 import Tensor, linear_forward
    x = synth.round_bf16(synth.normal(180, synth.TENSOR_Q, 0, n * k, 1.0)).reshape(n, k)
    w = synth.round_bf16(synth.normal(181, synth.TENSOR_K, 0, out * k, k ** -0.5)).reshape(out, k)
    y = linear_forward(Tensor.from_f32_as_bf16(x.reshape(-1), [n, k]), Tensor.from_f32_as_bf16(w.reshape(-1), [out, k]))
    assert it_ctx.poll_status() == 0
    want = x.astype(np.float64) @ w.astype(np.float64).T
    got = y.to_f32_host()
    assert np.linalg.norm(got - want) <= 2.0e-3 * np.linalg.norm(want)
    assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-4)


@pytest.mark.parametrize("B,S,hidden,H,Hkv,D,base,packed", [(4, 1, 256, 4, 2, 64, 10000.0, False), (1, 20, 512, 8, 8, 128, 10000.0, True),
                                                            (3, 5, 72, 2, 1, 96, 500.0, False), (9, 1, 128, 4, 1, 32, None, True)])
def test_qkv_projection_of_a_few_tokens(it_ctx, B, S, hidden, H, Hkv, D, base, packed):
    """The skinny kernel's Q/K/V epilogue (rotation evaluated in place, separate and packed outputs)."""
    from irontensor_b200 import Tensor, qkv_rope_forward
    n, width, pos = B * S, (H + 2 * Hkv) * D, 11
    x = synth.round_bf16(synth.normal(190, synth.TENSOR_Q, 0, n * hidden, 1.0)).reshape(n, hidden)
    w = synth.round_bf16(synth.normal(191, synth.TENSOR_K, 0, width * hidden, hidden ** -0.5)).reshape(width, hidden)
    out = qkv_rope_forward(Tensor.from_f32_as_bf16(x.reshape(-1), [B, S, hidden]), Tensor.from_f32_as_bf16(w.reshape(-1), [width, hidden]),
                           H, Hkv, D, base, pos, packed=packed)
    assert it_ctx.poll_status() == 0
    y = (x.astype(np.float64) @ w.astype(np.float64).T).astype(np.float32).reshape(B, S, width)
    q, k, v = y[..., :H * D].reshape(B, S, H, D), y[..., H * D:(H + Hkv) * D].reshape(B, S, Hkv, D), y[..., (H + Hkv) * D:].reshape(B, S, Hkv, D)
    if base is not None:
        q, k = ol.rope(np.ascontiguousarray(q), base, pos), ol.rope(np.ascontiguousarray(k), base, pos)
    if packed:
        got = out.to_f32_host()
        got = (got[..., :H * D].reshape(q.shape), got[..., H * D:(H + Hkv) * D].reshape(k.shape), got[..., (H + Hkv) * D:].reshape(v.shape))
    else:
        got = [t.to_f32_host() for t in out]
    for g, want in zip(got, (q, k, v)):
        # a bf16 rounding step of the result, and sines and products in fp32
        assert np.all(np.abs(g - want) <= 2.0 ** -8 * np.abs(want) + 1e-4)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,H,Hkv,D,kv_len,max_len", [
    (1, 4, 4, 64, 1, 1), (1, 1, 1, 8, 2, 5), (2, 4, 4, 64, 65, 128), (1, 8, 4, 40, 129, 129), (3, 6, 2, 96, 33, 64),   # one split
    (1, 4, 2, 128, 300, 512), (2, 8, 2, 64, 1111, 2000), (1, 5, 1, 128, 700, 701), (1, 9, 1, 64, 150, 150),            # clusters of 2 to 8
    (1, 4, 4, 64, 16500, 16500), (4, 16, 4, 128, 1000, 1024), (1, 32, 4, 128, 9000, 9000), (48, 8, 4, 128, 520, 600),  # merge launch, tensor cores
])
def test_decode_over_its_ranges(it_ctx, B, H, Hkv, D, kv_len, max_len, bf16):
    """Splits of one, clusters merging through distributed shared memory, merge launches; every head grouping.  Bounds: fp32
    sums of up to 16500 terms (1e-6 relative each way, 1e-5 in L2); bf16 the output's rounding and P's (2.5e-3, as O elsewhere)."""
    from irontensor_b200 import Tensor, attention_decode
    f = synth.round_bf16 if bf16 else (lambda a: a)
    q = f(synth.normal(200 + kv_len, synth.TENSOR_Q, 0, B * H * D)).reshape(B, H, D)
    k = f(synth.normal(200 + kv_len, synth.TENSOR_K, 0, B * max_len * Hkv * D)).reshape(B, max_len, Hkv, D)
    v = f(synth.normal(200 + kv_len, synth.TENSOR_V, 0, B * max_len * Hkv * D)).reshape(B, max_len, Hkv, D)
    mk = Tensor.from_f32_as_bf16 if bf16 else Tensor.from_f32_slice
    o = attention_decode(*(mk(t.reshape(-1), list(t.shape)) for t in (q, k, v)), kv_len)
    assert it_ctx.poll_status() == 0
    kk, vv = (t[:, :kv_len].astype(np.float64).repeat(H // Hkv, axis=2) for t in (k, v))
    s = np.einsum("bhd,blhd->bhl", q.astype(np.float64), kk) / math.sqrt(D)
    mx = s.max(-1, keepdims=True)
    p = np.exp(s - mx)
    want = np.einsum("bhl,blhd->bhd", p, vv) / p.sum(-1)[..., None]
    lse = (mx[..., 0] + np.log(p.sum(-1)))
    got = o.to_f32_host()
    assert np.abs(o.lse.to_f32_host() - lse).max() <= 1e-4
    assert np.linalg.norm(got - want) <= (2.5e-3 if bf16 else 1e-5) * np.linalg.norm(want)


@pytest.mark.parametrize("S,D", [(640, 64), (1024, 64), (777, 32)])
def test_fp32_backward_keeps_its_precision_over_many_tiles(it_ctx, S, D):
    """Gradients of long sequences against 64 bits.  fp32 sums of S terms, rounded to nearest, are off by about
    sqrt(S) * 2^-25 relative to the terms (1e-6 at 1024), the operands' 24 bits by less: 2e-6.  (Sums that stay in tensor memory
    over all tiles are truncated at every addition and drift to 7e-6.)"""
    import torch
    q, k, v, d_o = [torch.from_numpy(t.reshape(1, 2, S, D)).cuda() for t in synth.attention_inputs(960 + S, 1, 2, S, D)]
    from irontensor_b200 import Tensor, attention_backward_recompute, flash_attention
    from irontensor_b200 import Precision
    tq, tk, tv, tdo = (Tensor(t.reshape(-1), [1, 2, S, D], Precision.FP32) for t in (q, k, v, d_o))
    o = flash_attention(tq, tk, tv, True)
    got = attention_backward_recompute(tdo, tq, tk, tv, o, o.lse)
    q, k, v, d_o = (t.double() for t in (q, k, v, d_o))
    s = (q @ k.mT / math.sqrt(D)).masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), -math.inf)
    p = torch.softmax(s, -1)
    ds = p * (d_o @ v.mT - (d_o * (p @ v)).sum(-1, keepdim=True))
    want = (ds @ k / math.sqrt(D), ds.mT @ q / math.sqrt(D), p.mT @ d_o)
    for g, w, name in zip(got, want, ("dQ", "dK", "dV")):
        assert (g.torch().reshape(w.shape).double() - w).norm() <= 2e-6 * w.norm(), name


def test_out_of_memory_keeps_its_type(it_ctx):
    """An allocation that cannot succeed raises what torch raises for it, and the context stays usable."""
    import torch
    from irontensor_b200 import Precision, Tensor, flash_attention
    t = Tensor(torch.zeros(8 * 4 * 64 * 64, device="cuda"), [8, 4, 64, 64], Precision.FP32)
    keep = []
    torch.cuda.empty_cache()
    torch.cuda.memory.set_per_process_memory_fraction(1e-9)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(1000):   # until the allocator's cached blocks are used up
                keep.append(flash_attention(t, t, t, True))
    finally:
        torch.cuda.memory.set_per_process_memory_fraction(1.0)
    assert np.isfinite(flash_attention(t, t, t, True).to_f32_host()).all()


# pairs of CTAs on a tile of 256 x 256: remainders of rows (a whole CTA's rows missing), columns and K, several tiles per pair
@pytest.mark.parametrize("n,k,out", [(33, 72, 264), (130, 136, 200), (300, 264, 520), (257, 64, 256), (5000, 520, 5000)])
def test_projection_on_pairs_of_ctas(it_ctx, monkeypatch, n, k, out):
    """All three transposition cases, 1.7e-3 in L2 (2^-9 / sqrt(3) per bf16 element) for y and dx, fp32 sums for dW."""
    import torch
    from irontensor_b200 import Precision, Tensor, linear_backward, linear_forward
    monkeypatch.setenv("IT_GEMM_TILE", "512")
    gen = torch.Generator(device="cuda").manual_seed(7)
    x, w, dy = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((n, k), (out, k), (n, out)))
    tx, tw, tdy = (Tensor(t.reshape(-1), list(t.shape), Precision.BF16) for t in (x, w, dy))
    y, (dx, dw) = linear_forward(tx, tw), linear_backward(tdy, tx, tw)
    assert it_ctx.poll_status() == 0
    x, w, dy = x.double(), w.double(), dy.double()
    for got, want, bound in ((y, x @ w.T, 2e-3), (dx, dy @ w, 2e-3), (dw, dy.T @ x, 1e-5)):
        assert (got.torch().reshape(want.shape).double() - want).norm() <= bound * want.norm()


@pytest.mark.parametrize("D,kernel", [(64, "pp"), (128, "pp"), (64, "two"), (128, "two")])
@pytest.mark.parametrize("S,causal", [(128, True), (129, False), (300, True), (520, False)])
def test_bf16_forward_kernels_at_short_lengths(it_ctx, monkeypatch, D, kernel, S, causal):
    """Either forward kernel may get any full-width launch, by how it fills the GPU: both, from one key tile on."""
    monkeypatch.setenv("IT_FWD_KERNEL", kernel)
    H = 6
    q, k, v, d_o = seeded(970 + S + D, 1, H, S, D, bf16=True)
    o, lse, _, _, _ = gu.run_fwd_bwd(it_ctx, q, k, v, d_o, causal, bf16=True)
    ro, rlse = ol.fwd(q, k, v, causal)
    assert np.abs(lse - rlse).max() <= 1e-4
    check_bf16(o, ro, f"{(S, D, kernel)} O")


# rows of whole 16-byte chunks and others, one position per CTA and several with a remainder, heads of Q and K apart and alike
@pytest.mark.parametrize("B,S,H,Hkv,D,bf16", [(1, 1, 3, 1, 8, True), (2, 1003, 4, 2, 96, True), (3, 700, 2, 2, 128, True), (1, 2500, 1, 1, 4, False),
                                              (2, 333, 3, 1, 64, False), (1, 77, 2, 1, 20, True), (1, 50, 2, 2, 6, False)])
@pytest.mark.parametrize("inverse", [False, True])
def test_rope_of_any_row_width(it_ctx, B, S, H, Hkv, D, bf16, inverse):
    from irontensor_b200 import Tensor, rope_qk
    q, k = (synth.normal(995, t, 0, B * S * h * D, 1.0).reshape(B, S, h, D) for t, h in ((synth.TENSOR_Q, H), (synth.TENSOR_K, Hkv)))
    if bf16:
        q, k = synth.round_bf16(q), synth.round_bf16(k)
    make = Tensor.from_f32_as_bf16 if bf16 else Tensor.from_f32_slice
    got = rope_qk(make(q.reshape(-1), list(q.shape)), make(k.reshape(-1), list(k.shape)), 10000.0, 11, inverse=inverse)
    for g, x in zip(got, (q, k)):
        want = ol.rope(x, 10000.0, 11, inverse=inverse)
        assert np.abs(g.to_f32_host() - want).max() <= (2.0 ** -8 * np.abs(want).max() if bf16 else 1e-5)


@pytest.mark.parametrize("split", ["2", "4"])
@pytest.mark.parametrize("B,S,H,Hkv,D,causal,rope", [
    (1, 100, 4, 1, 64, True, False),     # one query tile per head: parts of one iteration
    (2, 128, 2, 2, 128, True, True),     # one iteration in all: parts without any
    (1, 300, 6, 2, 128, False, True), (2, 385, 4, 1, 64, True, True), (1, 640, 8, 2, 96, True, True), (1, 257, 3, 3, 40, True, False),
])
def test_bf16_backward_split_over_a_cluster(it_ctx, monkeypatch, split, B, S, H, Hkv, D, causal, rope):
    from irontensor_b200 import Tensor, attention_gqa, attention_gqa_backward
    q, _, _, d_o = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(980 + S, B, H, S, D, bf16=True)]
    _, k, v, _ = [np.ascontiguousarray(t.transpose(0, 2, 1, 3)) for t in seeded(981 + S, B, Hkv, S, D, bf16=True)]
    tq, tk, tv, tdo = (Tensor.from_f32_as_bf16(t.reshape(-1), list(t.shape)) for t in (q, k, v, d_o))
    o = attention_gqa(tq, tk, tv, causal)
    monkeypatch.setenv("IT_BWD_SPLIT", split)
    monkeypatch.setenv("IT_BWD_KEY_TILES", "1")
    dq, dk, dv = attention_gqa_backward(tdo, tq, tk, tv, o, causal, rope_base=10000.0 if rope else None, position_offset=3)
    assert it_ctx.poll_status() == 0
    rdq, rdk, rdv = ol.gqa_bwd(q, k, v, d_o, causal)
    if rope:
        rdq, rdk = ol.rope(rdq, 10000.0, 3, inverse=True), ol.rope(rdk, 10000.0, 3, inverse=True)
    for got, want, name in ((dq, rdq, "dQ"), (dk, rdk, "dK"), (dv, rdv, "dV")):
        scale = math.sqrt(H // Hkv) if name in ("dK", "dV") else 1.0   # sums over the group's heads
        check_bf16(got.to_f32_host() / scale, want / scale, f"{(B, S, H, Hkv, D)} {name}")


@pytest.mark.parametrize("S,D", [(100, 64), (127, 128), (300, 96), (200, 32), (260, 40)])
def test_bf16_padded_shapes_round_their_results_only(it_ctx, S, D):
    """Shapes of the padded tiles, whose P and dS are two bf16 terms, against 64 bits.  Rounding a result to bf16 costs 1.66e-3 of its norm (2^-9 of each element,
    uniform over the binades); delta, computed from the rounded O, adds to dQ and dK (1.9e-3 in all).  One bf16 term for P and
    dS would add as much again (2.0e-3, 2.3e-3 and 3.0e-3)."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_backward_recompute, flash_attention
    q, k, v, d_o = [torch.from_numpy(t.reshape(2, 8, S, D)).cuda() for t in synth.attention_inputs(990 + S, 2, 8, S, D, bf16=True)]
    tq, tk, tv, tdo = (Tensor(t.to(torch.bfloat16).reshape(-1), [2, 8, S, D], Precision.BF16) for t in (q, k, v, d_o))
    o = flash_attention(tq, tk, tv, True)
    got = (o,) + tuple(attention_backward_recompute(tdo, tq, tk, tv, o, o.lse))
    q, k, v, d_o = (t.double() for t in (q, k, v, d_o))
    s = (q @ k.mT / math.sqrt(D)).masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), -math.inf)
    p = torch.softmax(s, -1)
    ds = p * (d_o @ v.mT - (d_o * (p @ v)).sum(-1, keepdim=True))
    want = (p @ v, ds @ k / math.sqrt(D), ds.mT @ q / math.sqrt(D), p.mT @ d_o)
    for g, w, name, bound in zip(got, want, ("O", "dQ", "dK", "dV"), (1.75e-3, 2.1e-3, 2.1e-3, 1.75e-3)):
        err = ((g.torch().reshape(w.shape).double() - w).norm() / w.norm()).item()
        assert err <= bound, f"{name}: {err:.2e}"


def test_packed_layout_refuses_other_shapes(it_ctx):
    from irontensor_b200 import Tensor, attention_packed
    for S, D in ((100, 64), (200, 96)):
        with pytest.raises(_lib.ITError, match="head_dim 64 or 128 and seq >= 128"):
            attention_packed(Tensor.from_f32_as_bf16(np.zeros(S * 6 * D, np.float32), [1, S, 6 * D]), 2, 2, D, True)


def test_captured_forwards_replay_on_any_stream(it_ctx):
    """Two graphs captured through one stream, replayed side by side on two others and beside eager launches: a captured launch
    has a work-item counter of its own."""
    import torch
    from irontensor_b200 import Precision, Tensor, flash_attention
    B, H, S, D = 8, 16, 1024, 64   # 512 work items: more than SMs, so the launch draws from a counter
    ts = [Tensor(torch.randn(B * H * S * D, device="cuda").to(torch.bfloat16), [B, H, S, D], Precision.BF16) for _ in range(6)]
    want = [flash_attention(*ts[i:i + 3], True).torch().clone() for i in (0, 3)]
    side, graphs, outs = torch.cuda.Stream(), [], []
    for i in (0, 3):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            outs.append(flash_attention(*ts[i:i + 3], True))
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(50):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(side):
            eager = flash_attention(*ts[:3], True)
    torch.cuda.synchronize()
    assert it_ctx.poll_status() == 0
    for o, w in zip(outs + [eager], want + want[:1]):
        assert torch.equal(o.torch(), w)


@pytest.mark.parametrize("B,Hkv,kv_len,D", [(19, 8, 8150, 128), (37, 4, 8064, 64), (37, 6, 8190, 64)])
def test_decode_of_a_second_wave_less_than_half_full(it_ctx, B, Hkv, kv_len, D):
    """Long caches of 149 to 222 (batch, K/V head) pairs are split over clusters of two; against fp32 of the same bf16 values."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_decode
    G, L = 2, 8192
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((B, Hkv * G, D), (B, L, Hkv, D), (B, L, Hkv, D)))
    got = attention_decode(*(Tensor(t.reshape(-1), list(t.shape), Precision.BF16) for t in (q, k, v)), kv_len)
    assert it_ctx.poll_status() == 0
    for b in (0, B - 1):
        s = torch.einsum("hgd,lhd->hgl", q[b].float().reshape(Hkv, G, D), k[b, :kv_len].float()) / math.sqrt(D)
        want = torch.einsum("hgl,lhd->hgd", torch.softmax(s, -1), v[b, :kv_len].float()).reshape(Hkv * G, D)
        o = got.torch().reshape(B, Hkv * G, D)[b].float()
        assert (o - want).norm() <= 4e-3 * want.norm()   # bf16 output (1.7e-3) and bf16 probabilities (2e-3)


def test_arguments_that_are_no_plain_numbers(it_ctx):
    """What the native host path does not take itself is converted, or refused, as the Python functions do it."""
    import ctypes

    import torch
    from irontensor_b200 import Precision, Tensor, attention_decode, flash_attention, rope, rope_qk

    def make(*shape):
        return Tensor(torch.randn(shape, device="cuda"), list(shape), Precision.FP32)

    x, k = make(1, 40, 2, 32), make(1, 40, 2, 32)
    want = rope(x, 10000.0, 3).torch()
    for base, offset in ((10000, 3), ("10000", 3), (np.float32(10000), np.int64(3)), (10000.0, 3.0), (10000.0, True + 2)):
        assert torch.equal(rope(x, base, offset).torch(), want)
        assert torch.equal(rope_qk(x, k, base, offset)[0].torch(), want)
    with pytest.raises(TypeError):
        rope(x, 10000.0, None)
    want = flash_attention(x, x, x, True).torch()
    for causal in (1, 2, np.True_, np.int32(1)):
        assert torch.equal(flash_attention(x, x, x, causal).torch(), want)
    for causal in (None, [1]):
        with pytest.raises(TypeError):
            flash_attention(x, x, x, causal)
    q, cache = make(1, 2, 32), make(1, 40, 2, 32)
    want = attention_decode(q, cache, cache, 7).torch()
    assert torch.equal(attention_decode(q, cache, cache, np.int64(7)).torch(), want)
    with pytest.raises(ctypes.ArgumentError):
        attention_decode(q, cache, cache, 7.0)
    for kv_len in (0, 41, 2 ** 40, -2 ** 70):
        with pytest.raises(AssertionError):
            attention_decode(q, cache, cache, kv_len)


def test_work_counters_survive_launches_that_did_not_start(it_ctx):
    """A wait runs out on one stream while forwards that draw their work items from a counter run on another: some of their CTAs
    start, some see the status word and do not, and the word is cleared while they run.  The next forward computes every row."""
    import torch
    from irontensor_b200 import Precision, Tensor, flash_attention
    B, H, S, D = 8, 16, 1024, 64   # 512 work items
    q, k, v = (Tensor(torch.randn(B * H * S * D, device="cuda").to(torch.bfloat16), [B, H, S, D], Precision.BF16) for _ in range(3))
    want = flash_attention(q, k, v, True).torch().clone()
    busy = torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(6):
        _lib.check(it_ctx.lib.it_selftest_wait_timeout(it_ctx.handle, it_ctx.stream(), 3 + i))
        with torch.cuda.stream(busy):
            for _ in range(150):
                flash_attention(q, k, v, True)
        with pytest.raises(_lib.ITError):
            it_ctx.poll_status()          # of the other stream: clears the word under the busy one
        with torch.cuda.stream(busy):
            o = flash_attention(q, k, v, True)
            o.torch().fill_(float("nan"))
            busy.synchronize()
            for _ in range(2):
                o = flash_attention(q, k, v, True)
        busy.synchronize()
        assert it_ctx.poll_status() == 0
        assert torch.equal(o.torch(), want)


def test_captured_forwards_give_their_counters_back(it_ctx):
    """More captured forwards than there are counters, a graph at a time: the last one still gets one (its grid is the number of
    SMs and not the number of work items)."""
    import torch
    from cuda.bindings import driver
    from irontensor_b200 import Precision, Tensor, raw
    B, H, S, D = 4, 16, 1024, 64   # 256 work items
    q = Tensor(torch.randn(B * H * S * D, device="cuda").to(torch.bfloat16), [B, H, S, D], Precision.BF16)
    o, lse = Tensor.empty([B, H, S, D], Precision.BF16), Tensor.empty([B, H, S], Precision.FP32)
    per_graph, sms = 2000, torch.cuda.get_device_properties(0).multi_processor_count

    def capture(n):
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            for _ in range(n):
                raw.fwd(_lib.IT_BF16, B, H, S, D, True, q.data_ptr(), q.data_ptr(), q.data_ptr(), o.data_ptr(), lse.data_ptr(), ctx=it_ctx)
        return g

    for i in range(34):            # 68000
        g = capture(per_graph)
        if i % 16 == 0:
            g.instantiate()
            g.replay()
        torch.cuda.synchronize()
        g.reset()
    g = capture(1)
    _, nodes, n = driver.cuGraphGetNodes(g.raw_cuda_graph(), 8)
    err, params = driver.cuGraphKernelNodeGetParams(nodes[0])
    assert n == 1 and int(err) == 0 and params.gridDimX == sms
    raw.fwd(_lib.IT_BF16, B, H, S, D, True, q.data_ptr(), q.data_ptr(), q.data_ptr(), o.data_ptr(), lse.data_ptr(), ctx=it_ctx)
    want = o.torch().clone()
    o.torch().fill_(float("nan"))
    g.instantiate()
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert it_ctx.poll_status() == 0 and torch.equal(o.torch(), want)


@pytest.mark.parametrize("B,H,Hkv,D,kv_len", [(4, 16, 2, 64, 64), (4, 16, 2, 128, 255), (4, 32, 1, 128, 129), (2, 96, 1, 64, 200),
                                              (64, 32, 8, 128, 200), (40, 16, 16, 128, 255), (4, 16, 2, 128, 24),
                                              (32, 16, 2, 64, 48), (2, 40, 4, 128, 23)])
def test_short_bf16_decode_rounds_its_result_only(it_ctx, B, H, Hkv, D, kv_len):
    """Below 256 positions the rounding of the result is all the error, whatever the group and the batch (fp32 probabilities, or two
    bf16 terms of them).  Rounding to 8 bits costs a value
    x in [1, 2) 2^-9 / sqrt(3) in the root mean square; relative to values spread over a binade that is 1.63e-3 in the 2-norm.
    Probabilities rounded to bf16 add an independent error of their own of 1.3e-3: 2.1e-3 in all.  The line lies between."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_decode
    gen = torch.Generator(device="cuda").manual_seed(B + kv_len)
    q, k, v = (torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ([B, H, D], [B, 256, Hkv, D], [B, 256, Hkv, D]))
    got = attention_decode(*(Tensor(t, list(t.shape), Precision.BF16) for t in (q, k, v)), kv_len).torch().double()
    assert it_ctx.poll_status() == 0
    qd, kd, vd = q.double().view(B, Hkv, H // Hkv, D), k[:, :kv_len].double(), v[:, :kv_len].double()
    want = torch.einsum("bhgk,bkhd->bhgd", (torch.einsum("bhgd,bkhd->bhgk", qd, kd) / D ** 0.5).softmax(-1), vd).reshape(B, H, D)
    assert ((got - want).norm() / want.norm()).item() < 1.85e-3


@pytest.mark.parametrize("tokens", [1, 8, 40])
def test_qkv_rope_asks_for_its_workspace_at_every_size(it_ctx, tokens):
    """Few tokens need no table of sines; the call is refused all the same, as it is for more."""
    import torch
    H, D, hidden = 4, 64, 256
    x = torch.zeros(tokens, hidden, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(3 * H * D, hidden, dtype=torch.bfloat16, device="cuda")
    outs = [torch.empty(tokens, H, D, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")

    def call(base, pointer, nbytes):
        return it_ctx.lib.it_qkv_rope_fwd(it_ctx.handle, it_ctx.stream(), 1, tokens, hidden, H, H, D, base, 0, x.data_ptr(), w.data_ptr(),
                                          *(o.data_ptr() for o in outs), pointer, nbytes)

    assert call(10000.0, None, 0) == _lib.IT_ERR_INVALID_ARG
    assert call(10000.0, ws.data_ptr(), 8 * tokens) == _lib.IT_ERR_INVALID_ARG
    assert call(10000.0, ws.data_ptr() + 16, 1 << 19) == _lib.IT_ERR_ALIGNMENT
    assert call(10000.0, ws.data_ptr(), 1 << 20) == _lib.IT_OK
    assert call(0.0, None, 0) == _lib.IT_OK       # without rotation there is nothing to ask for
    assert it_ctx.poll_status() == 0


@pytest.mark.parametrize("dtype,D", [("bf16", 96), ("bf16", 64), ("bf16", 128), ("bf16", 40), ("fp32", 64), ("fp32", 32)])
def test_keys_past_the_sequence_weigh_nothing(it_ctx, dtype, D):
    """Without the causal mask the last key tile of a ragged sequence holds rows past it.  Where all scores of a query are very
    low, 2^(0 - LSE) of such a row is infinite; it must not meet its zeros."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_backward_recompute, flash_attention
    B, H, S = 1, 2, 200
    gen = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, d_o = (torch.randn(B, H, S, D, generator=gen, device="cuda") for _ in range(4))
    up = round(math.sqrt(200.0 * math.sqrt(D)))    # one column that puts all scores around -200
    q[..., 0], k[..., 0] = up, -up
    t = torch.bfloat16 if dtype == "bf16" else torch.float32
    q, k, v, d_o = (x.to(t) for x in (q, k, v, d_o))
    args = [Tensor(x, [B, H, S, D], Precision.BF16 if dtype == "bf16" else Precision.FP32) for x in (q, k, v, d_o)]
    o = flash_attention(*args[:3], False)
    grads = attention_backward_recompute(args[3], *args[:3], o, o.lse, causal=False)
    assert it_ctx.poll_status() == 0
    qd, kd, vd = (x.double().requires_grad_() for x in (q, k, v))
    want = ((qd @ kd.transpose(-1, -2)) / D ** 0.5).softmax(-1) @ vd
    want.backward(d_o.double())
    for got, exact in zip((o,) + tuple(grads), (want.detach(), qd.grad, kd.grad, vd.grad)):
        got = got.torch().double()
        assert torch.isfinite(got).all()
        # Column 0 of dQ and dK is a difference of large terms.  Scores of 200 are held to 200 * 2^-24 * log2(e) in fp32, and each
        # of the D products rounds: probabilities are off by about 1e-4, whatever the type.
        err = (got - exact)[..., 1:].norm() / exact[..., 1:].norm()
        assert err.item() < (1e-2 if dtype == "bf16" else 5e-4)


def visible_pairs_oracle(q, k, v, d_o, o, lse):
    """Causal attention and its gradients, [B, S, H, D] in 64 bits, each row from the rows that it sees and no others."""
    import torch
    B, S, H, D = q.shape
    G = H // k.shape[2]
    kk, vv = (t.repeat_interleave(G, 2) for t in (k, v))
    out, dq, dk, dv = (torch.zeros_like(q) for _ in range(4))
    delta = (d_o * o).sum(-1)
    for i in range(S):
        s = torch.einsum("bhd,bkhd->bhk", q[:, i], kk[:, :i + 1]) / D ** 0.5
        out[:, i] = torch.einsum("bhk,bkhd->bhd", s.softmax(-1), vv[:, :i + 1])
        p = (s - lse[:, :, i, None]).exp()
        ds = p * (torch.einsum("bhd,bkhd->bhk", d_o[:, i], vv[:, :i + 1]) - delta[:, i, :, None])
        dq[:, i] = torch.einsum("bhk,bkhd->bhd", ds, kk[:, :i + 1]) / D ** 0.5
        s = torch.einsum("bqhd,bhd->bhq", q[:, i:], kk[:, i]) / D ** 0.5
        p = (s - lse[:, :, i:]).exp()
        ds = p * (torch.einsum("bqhd,bhd->bhq", d_o[:, i:], vv[:, i]) - delta[:, i:].transpose(1, 2))
        dk[:, i] = torch.einsum("bhq,bqhd->bhd", ds, q[:, i:]) / D ** 0.5
        dv[:, i] = torch.einsum("bhq,bqhd->bhd", p, d_o[:, i:])
    return out, dq, dk.view(B, S, H // G, G, D).sum(3), dv.view(B, S, H // G, G, D).sum(3)


@pytest.mark.parametrize("dtype,B,S,H,Hkv,D,env", [
    ("fp32", 2, 200, 2, 2, 64, {}), ("fp32", 1, 300, 4, 2, 32, {}), ("fp32", 2, 40, 2, 1, 60, {}),
    ("bf16", 1, 300, 4, 4, 96, {"IT_BWD_SPLIT": "1"}), ("bf16", 1, 300, 8, 2, 96, {"IT_BWD_SPLIT": "2"}),
    ("bf16", 1, 300, 4, 2, 40, {"IT_BWD_SPLIT": "4"}), ("bf16", 1, 300, 4, 4, 48, {"IT_BWD_KEY_TILES": "2"}),
    ("bf16", 2, 100, 2, 2, 64, {}), ("bf16", 2, 70, 4, 1, 128, {}),
])
@pytest.mark.parametrize("where,value", [("tail of K and V", float("nan")), ("tail of K and V", float("inf")), ("head of Q and dO", float("nan")),
                                         ("one value of V", float("-inf")), ("one value of dO", float("inf"))])
def test_rows_that_are_not_finite_stay_with_those_who_see_them(it_ctx, monkeypatch, dtype, B, S, H, Hkv, D, env, where, value):
    """A masked probability of 0 times an infinity is no 0: on the diagonal tile it must not meet one.  Every row of O, dQ, dK and dV
    that sees finite rows only is finite, and right; the others are not finite, as in the oracle."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_gqa, attention_gqa_backward
    for name, val in env.items():
        monkeypatch.setenv(name, val)
    gen = torch.Generator(device="cuda").manual_seed(S + D)
    t = torch.bfloat16 if dtype == "bf16" else torch.float32
    q, d_o = (torch.randn(B, S, H, D, generator=gen, device="cuda").to(t) for _ in range(2))
    k, v = (torch.randn(B, S, Hkv, D, generator=gen, device="cuda").to(t) for _ in range(2))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hkv, 2)) / D ** 0.5
    s = s.masked_fill(torch.ones(S, S, device="cuda").triu(1).bool(), float("-inf"))
    o = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v.double().repeat_interleave(H // Hkv, 2)).to(t).contiguous()
    lse = s.logsumexp(-1).float().contiguous()
    at = S - 25
    if where == "tail of K and V":
        k[:, at:, 0, 1], v[:, at:, 0] = value, value
    elif where == "head of Q and dO":
        q[:, :25, 0, 0], d_o[:, :25, H - 1] = value, value
    elif where == "one value of V":
        v[:, at, 0, 3] = value
    else:
        d_o[:, 30, 0, D - 1] = value
    want = visible_pairs_oracle(*(x.double() for x in (q, k, v, d_o, o, lse)))
    P = Precision.BF16 if dtype == "bf16" else Precision.FP32
    args = [Tensor(x, list(x.shape), P) for x in (q, k, v, d_o, o)]
    got = [attention_gqa(*args[:3], True)]
    args[4].lse = Tensor(lse, [B, H, S], Precision.FP32)
    got += attention_gqa_backward(args[3], *args[:3], args[4], True)
    assert it_ctx.poll_status() == 0
    tol = 6e-3 if dtype == "bf16" else 1e-5
    for name, g, w in zip(("o", "dq", "dk", "dv"), got, want):
        if name == "o" and dtype == "fp32":
            continue       # the fp32 forward's row tiles multiply masked zeros, as they always did
        g, fine = g.torch().double(), torch.isfinite(w)
        assert torch.equal(torch.isfinite(g), fine), f"{name}: {(torch.isfinite(g) != fine).sum().item()} values of {fine.numel()}"
        assert ((g - w)[fine].norm() / w[fine].norm()).item() < tol if fine.any() else True, name


@pytest.mark.parametrize("lowest", [float("-inf"), -3e38])
def test_leading_keys_that_score_minus_infinity(it_ctx, lowest):
    """Keys switched off by a column of the lowest value: a whole first tile of scores of -inf weighs nothing, in the padded forward
    and in the decode of fewer than 256 positions (fp32 tensors too)."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_decode, attention_gqa
    gen = torch.Generator(device="cuda").manual_seed(3)

    def softmax_v(q, k, v, G):     # q [.., h, n, d] over the keys that are on
        k, v = (x.double().repeat_interleave(G, 2).transpose(1, 2) for x in (k, v))
        s = (q[..., 1:].double() @ k[..., 1:].transpose(-1, -2) + q[..., :1].double() * k[..., :1].transpose(-1, -2).clamp(min=-1e30)) / q.shape[-1] ** 0.5
        return s, v

    for t, P in ((torch.bfloat16, Precision.BF16), (torch.float32, Precision.FP32)):
        B, S, H, D, off = 1, 300, 2, 96 if t == torch.bfloat16 else 64, 140
        q, k, v = (torch.randn(B, S, H, D, generator=gen, device="cuda").to(t) for _ in range(3))
        q[..., 0], k[..., 0] = 100.0, 0.0
        k[:, :off, :, 0] = lowest
        if t == torch.bfloat16:    # fp32 operands beyond bf16's range are beyond the split of the fp32 tensor-core forward
            o = attention_gqa(*(Tensor(x, list(x.shape), P) for x in (q, k, v)), True).torch().double()
            s, vd = softmax_v(q.transpose(1, 2), k, v, 1)
            s = s.masked_fill(torch.ones(S, S, device="cuda").triu(1).bool(), float("-inf"))
            want = (s.softmax(-1) @ vd).transpose(1, 2)
            assert torch.isfinite(o[:, off:]).all()
            assert ((o - want)[:, off:].norm() / want[:, off:].norm()).item() < 6e-3
        for H, Hkv, n, off in ((16, 2, 250, 130), (16, 2, 100, 70), (32, 1, 255, 128), (8, 8, 250, 130)):
            q = torch.randn(2, H, 64, generator=gen, device="cuda").to(t)
            k, v = (torch.randn(2, 256, Hkv, 64, generator=gen, device="cuda").to(t) for _ in range(2))
            q[..., 0], k[..., 0] = 100.0, 0.0
            k[:, :off, :, 0] = lowest
            o = attention_decode(*(Tensor(x, list(x.shape), P) for x in (q, k, v)), n).torch().double()
            s, vd = softmax_v(q[:, :, None], k[:, :n], v[:, :n], H // Hkv)
            want = (s.softmax(-1) @ vd)[:, :, 0]
            assert ((o - want).norm() / want.norm()).item() < (1.85e-3 if t == torch.bfloat16 else 1e-5)
    assert it_ctx.poll_status() == 0


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S,D", [(200, 64), (40, 32)])
def test_fp32_backward_with_keys_at_the_lowest_value(it_ctx, causal, S, D):
    """Keys switched off by a column of -FLT_MAX, which no bf16 term holds: their probabilities are 0 and so are their parts."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_backward_recompute
    gen = torch.Generator(device="cuda").manual_seed(S)
    B, H = 1, 2
    q, k, v, d_o = (torch.randn(B, H, S, D, generator=gen, device="cuda") for _ in range(4))
    q[..., 0], k[..., 0] = 1000.0, 0.0
    on = torch.arange(S, device="cuda") % 5 != 3
    k[:, :, ~on, 0] = torch.finfo(torch.float32).min
    seen = (torch.ones(S, S, device="cuda").tril().bool() if causal else torch.ones(S, S, device="cuda").bool()) & on
    qd, kd, vd = (x.double().requires_grad_() for x in (q, k.masked_fill(~on[None, None, :, None], 0.0), v))
    s = ((qd @ kd.transpose(-1, -2)) / D ** 0.5).masked_fill(~seen, float("-inf"))
    o = s.softmax(-1) @ vd
    o.backward(d_o.double())
    args = [Tensor(x.contiguous(), [B, H, S, D], Precision.FP32) for x in (d_o, q, k, v, o.detach().float())]
    lse = Tensor(s.detach().logsumexp(-1).float().contiguous(), [B, H, S], Precision.FP32)
    got = attention_backward_recompute(*args, lse, causal=causal)
    assert it_ctx.poll_status() == 0
    for g, want in zip(got, (qd.grad, kd.grad, vd.grad)):
        g = g.torch().double()
        assert torch.isfinite(g).all()
        err = (g - want)[..., 1:].norm() / want[..., 1:].norm()     # column 0: differences of terms 1000 times larger
        assert err.item() < 1e-5


def _attention_and_gradients(q, k, v, d_o, causal, rope_base=None):
    """O, dQ, dK, dV of [B, S, heads, D] tensors in 64 bits; with `rope_base` q and k are rotated tensors and dQ, dK those of the
    tensors before the rotation."""
    import torch
    B, S, H, D = q.shape
    q, k, v = (x.double().detach().requires_grad_() for x in (q, k, v))
    kk, vv = (x.repeat_interleave(H // k.shape[2], 2) for x in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q, kk) / D ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, device="cuda").triu(1).bool(), float("-inf"))
    o = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), vv)
    o.backward(d_o.double())
    dq, dk = q.grad, k.grad
    if rope_base is not None:
        inv = 1.0 / rope_base ** (torch.arange(0, D, 2, device="cuda").double() / D)
        angle = torch.arange(S, device="cuda").double()[:, None, None] * inv
        c, sn = angle.cos(), angle.sin()
        dq, dk = (torch.stack((g[..., 0::2] * c + g[..., 1::2] * sn, g[..., 1::2] * c - g[..., 0::2] * sn), -1).flatten(-2) for g in (dq, dk))
    return o.detach(), dq, dk, v.grad


@pytest.mark.parametrize("B,S,H,Hkv,D,causal,rope,force", [
    (1, 300, 4, 4, 32, True, True, True), (1, 300, 4, 2, 40, False, False, True), (2, 512, 4, 1, 56, True, True, True),
    (1, 257, 4, 4, 56, False, True, True), (2, 130, 4, 2, 24, True, False, True), (1, 640, 2, 2, 40, True, False, True),
    (16, 300, 8, 8, 32, True, True, False), (32, 200, 8, 8, 48, False, True, False),    # more than two CTAs per SM with one tile each
])
def test_bf16_padded_backward_with_two_key_tiles_per_cta(it_ctx, monkeypatch, B, S, H, Hkv, D, causal, rope, force):
    """The padded backward whose CTAs own two key tiles, odd and even numbers of them: by the switch, and by the launcher's own rule."""
    import torch
    from irontensor_b200 import Precision, Tensor, attention_gqa, attention_gqa_backward
    if force:
        monkeypatch.setenv("IT_BWD_KEY_TILES", "2")
    gen = torch.Generator(device="cuda").manual_seed(S + D)
    q, d_o = (torch.randn(B, S, H, D, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, S, Hkv, D, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    args = [Tensor(x, list(x.shape), Precision.BF16) for x in (q, k, v, d_o)]
    o = attention_gqa(*args[:3], causal)
    got = (o,) + tuple(attention_gqa_backward(args[3], *args[:3], o, causal, rope_base=10000.0 if rope else None))
    assert it_ctx.poll_status() == 0
    want = _attention_and_gradients(q, k, v, d_o, causal, 10000.0 if rope else None)
    # the bounds of test_bf16_padded_shapes_round_their_results_only, 6 % wider for dV: some of these tensors have 6000 values
    for name, g, w, bound in zip(("o", "dq", "dk", "dv"), got, want, (1.75e-3, 2.1e-3, 2.1e-3, 1.85e-3)):
        rel = ((g.torch().double() - w).norm() / w.norm()).item()
        assert rel < bound, f"{name}: {rel:.2e}"

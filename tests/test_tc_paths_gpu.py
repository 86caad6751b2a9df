"""GPU numerics for the tcgen05 paths: block-scaled NVFP4 GEMM + residual-term activation quantiser, FP8
tensor-core decode attention, FP8 tensor-core prefill flash attention.  Every kernel is compared with a plain
PyTorch fp32 restatement of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda:0")


@pytest.mark.parametrize("terms,tol", [(1, 0.2), (2, 2.5e-2), (3, 3e-3)])
def test_act_quant_residual_terms_round_trip(dev, terms, tol):
    from dgpp_b200.ops import core as ops

    torch.manual_seed(1)
    x = torch.randn(8, 1024, device=dev).to(BF)
    xa = ops.act_quant_nvfp4(x, terms)
    rel = (xa.dequant() - x.float()).abs().max().item() / x.float().abs().max().item()
    assert rel < tol


@pytest.mark.parametrize("rows,bn,terms,splits,n,k", [(4, 16, 1, 1, 384, 1024), (4, 16, 3, 1, 384, 1024), (8, 16, 3, 2, 448, 2048),
                                                       (40, 64, 3, 1, 256, 1024), (100, 128, 1, 1, 256, 1024),
                                                       (300, 256, 1, 1, 384, 1024), (30, 32, 2, 2, 256, 2048),
                                                       (8, 16, 3, 5, 640, 5120), (1, 16, 3, 7, 256, 17408),
                                                       (13, 16, 3, 8, 128, 4096)])
def test_gemm_fp4_matches_fp32_reference(dev, rows, bn, terms, splits, n, k):
    from dgpp_b200.ops import core as ops, reference as ref
    from dgpp_b200.quant.formats import quantize

    torch.manual_seed(2)
    w = quantize(torch.randn(n, k, device=dev) * 0.05, "nvfp4")
    x = torch.randn(rows, k, device=dev).to(BF)
    xa = ops.act_quant_nvfp4(x, terms, bn=bn)
    y = ops.gemm_fp4(xa, w, splits=splits)
    torch.cuda.synchronize()
    ops.check_status()
    if splits > 1:
        # both split-K forms (cluster fold through distributed shared memory, workspace fold by the last CTA) add
        # the same partials in the same order: identical bits, and repeatable
        y_ws = ops.gemm_fp4(xa, w, splits=splits, cluster=False)
        y_cl = ops.gemm_fp4(xa, w, splits=splits, cluster=True)
        torch.cuda.synchronize()
        ops.check_status()
        assert torch.equal(y_cl, y) and torch.equal(y_ws, y_cl)
    # against the product of the operands the kernel actually saw (exact up to fp32 order + one bf16 rounding)
    yq = xa.dequant() @ w.dequant().t()
    assert (y.float() - yq).abs().max().item() <= 1e-2 * yq.abs().max().item()
    # against exact bf16 activations: three residual terms are bf16-grade
    if terms == 3:
        yx = ref.linear(x, w, out_fp32=True)
        assert (y.float() - yx).abs().max().item() <= 1.2e-2 * yx.abs().max().item()


def test_fused_producers_match_reference(dev):
    from dgpp_b200.ops import core as ops, reference as ref

    torch.manual_seed(3)
    H, I = 1024, 2048
    x = torch.randn(5, H, device=dev).to(BF)
    d = torch.randn(5, H, device=dev).to(BF)
    wn = (1 + 0.1 * torch.randn(H, device=dev)).to(BF)
    xr, xo = x.clone(), torch.empty_like(x)
    xa = ops.act_quant_nvfp4(xr, 3, mode="rmsnorm", delta=d, norm_w=wn, x_out=xo)
    yr, res = ref.rmsnorm(x, wn, 1e-6, d)
    assert torch.equal(xr, res)                                           # residual stream updated in place
    assert (xo.float() - yr.float()).abs().max().item() <= 0.04
    assert ((xa.dequant() - yr.float()).abs().max() / yr.float().abs().max()).item() < 1e-2
    gu = (torch.randn(5, 2 * I, device=dev) * 2).to(BF)
    ao = torch.empty(5, I, device=dev, dtype=BF)
    xa = ops.act_quant_nvfp4(gu, 3, mode="swiglu", x_out=ao)
    ar = ref.swiglu(gu)
    assert (ao.float() - ar.float()).abs().max().item() <= 0.07
    assert ((xa.dequant() - ar.float()).abs().max() / ar.float().abs().max()).item() < 1e-2


@pytest.mark.parametrize("rows,k,terms", [(1, 256, 3), (3, 768, 2), (16, 2304, 3), (5, 17408, 3), (2, 36864, 1)])
def test_cluster_quantiser_matches_the_single_cta_one(dev, rows, k, terms):
    """Rows split over a cluster: segments of less than a warp, of no whole number of warps, of more columns than threads hold at
    once.  Plain and SwiGLU rows give the same codes, block scales and row scale as the one-CTA kernel (a maximum does not
    depend on its order); the norm's sum of squares is added in another order, so its rows are compared as values."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(33)
    bn = 16
    x = torch.randn(rows, k, device=dev).to(BF)
    gu = (2 * torch.randn(rows, 2 * k, device=dev)).to(BF)
    d, w = torch.randn(rows, k, device=dev).to(BF), (1 + 0.1 * torch.randn(k, device=dev)).to(BF)
    for m, (mode, inp, kw) in enumerate((("plain", x, {}), ("swiglu", gu, {}), ("rmsnorm", x, dict(delta=d, norm_w=w)))):
        got, want = ops.QuantAct(bn, k, terms, bn, dev), ops.QuantAct(bn, k, terms, bn, dev)
        ops.act_quant_nvfp4(inp.clone(), terms, out=got, mode=mode, **kw)
        want.rows, x2 = rows, inp.clone()
        ops.call("dgpp_act_quant_nvfp4", m, ops.ptr(x2), x2.stride(0), ops.ptr(kw.get("delta")), ops.ptr(kw.get("norm_w")), ops.ptr(x2), None,
                 ops.ptr(want.q), ops.ptr(want.sf), ops.ptr(want.g), rows, bn, k, terms, bn, 1e-6, 0.0, 0.0, 0, ops.stream_ptr())
        torch.cuda.synchronize()
        ops.check_status()
        if mode != "rmsnorm":
            assert torch.equal(got.g, want.g) and torch.equal(got.q, want.q) and torch.equal(got.sf, want.sf), mode
        else:      # one bf16 rounding of the normed value may fall the other way: 2^-8 of it, plus a step of the last term
            a, b = got.dequant(), want.dequant()
            assert ((a - b).norm() / b.norm()).item() < 2.0 ** -8 * (1 if terms > 1 else 8)


@pytest.mark.parametrize("rows,k,terms,bn", [(65, 256, 3, 16), (130, 5120, 3, 64), (129, 2304, 1, 128), (66, 24320, 2, 16)])
def test_bulk_quantiser_matches_the_cluster_one(dev, rows, k, terms, bn):
    """One CTA per row above 64 rows: fewer blocks of 16 than threads, a remainder of them, a wide row; the same bits as the
    cluster form (the row statistic is a maximum), the copy of the rows included."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(34)
    pad = (rows + bn - 1) // bn * bn
    for m, (mode, cols) in enumerate((("plain", k), ("swiglu", 2 * k))):
        inp = (2 * torch.randn(rows, cols, device=dev)).to(BF)
        inp[1].zero_()
        got, want = ops.QuantAct(pad, k, terms, bn, dev), ops.QuantAct(pad, k, terms, bn, dev)
        x1, x2 = (torch.empty(rows, k, device=dev, dtype=BF) for _ in range(2))
        ops.act_quant_nvfp4(inp, terms, out=got, mode=mode, x_out=x1)
        ops.call("dgpp_act_quant_nvfp4_cluster", m, ops.ptr(inp), inp.stride(0), None, None, None, ops.ptr(x2), ops.ptr(want.q), ops.ptr(want.sf),
                 ops.ptr(want.g), rows, pad, k, terms, bn, 8, 1e-6, 0.0, 0.0, 0, None, None, 0, ops.stream_ptr())
        torch.cuda.synchronize()
        ops.check_status()
        assert torch.equal(got.g, want.g) and torch.equal(got.q, want.q) and torch.equal(got.sf, want.sf) and torch.equal(x1, x2), mode


@pytest.mark.parametrize("rows,k,mode", [(65, 24576, "plain"), (65, 24576, "swiglu"), (65, 24832, "plain"), (66, 48640, "swiglu"),
                                         (65, 49152, "plain"), (2, 49152, "rmsnorm"), (1, 196608, "plain")])
def test_quantiser_of_the_widest_rows(dev, rows, k, mode):
    """Row segments up to the 48 KB that a CTA takes, and one past it (two CTAs): every width that the entry point's own
    bound admits is launched.  Three terms keep a value to 2^-3 of a 4-bit step each: well below 1e-2 of a row's largest."""
    from dgpp_b200.ops import core as ops, reference as ref

    torch.manual_seed(35)
    x = torch.randn(rows, 2 * k if mode == "swiglu" else k, device=dev).to(BF)
    w = (1 + 0.1 * torch.randn(k, device=dev)).to(BF) if mode == "rmsnorm" else None
    got = ops.act_quant_nvfp4(x, 3, mode=mode, norm_w=w)
    torch.cuda.synchronize()
    ops.check_status()
    want = x if mode == "plain" else ops.swiglu(x) if mode == "swiglu" else ref.rmsnorm(x, w, 1e-6)[0]
    err = (got.dequant() - want.float()).abs().amax(1) / want.float().abs().amax(1)
    assert err.max().item() < 1e-2


@pytest.mark.parametrize("m,k", [(0, 24576), (1, 24576), (2, 24320), (2, 24576)])
def test_quantiser_of_one_whole_row_per_cta(dev, m, k):
    """One CTA per row up to 48 KB of it, all modes; plain and SwiGLU rows bit for bit as in a cluster of eight."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(36)
    x = torch.randn(3, 2 * k if m == 1 else k, device=dev).to(BF)
    w = (1 + 0.1 * torch.randn(k, device=dev)).to(BF)
    got = []
    for cl in (1, 8):
        a = ops.QuantAct(16, k, 3, 16, dev)
        a.rows = 3
        ops.call("dgpp_act_quant_nvfp4_cluster", m, ops.ptr(x), x.stride(0), None, ops.ptr(w), None, None, ops.ptr(a.q), ops.ptr(a.sf), ops.ptr(a.g),
                 3, 16, k, 3, 16, cl, 1e-6, 0.0, 0.0, 0, None, None, 0, ops.stream_ptr())
        got.append(a)
    torch.cuda.synchronize()
    ops.check_status()
    a, b = got
    if m != 2:
        assert torch.equal(a.g, b.g) and torch.equal(a.q, b.q) and torch.equal(a.sf, b.sf)
    else:      # the sum of squares in another order: one bf16 rounding of the normed value may fall the other way
        assert ((a.dequant() - b.dequant()).norm() / b.dequant().norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("k,one_plus,with_delta", [(256, 0, True), (2048, 1, False), (5120, 0, True), (5888, 1, True), (8192, 0, True), (17408, 0, False)])
def test_bulk_quantiser_of_normed_rows_matches_the_cluster_one(dev, k, one_plus, with_delta):
    """Above the line one CTA per row, in passes of 64 rows a cluster each: the same codes, scales, normed rows and sums, bit for
    bit (segments of less than a warp, of no whole number of warps, and of several columns per thread)."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(37)
    rows, terms, bn = 272, 2, 16
    x, d = torch.randn(rows, k, device=dev).to(BF), torch.randn(rows, k, device=dev).to(BF)
    x[5].zero_()
    w = (0.1 * torch.randn(k, device=dev) + 1 - one_plus).to(BF)
    args = dict(mode="rmsnorm", norm_w=w, one_plus_w=bool(one_plus))
    got, xs, xn = ops.QuantAct(rows, k, terms, bn, dev), x.clone(), torch.empty_like(x)
    ops.act_quant_nvfp4(xs, terms, out=got, x_out=xn, delta=d if with_delta else None, **args)
    for r in range(0, rows, 64):
        part = x[r:r + 64].clone()
        want, n = ops.QuantAct(part.shape[0], k, terms, bn, dev), torch.empty_like(part)
        ops.act_quant_nvfp4(part, terms, out=want, x_out=n, delta=d[r:r + 64] if with_delta else None, **args)
        torch.cuda.synchronize()
        ops.check_status()
        at = slice(r, r + part.shape[0])
        assert torch.equal(got.g[at], want.g) and torch.equal(xn[at], n) and torch.equal(xs[at], part)
        assert torch.equal(got.q.view(rows, -1)[at], want.q.view(part.shape[0], -1))
        assert torch.equal(got.sf.view(rows, -1)[at], want.sf.view(part.shape[0], -1))


def _filled_cache(dev, hq, hkv, ctx, page, slot, d=128):
    from dgpp_b200.engine.kv_cache import PagedKV
    from dgpp_b200.ops import core as ops, reference as ref

    kv = PagedKV(1, hkv, d, max(64, 4 * (ctx // page + 2)), 4, ctx // page + 2, page, True, dev)
    inv_freq, _ = ref.rope_inv_freq(d, 1e4, dev)
    qkv = torch.randn(ctx, (hq + 2 * hkv) * d, device=dev).to(BF)
    pos = torch.arange(ctx, device=dev, dtype=torch.int32)
    req = torch.full((ctx,), slot, device=dev, dtype=torch.int32)
    assert kv.reserve(slot, ctx)
    ops.rope_kv_write(qkv, pos, req, kv.block_table, inv_freq, kv.layers[0], hq, hkv, d)
    return kv, qkv, pos, req


def _torch_attention(kv, qkv, slot, rows_pos, hq, hkv, scale, d=128):
    """fp32 attention over the dequantised cache contents for the query rows at positions rows_pos."""
    from dgpp_b200.ops import reference as ref

    cache = kv.layers[0]
    ctx = int(rows_pos.max().item()) + 1
    blocks = kv.block_table[slot].long()
    page = cache.page
    tok = torch.arange(ctx, device=qkv.device)
    blk, off = blocks[tok // page], tok % page
    k = cache.k[blk, :, off].view(torch.float8_e4m3fn).float() * cache.k_scale[blk, :, off].unsqueeze(-1)
    v = cache.v[blk, :, off].view(torch.float8_e4m3fn).float() * cache.v_scale[blk, :, off].unsqueeze(-1)
    outs = []
    for p in rows_pos.tolist():
        q = qkv[p, :hq * d].float().view(1, hq, d)
        outs.append(ref.attention(q, k[:p + 1], v[:p + 1], scale).reshape(1, hq * d))
    return torch.cat(outs)


@pytest.mark.parametrize("hq,hkv,ctx,page,splits", [(10, 2, 333, 64, 1), (10, 2, 333, 64, 2), (40, 8, 2048, 64, 4),
                                                    (8, 1, 700, 16, 2), (16, 2, 1000, 128, 3)])
def test_attn_decode_tc(dev, hq, hkv, ctx, page, splits):
    from dgpp_b200.ops import core as ops

    torch.manual_seed(4)
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, page, slot=2)
    scale = 1.0 / math.sqrt(128)
    sel = torch.tensor([ctx - 1, ctx // 2, 5], device=dev)
    q, p_, r_ = qkv[sel].contiguous(), pos[sel].contiguous(), req[sel].contiguous()
    out = ops.attn_decode_tc(q, q.stride(0), kv.layers[0], kv.block_table, r_, p_, hq, hkv, 128, scale, splits=splits)
    torch.cuda.synchronize()
    ops.check_status()
    want = _torch_attention(kv, qkv, 2, sel, hq, hkv, scale)
    assert (out.float() - want).abs().max().item() < 0.02


@pytest.mark.parametrize("hq,hkv,ctx,splits", [(40, 8, 2048, 4), (16, 2, 700, 3), (8, 8, 333, 2)])
def test_attn_combine_quant_matches_unfused(dev, hq, hkv, ctx, splits):
    """The quantiser that folds the split-KV partials itself writes the same bf16 rows and the same NVFP4 terms
    (payload, block scales, row scales) as the stand-alone combine kernel followed by the plain quantiser."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(14)
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, 64, slot=2)
    scale = 1.0 / math.sqrt(128)
    sel = torch.tensor([ctx - 1, ctx // 2, 5, ctx // 3, 64], device=dev)
    q, p_, r_ = qkv[sel].contiguous(), pos[sel].contiguous(), req[sel].contiguous()
    rows, k = sel.numel(), hq * 128
    scratch = (torch.empty(rows * hq * splits * 2, dtype=torch.float32, device=dev),
               torch.empty(rows * hq * splits * 128, dtype=torch.float32, device=dev))
    want_x = ops.attn_decode_tc(q, q.stride(0), kv.layers[0], kv.block_table, r_, p_, hq, hkv, 128, scale,
                                splits=splits, scratch=scratch)
    want = ops.act_quant_nvfp4(want_x, terms=3, bn=16, mode="plain")
    assert ops.attn_decode_tc(q, q.stride(0), kv.layers[0], kv.block_table, r_, p_, hq, hkv, 128, scale,
                              splits=splits, scratch=scratch, partials_only=True) is None
    got = ops.QuantAct(want.rows_pad, k, 3, 16, dev)
    got_x = torch.zeros(rows, k, dtype=torch.bfloat16, device=dev)
    ops.attn_combine_quant(scratch, rows, splits, hq, 128, out=got, x_out=got_x)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(got_x, want_x)
    assert torch.equal(got.g, want.g) and torch.equal(got.q, want.q) and torch.equal(got.sf, want.sf)


@pytest.mark.parametrize("hq,hkv,ctx,page,pos0,T", [(10, 2, 256, 64, 0, 256), (10, 2, 700, 64, 0, 700),
                                                   (40, 8, 1000, 64, 300, 513), (8, 2, 400, 16, 77, 200),
                                                   (4, 4, 130, 128, 1, 129)])
def test_attn_prefill_tc(dev, hq, hkv, ctx, page, pos0, T):
    from dgpp_b200.ops import core as ops

    torch.manual_seed(5)
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, page, slot=1)
    scale = 1.0 / math.sqrt(128)
    q = qkv[pos0:pos0 + T]
    out = ops.attn_prefill_tc(q, q.stride(0), kv.layers[0], kv.block_table[1], pos0, hq, hkv, 128, scale)
    torch.cuda.synchronize()
    ops.check_status()
    # spot-check rows spread over the chunk (first, tile edges, last) against fp32 attention
    rows = sorted({0, 1, min(T - 1, 127), min(T - 1, 128), T // 2, T - 1})
    want = _torch_attention(kv, qkv, 1, torch.tensor([pos0 + r for r in rows], device=dev), hq, hkv, scale)
    got = out[torch.tensor(rows, device=dev)].float()
    assert (got - want).abs().max().item() < 0.02
    # and every row against the CUDA-core decode kernel
    base = ops.attn_decode(q, q.stride(0), kv.layers[0], kv.block_table, req[pos0:pos0 + T].contiguous(),
                           pos[pos0:pos0 + T].contiguous(), hq, hkv, 128, scale, splits=1)
    assert (out.float() - base.float()).abs().max().item() < 0.03


@pytest.mark.parametrize("hq,hkv,ctx,page,pos0,T,window", [(4, 1, 1, 64, 0, 1, 0), (5, 1, 200, 64, 73, 127, 0), (4, 4, 300, 128, 172, 128, 0),
                                                          (10, 2, 1500, 16, 1371, 129, 0), (40, 8, 1000, 64, 300, 513, 0),
                                                          (48, 16, 700, 64, 0, 500, 200), (8, 2, 900, 32, 640, 260, 130)])
def test_attn_prefill_tc_error(dev, hq, hkv, ctx, page, pos0, T, window):
    """Edges of the row and token tiles, one unit per CTA and two (an odd number of units among them), windows, block scales that
    differ by 2^16 inside a tile, and whatever bytes the unwritten rest of a page holds.  Q is exact, K, V and P are rounded
    once to 11 bits and the output to 8: 2^-9 relative error of an output element, twice that allowed for the sums."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(6)
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, page, slot=1)
    cache, scale = kv.layers[0], 1.0 / math.sqrt(128)
    tok = torch.arange(ctx, device=dev)
    blk, off = kv.block_table[1].long()[tok // page], tok % page
    written = torch.zeros(cache.k.shape[0], page, dtype=torch.bool, device=dev)
    written[blk, off] = True
    k0, v0 = cache.k_scale[blk, :, off].clone(), cache.v_scale[blk, :, off].clone()
    cache.k.view(torch.uint8).masked_fill_(~written[:, None, :, None], 0x7F)          # e4m3 NaN
    cache.v.view(torch.uint8).masked_fill_(~written[:, None, :, None], 0x7F)
    cache.k_scale.masked_fill_(~written[:, None, :], float("nan"))
    cache.v_scale.masked_fill_(~written[:, None, :], float("nan"))
    spread = torch.exp2(-torch.randint(0, 17, (ctx, 1), device=dev).float())
    cache.k_scale[blk, :, off] = k0 * spread.flip(0)
    cache.v_scale[blk, :, off] = v0 * spread
    q = qkv[pos0:pos0 + T]
    out = ops.attn_prefill_tc(q, q.stride(0), cache, kv.block_table[1], pos0, hq, hkv, 128, scale, window=window)
    torch.cuda.synchronize()
    ops.check_status()
    K = (cache.k[blk, :, off].view(torch.float8_e4m3fn).double() * cache.k_scale[blk, :, off].double().unsqueeze(-1)).permute(1, 2, 0)
    V = (cache.v[blk, :, off].view(torch.float8_e4m3fn).double() * cache.v_scale[blk, :, off].double().unsqueeze(-1)).transpose(0, 1)
    Q = q[:, :hq * 128].double().view(T, hkv, hq // hkv, 128).permute(1, 2, 0, 3)
    S = torch.einsum("ghtd,gdc->ghtc", Q, K) * scale
    mine = torch.arange(pos0, pos0 + T, device=dev)
    seen = tok[None, :] <= mine[:, None]
    if window:
        seen &= tok[None, :] > mine[:, None] - window
    want = torch.einsum("ghtc,gcd->ghtd", S.masked_fill(~seen, float("-inf")).softmax(-1), V).permute(2, 0, 1, 3).reshape(T, hq * 128)
    err = (out.double() - want).view(T, hq, 128).norm(dim=-1) / want.view(T, hq, 128).norm(dim=-1)
    assert err.max().item() < 2.0 ** -8, err.max().item()
    # a row's bits do not depend on the chunk it came in
    if T > 129:
        part = ops.attn_prefill_tc(q[-129:], q.stride(0), cache, kv.block_table[1], pos0 + T - 129, hq, hkv, 128, scale, window=window)
        assert torch.equal(part, out[-129:])


@pytest.mark.parametrize("hq,hkv,pos0,T,part", [(4, 1, 0, 513, 200), (5, 1, 70, 300, 131), (40, 8, 300, 1000, 300), (10, 2, 1371, 129, 3),
                                                (40, 8, 0, 1100, 613)])
def test_attn_prefill_tc_rows_do_not_depend_on_later_tokens(dev, hq, hkv, pos0, T, part):
    """A chunk and a prefix of it that ends inside a tile of tokens (one unit per CTA and two, another partner among them), the
    tokens behind the prefix with the largest scales: the same bits.  V's elements stay above 2^-14 of the largest scale here."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(7)
    ctx = pos0 + T
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, 64, slot=1)
    cache, scale = kv.layers[0], 1.0 / math.sqrt(128)
    tok = torch.arange(ctx, device=dev)
    blk, off = kv.block_table[1].long()[tok // 64], tok % 64
    grow = torch.where(tok >= pos0 + part, 4.0, torch.where(tok >= ctx // 2, 1.0, 0.5)).unsqueeze(1)
    cache.k_scale[blk, :, off] *= grow
    cache.v_scale[blk, :, off] *= grow
    q = qkv[pos0:]
    whole = ops.attn_prefill_tc(q, q.stride(0), cache, kv.block_table[1], pos0, hq, hkv, 128, scale)
    few = ops.attn_prefill_tc(q[:part], q.stride(0), cache, kv.block_table[1], pos0, hq, hkv, 128, scale)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(whole[:part], few)


@pytest.mark.parametrize("small", [-17, -22])
@pytest.mark.parametrize("hq,hkv", [(4, 2), (40, 8)])
def test_attn_prefill_tc_small_rows_beside_zero_ones(dev, small, hq, hkv):
    """Keys and values of small amplitude next to rows of zeros, which carry a scale of one, seen and not yet visible: the same
    relative error as everywhere (K is exact, V and P are rounded once to 11 bits, the output to 8)."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(8)
    ctx, pos0 = 700, 100
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, 64, slot=1)
    cache, scale = kv.layers[0], 2.0 ** -small / math.sqrt(128)
    tok = torch.arange(ctx, device=dev)
    blk, off = kv.block_table[1].long()[tok // 64], tok % 64
    zero = torch.tensor([5, 127, 130, 240, 600, 699], device=dev)
    for t, sc in ((cache.k, cache.k_scale), (cache.v, cache.v_scale)):
        sc[blk, :, off] *= 2.0 ** small
        t.view(torch.uint8)[blk[zero], :, off[zero]] = 0
        sc[blk[zero], :, off[zero]] = 1.0
    q = qkv[pos0:]
    out = ops.attn_prefill_tc(q, q.stride(0), cache, kv.block_table[1], pos0, hq, hkv, 128, scale)
    torch.cuda.synchronize()
    ops.check_status()
    K = (cache.k[blk, :, off].view(torch.float8_e4m3fn).double() * cache.k_scale[blk, :, off].double().unsqueeze(-1)).permute(1, 2, 0)
    V = (cache.v[blk, :, off].view(torch.float8_e4m3fn).double() * cache.v_scale[blk, :, off].double().unsqueeze(-1)).transpose(0, 1)
    Q = q[:, :hq * 128].double().view(ctx - pos0, hkv, hq // hkv, 128).permute(1, 2, 0, 3)
    S = torch.einsum("ghtd,gdc->ghtc", Q, K) * scale
    seen = tok[None, :] <= tok[pos0:, None]
    want = torch.einsum("ghtc,gcd->ghtd", S.masked_fill(~seen, float("-inf")).softmax(-1), V).permute(2, 0, 1, 3).reshape(ctx - pos0, hq * 128)
    err = (out.double() - want).view(-1, hq, 128).norm(dim=-1) / want.view(-1, hq, 128).norm(dim=-1)
    assert err.max().item() < 2.0 ** -8, err.max().item()


@pytest.mark.parametrize("hq,hkv,ctx,page,splits", [(16, 2, 333, 64, 1), (16, 2, 1500, 64, 5), (8, 2, 700, 16, 2),
                                                    (4, 4, 130, 128, 3), (16, 2, 300, 64, 16)])
def test_attn_decode_tc_head_dim_256(dev, hq, hkv, ctx, page, splits):
    """head_dim 256: two 128-byte halves per K / V / q tile; splits past the end of a short context write empty partials."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(14)
    d = 256
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, page, slot=2, d=d)
    scale = 1.0 / math.sqrt(d)
    sel = torch.tensor([ctx - 1, ctx // 2, 5], device=dev)
    q, p_, r_ = qkv[sel].contiguous(), pos[sel].contiguous(), req[sel].contiguous()
    out = ops.attn_decode_tc(q, q.stride(0), kv.layers[0], kv.block_table, r_, p_, hq, hkv, d, scale, splits=splits)
    torch.cuda.synchronize()
    ops.check_status()
    want = _torch_attention(kv, qkv, 2, sel, hq, hkv, scale, d=d)
    assert (out.float() - want).abs().max().item() < 0.02


@pytest.mark.parametrize("hq,hkv,ctx,page,pos0,T", [(16, 2, 256, 64, 0, 256), (16, 2, 700, 64, 0, 700),
                                                   (8, 2, 1000, 64, 300, 513), (8, 2, 400, 16, 77, 200),
                                                   (4, 4, 130, 128, 1, 129)])
def test_attn_prefill_tc_head_dim_256(dev, hq, hkv, ctx, page, pos0, T):
    """head_dim 256 prefill kernel (two softmax sets, one per output half) against fp32 attention and the CUDA-core rows."""
    from dgpp_b200.ops import core as ops

    torch.manual_seed(15)
    d = 256
    kv, qkv, pos, req = _filled_cache(dev, hq, hkv, ctx, page, slot=1, d=d)
    scale = 1.0 / math.sqrt(d)
    q = qkv[pos0:pos0 + T]
    out = ops.attn_prefill_tc(q, q.stride(0), kv.layers[0], kv.block_table[1], pos0, hq, hkv, d, scale)
    torch.cuda.synchronize()
    ops.check_status()
    rows = sorted({0, 1, min(T - 1, 127), min(T - 1, 128), T // 2, T - 1})
    want = _torch_attention(kv, qkv, 1, torch.tensor([pos0 + r for r in rows], device=dev), hq, hkv, scale, d=d)
    got = out[torch.tensor(rows, device=dev)].float()
    assert (got - want).abs().max().item() < 0.02
    base = ops.attn_decode(q, q.stride(0), kv.layers[0], kv.block_table, req[pos0:pos0 + T].contiguous(),
                           pos[pos0:pos0 + T].contiguous(), hq, hkv, d, scale, splits=1)
    assert (out.float() - base.float()).abs().max().item() < 0.03


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
@pytest.mark.parametrize("rows,n,k", [(512, 512, 1024), (700, 1024, 512), (300, 256, 2048), (2048, 5120, 1024)])
def test_pair_gemm_is_bit_identical_to_the_single_cta_kernel(fmt, rows, n, k):
    """4-bit prefill GEMM on CTA pairs (one 256 x 256 MMA tile per pair, each CTA converting its own weight rows and
    loading its own token half): same bits as the single-CTA kernel, with and without the residual add, for token
    counts that leave the second CTA's half partly or wholly outside the matrix."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(rows + n)
    w = random_quant_linear(n, k, fmt, dev)
    x = torch.randn(rows, k, device=dev).to(torch.bfloat16)
    resid = torch.randn(rows, n, device=dev).to(torch.bfloat16)
    old = ops.PAIR_GEMM
    try:
        ops.PAIR_GEMM = False
        want, want_r = ops.gemm_tc(x, w, splits=1), ops.gemm_tc(x, w, resid=resid, splits=1)
    finally:
        ops.PAIR_GEMM = old
    got, got_r = ops.gemm_tc_pair(x, w), ops.gemm_tc_pair(x, w, resid=resid)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(got, want) and torch.equal(got_r, want_r)
    ref = (x.float() @ w.dequant().float().t())
    assert (got.float() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item() + 1e-2


@pytest.mark.parametrize("rows,n,k,bn,splits", [(1, 256, 256, 0, 1), (15, 8224, 512, 16, 1), (17, 520, 1024, 32, 1), (257, 768, 768, 256, 1),
                                                (300, 384, 512, 240, 1), (8, 512, 2048, 0, 3), (173, 1000, 2048, 96, 4),
                                                (64, 260, 1024, 0, 2)])
def test_pair_gemm_tiles_and_splits(rows, n, k, bn, splits):
    """Token tiles of any multiple of 16, ragged N (full and partial row vectors), one round and several: the single-CTA kernel's
    bits without splits.  With splits only the fp32 sums are grouped differently (1e-5 of the sum of |terms|, k <= 2048 adds
    in 2^-24), then one bf16 rounding of each (2^-8)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(rows * n)
    w = random_quant_linear(n, k, "nvfp4", dev)
    x = torch.randn(rows, k, device=dev).to(torch.bfloat16)
    resid = torch.randn(rows, n, device=dev).to(torch.bfloat16)
    old = ops.PAIR_GEMM
    try:
        ops.PAIR_GEMM = False
        want, want_r = ops.gemm_tc(x, w, splits=1), ops.gemm_tc(x, w, resid=resid, splits=1)
    finally:
        ops.PAIR_GEMM = old
    for _ in range(2):                                   # the second call finds the counters as the first left them
        got, got_r = ops.gemm_tc_pair(x, w, bn=bn, splits=splits), ops.gemm_tc_pair(x, w, resid=resid, bn=bn, splits=splits)
        torch.cuda.synchronize()
        ops.check_status()
        if splits == 1:
            assert torch.equal(got, want) and torch.equal(got_r, want_r)
        else:
            terms = x.float().abs() @ w.dequant().abs().t()
            assert ((got.float() - want.float()).abs() <= 2 ** -7 * want.float().abs() + 1e-5 * terms).all()
            assert ((got_r.float() - want_r.float()).abs() <= 2 ** -7 * (want.float().abs() + want_r.float().abs()) + 1e-5 * terms).all()


@pytest.mark.parametrize("bn", [32, 128, 192])
def test_pair_gemm_grouped_equals_the_plain_form_per_matrix(bn):
    """Stacked matrices, tiles in any order with skipped ones between: every tile's rows are those of the plain product with its
    matrix, skipped tiles keep what was there."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(bn)
    n, k, experts = 512, 768, 5
    ws = [random_quant_linear(n, k, "nvfp4", dev) for _ in range(experts)]
    q, sf = torch.cat([w.payload for w in ws]), torch.cat([w.tiled_scales().reshape(-1) for w in ws])
    alphas = torch.tensor([w.alpha for w in ws], device=dev)
    groups = [3, 0, 0, -1, 4, 1, -1]
    x = torch.randn(len(groups) * bn, k, device=dev).to(torch.bfloat16)
    out = torch.full((len(groups) * bn, n), 7.0, device=dev, dtype=torch.bfloat16)
    ops.gemm_tc_pair_grouped(x, q, sf, alphas, out, n, k, experts, torch.tensor(groups, dtype=torch.int32, device=dev), bn)
    torch.cuda.synchronize()
    ops.check_status()
    for t, e in enumerate(groups):
        rows = slice(t * bn, (t + 1) * bn)
        want = ops.gemm_tc_pair(x[rows], ws[e]) if e >= 0 else torch.full_like(out[rows], 7.0)
        assert torch.equal(out[rows], want), (t, e)


@pytest.mark.parametrize("bn,terms,slots", [(16, 1, 5), (16, 2, 5), (16, 3, 300), (64, 1, 5), (32, 3, 170), (128, 1, 5), (64, 3, 160), (256, 1, 80)])
@pytest.mark.parametrize("own_rows", [False, True])
def test_grouped_block_scaled_linear_equals_the_plain_one_per_matrix(bn, terms, slots, own_rows):
    """Every tile width, one unit per CTA and several (both accumulators, or the one that 256 columns leave room for), unused
    slots between, shared rows and the slots' own: the bits of the plain product with the slot's matrix.  The debug stamps
    are written by the grouped form as well."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(bn + terms)
    n, k, experts, rows = 256, 768, 3, bn - 3
    ws = [random_quant_linear(n, k, "nvfp4", dev) for _ in range(experts)]
    q, sf = torch.cat([w.payload for w in ws]), torch.cat([w.tiled_scales().reshape(-1) for w in ws])
    alphas = torch.tensor([w.alpha for w in ws], device=dev)
    groups = [-1 if i % 4 == 1 else (i * 7 // 3) % experts for i in range(slots)]
    tiles = slots if own_rows else 1
    xa = ops.QuantAct(tiles * bn, k, terms, bn, dev)
    ops.act_quant_nvfp4(torch.randn(tiles * bn, k, device=dev).to(BF), terms, out=xa)
    out = torch.full((slots, bn, n), 7.0, device=dev, dtype=BF)
    stamps = torch.zeros(8, dtype=torch.int64, device=dev)
    ops.call("dgpp_gemm_fp4_set_trace", ops.ptr(stamps))
    try:
        ops.gemm_fp4_grouped(xa, q, sf, alphas, out, rows, n, k, experts, torch.tensor(groups, dtype=torch.int32, device=dev), own_rows)
    finally:
        ops.call("dgpp_gemm_fp4_set_trace", None)
    torch.cuda.synchronize()
    ops.check_status()
    for s, e in enumerate(groups):
        if e < 0:
            assert (out[s] == 7.0).all()
            continue
        one = ops.QuantAct(bn, k, terms, bn, dev)
        t = s if own_rows else 0
        one.q, one.sf, one.g = (v.reshape(tiles, -1)[t].reshape(shape) for v, shape in ((xa.q, one.q.shape), (xa.sf, one.sf.shape), (xa.g, one.g.shape)))
        one.rows = rows
        assert torch.equal(out[s, :rows], ops.gemm_fp4(one, ws[e], splits=1)), (s, e)
        assert (out[s, rows:] == 7.0).all()
    st = stamps.tolist()[:7]
    assert 0 < st[0] <= st[1] <= st[2] <= st[3] <= min(st[4], st[5]) and max(st[4], st[5]) <= st[6], st


@pytest.mark.parametrize("rows,n,k,splits", [(8, 40960, 512, 2), (128, 10240, 2048, 8)])
def test_pair_gemm_split_counters_are_at_rest_after_several_units_per_pair(rows, n, k, splits):
    """More (tile, split) units than pairs, so that every pair counts itself in at several tiles: all counters end at zero, and a second
    product through the same workspace gives the same bits."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(n)
    w = random_quant_linear(n, k, "nvfp4", dev)
    x = torch.randn(rows, k, device=dev).to(torch.bfloat16)
    ws = ops.GemmWorkspace(dev)
    one = ops.gemm_tc_pair(x, w, splits=splits, ws=ws)
    torch.cuda.synchronize()
    ops.check_status()
    assert not ws.counters.any()
    assert torch.equal(ops.gemm_tc_pair(x, w, splits=splits, ws=ws), one)


@pytest.mark.parametrize("n,k", [(5120, 17408), (2048, 5632), (520, 2048)])
def test_pair_gemm_rows_do_not_depend_on_the_batch(n, k):
    """Up to 128 rows all passes split K alike, above none does (the single-CTA kernel's unsplit bits): on either side of that line a
    row has the same bits whatever the number of rows."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import random_quant_linear

    dev = torch.device("cuda:0")
    torch.manual_seed(n)
    w = random_quant_linear(n, k, "nvfp4", dev)
    x = torch.randn(2048, k, device=dev).to(torch.bfloat16)
    some = ops.gemm_tc(x[:128], w)
    for rows in (1, 8, 63, 64, 65, 100):
        assert torch.equal(ops.gemm_tc(x[:rows], w), some[:rows]), rows
    many = ops.gemm_tc(x, w)
    for rows in (129, 173, 256, 300, 512, 953, 1024):
        assert torch.equal(ops.gemm_tc(x[:rows], w), many[:rows]), rows
    old = ops.PAIR_GEMM
    try:
        ops.PAIR_GEMM = False
        assert torch.equal(ops.gemm_tc(x[:173], w, splits=1), many[:173])
    finally:
        ops.PAIR_GEMM = old
    torch.cuda.synchronize()
    ops.check_status()

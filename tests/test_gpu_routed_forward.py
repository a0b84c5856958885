"""The forward with the online router inside it (attention_forward_routed: no stand-alone statistic pass) against the
stand-alone form (router_statistic -> precision_map_online -> attention_forward_quantized) and against the CPU oracle:
the precision map must be identical, the outputs equal within the merge's rounding, and the oracle tolerance holds."""
import pytest
import torch

from oracle import mx_oracle as O

pytestmark = pytest.mark.gpu
COS_MIN, REL_L2_MAX = 0.9999, 1e-2


def _operands(q, k, v):
    import mpsa
    from mpsa import ops
    D = q.shape[-1]
    qq = mpsa.quantize_mx(ops._pad_depth_128(q.cuda()), ops.q_side_scale(D))
    kq = mpsa.quantize_mx(ops._pad_depth_128(k.cuda()), 1.0)
    return qq, kq, mpsa.quantize_v_seq(v.cuda())


@pytest.mark.parametrize("shape,tau", [
    ((1, 4, 2, 1024, 128), 1.02),      # a good share of promoted tiles
    ((1, 4, 2, 1024, 128), 1e9),       # none promoted: nothing is appended to any row's visit list
    ((1, 4, 2, 1024, 128), 0.5),       # every tile promoted, the row's first one included: every MXFP4 tile is done twice
    ((2, 2, 1, 333, 128), 1.0),        # ragged length, two batches
    ((1, 8, 8, 640, 64), 1.05),        # head_dim 64
])
def test_router_inside_the_forward_equals_the_stand_alone_router(shape, tau):
    import mpsa
    from mpsa import ops
    B, Hq, Hkv, S, D = shape
    q, k, v = O.make_qkv(11, B, Hq, Hkv, S, D, outliers=4)
    qq, kq, vq = _operands(q, k, v)
    stat = mpsa.router_statistic(qq, kq, B, Hq, Hkv, S, S, causal=True, check=True)
    pm_ref = mpsa.precision_map_online(stat, S, S, causal=True, band=1, tau=tau)
    out_ref, lse_ref = ops.attention_forward_quantized(qq, kq, vq, B, Hq, Hkv, S, S, D, causal=True, prec_map=pm_ref,
                                                       out_dtype=torch.float32, check=True, return_lse=True)
    out, pm, lse = ops.attention_forward_routed(qq, kq, vq, B, Hq, Hkv, S, S, D, band=1, tau=tau, out_dtype=torch.float32,
                                                check=True, return_map=True, return_lse=True)
    assert int(ops._last_range_flag.item()) == 0
    assert torch.equal(pm, pm_ref), (int((pm != pm_ref).sum()), pm.unique().tolist())
    n_promoted = int(((pm == mpsa.TILE_FP8) & (mpsa.precision_map_band(S, S, True, 1, 128, pm.device) == mpsa.TILE_FP4)).sum())
    if tau == 1e9:
        assert n_promoted == 0
    if tau == 0.5:
        assert int((pm == mpsa.TILE_FP4).sum()) == 0
    m = O.parity_metrics(out.cpu(), out_ref.cpu())
    assert m["rel_l2"] <= 1e-5, (m, n_promoted)                # two passes merged vs one pass: fp32 rounding only
    assert torch.allclose(lse.cpu(), lse_ref.cpu(), rtol=1e-5, atol=1e-4)
    ref = O.attention_mxfp(q, k, v, causal=True, prec_map=pm.cpu(), pv_mode="requant")
    m = O.parity_metrics(out.cpu(), ref)
    assert m["cos"] >= COS_MIN and m["rel_l2"] <= REL_L2_MAX, m


def test_one_call_form_uses_the_router_inside_and_matches_the_stand_alone_form():
    import mpsa
    q, k, v = (t.cuda() for t in O.make_qkv(2, 1, 8, 2, 2048, 128, outliers=5))
    kw = dict(causal=True, pv_mode="requant", router="online", tau=1.05, check=True)
    a = mpsa.attention_forward(q, k, v, out_dtype=torch.bfloat16, **kw)
    b = mpsa.attention_forward(q, k, v, out_dtype=torch.bfloat16, fused_router=False, **kw)
    m = O.parity_metrics(a.float().cpu(), b.float().cpu())
    assert m["rel_l2"] <= 4e-3, m          # bf16 outputs of two different accumulation orders


def test_items_done_again_when_scores_leave_the_fixed_reference():
    """Row maxima beyond the window of the row reference: the forward does those items again over the map that its first pass left, and
    says so; the result still matches the oracle, and the map is the one the stand-alone router gives."""
    import mpsa
    from mpsa import ops
    q, k, v = O.make_qkv(9, 1, 4, 2, 1024, 128, outliers=3)
    k2 = k.clone().float()
    k2[:, :, 128:] *= 60.0
    k2 = k2.to(torch.bfloat16)
    qq, kq, vq = _operands(q, k2, v)
    out, pm = ops.attention_forward_routed(qq, kq, vq, 1, 4, 2, 1024, 1024, 128, band=1, tau=1.1, out_dtype=torch.float32,
                                           check=True, return_map=True)
    assert int(ops._last_range_flag.item()) == 1
    assert set(pm.unique().tolist()) <= {0, 1, 2}
    stat = ops.router_statistic(qq, kq, 1, 4, 2, 1024, 1024, causal=True, check=True)
    assert torch.equal(pm, ops.precision_map_online(stat, 1024, 1024, causal=True, band=1, tau=1.1))
    ref = O.attention_mxfp(q, k2, v, causal=True, prec_map=pm.cpu(), pv_mode="requant")
    m = O.parity_metrics(out.cpu(), ref)
    assert m["cos"] >= COS_MIN and m["rel_l2"] <= REL_L2_MAX, m


def test_promoted_tiles_whose_mxfp4_scores_lie_far_above():
    """Queries a hundred times as large against keys with outlier channels: the MXFP4 scores of promoted tiles exceed the MXFP8 ones that
    replace them by more octaves than a reference serves.  Every row stays finite and equals the forward over the router's own map,
    whose references are exact; bound: P in the tile's format, both in fp32."""
    import mpsa
    from mpsa import ops
    B, Hq, Hkv, S, D = 2, 20, 5, 1332, 128
    g = torch.Generator("cuda").manual_seed(579)
    q, k, v = (torch.randn(B, h, S, D, generator=g, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    k[..., :5] *= 20
    q[:, :, ::3] *= 100
    for turn in range(3):
        k = k.roll(7 * turn, dims=2)
        out = mpsa.attention_forward(q, k, v, causal=True, pv_mode="requant", router="online", tau=1.1, out_dtype=torch.float32, check=True)
        assert bool(torch.isfinite(out).all())
        qq, kq = mpsa.quantize_mx(q, ops.q_side_scale(D)), mpsa.quantize_mx(k, 1.0)
        stat = mpsa.router_statistic(qq, kq, B, Hq, Hkv, S, S, causal=True, check=True)
        pm = mpsa.precision_map_online(stat, S, S, causal=True, band=1, tau=1.1)
        ref = mpsa.attention_forward(q, k, v, causal=True, pv_mode="requant", prec_map=pm, out_dtype=torch.float32, check=True)
        assert float((out - ref).norm() / ref.norm()) < 1e-5


@pytest.mark.parametrize("S", [300, 512])
def test_promoted_tiles_whose_mxfp4_scores_lie_far_below(S):
    """The other side: MXFP4 scores of promoted tiles inside the range that one reference serves, MXFP8 scores that replace them and all
    the others far below it.  Key elements next to a block's large one are zero in MXFP4 (1/16 and 5/64 of its scale) and exact in
    MXFP8, and the queries are zero where the large one stands: every MXFP4 score is 0, the others are about -175."""
    import mpsa
    from mpsa import ops
    B, Hq, Hkv, D = 1, 2, 1, 128
    g = torch.Generator("cuda").manual_seed(S)
    q = torch.full((B, Hq, S, D), 1.25 / ops.q_side_scale(D), device="cuda", dtype=torch.bfloat16)
    k = -1.0 - 0.25 * torch.randint(0, 2, (B, Hkv, S, D), generator=g, device="cuda").to(torch.bfloat16)
    q[..., ::32], k[..., ::32] = 0.0, 128.0
    v = torch.randn(B, Hkv, S, D, generator=g, device="cuda", dtype=torch.bfloat16)
    qq, kq = mpsa.quantize_mx(q, ops.q_side_scale(D)), mpsa.quantize_mx(k, 1.0)
    stat = mpsa.router_statistic(qq, kq, B, Hq, Hkv, S, S, causal=True, check=True)
    assert float(stat.abs().max()) == 0.0
    pm = mpsa.precision_map_online(stat, S, S, causal=True, band=1, tau=1.1)
    assert bool((pm != ops.TILE_FP4).all())
    out = mpsa.attention_forward(q, k, v, causal=True, pv_mode="requant", router="online", tau=1.1, out_dtype=torch.float32, check=True)
    ref = mpsa.attention_forward(q, k, v, causal=True, pv_mode="requant", prec_map=pm, out_dtype=torch.float32, check=True)
    assert float(ref.norm(dim=-1).min()) > 0.0
    assert float((out - ref).norm() / ref.norm()) < 1e-5

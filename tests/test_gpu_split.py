"""The forward with an item's keys divided among CTAs, against the undivided forward on the same quantised operands: grids
with fewer query tiles than SMs, and with a last wave that is nearly empty."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,Skv,Hq,Hkv,D,causal,pv_mode,gain", [
    (16, 2048, 32, 8, 128, True, "requant", 1.0),       # two runs of a row, 16 rows of a tile in use
    (1, 16300, 3, 1, 128, True, "requant", 1.0),        # one row, a ragged last key tile, most runs inside one item
    (900, 1300, 4, 2, 128, True, "fp16", 1.0),          # three parts with a CTA each, the last one empty for the shorter rows
    (130, 20000, 8, 2, 64, True, "fp16", 1.0),          # two query tiles of different length, depth 64
    (1560, 1560, 12, 12, 128, False, "requant", 1.0),   # 156 items on 148 SMs
    (700, 9000, 16, 4, 128, False, "fp16", 1.0),
    (300, 9000, 8, 8, 128, True, "requant", 60.0),      # row maxima outside the reference's window: shares done again
    (300, 9000, 8, 8, 128, True, "fp16", 60.0),
])
def test_divided_keys(S, Skv, Hq, Hkv, D, causal, pv_mode, gain):
    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(S + Skv)
    q, k, v = (torch.randn(1, h, n, D, generator=g, device="cuda", dtype=torch.bfloat16) for h, n in ((Hq, S), (Hkv, Skv), (Hkv, Skv)))
    q[:, :, ::7] *= gain
    kv = mpsa.prepare_kv(k, v, pv_mode=pv_mode)
    qq = mpsa.quantize_qk(ops._pad_depth_128(q), ops.q_side_scale(D))
    for out_dtype in (torch.float32, torch.bfloat16):
        out = mpsa.attention_forward(q, k, v, causal=causal, pv_mode=pv_mode, out_dtype=out_dtype, check=True).float()
        kept = mpsa.attention_forward(q, None, None, causal=causal, kv=kv, out_dtype=out_dtype, check=True).float()
        ref = mpsa.attention_forward_quantized(qq, *kv, 1, Hq, Hkv, S, Skv, D, causal=causal, out_dtype=torch.float32, check=True)
        assert torch.equal(out, kept)
        rel = float((out - ref).norm() / ref.norm())
        assert rel <= (4e-3 if out_dtype is torch.bfloat16 else (1e-5 if pv_mode == "requant" and gain == 1.0 else 1e-3)), rel

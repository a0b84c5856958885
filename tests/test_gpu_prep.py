"""Operand preparation in one launch: codes from 16-bit patterns against the oracle on every magnitude a block can hold, the
one-call attention against the separate steps, and the NVFP4 quantizer next to its rounding boundaries."""
import pytest
import torch

from oracle import mx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scale", [1.0, 128 ** -0.5 * 1.4426950408889634, 0.0371, 96.5])
def test_codes_of_every_pattern(dtype, scale):
    """Rows of 64 / 128 / 256 depth elements: each 32-element block holds its largest element, then patterns from that down
    to far below the last code boundary, both zeros and both signs.  Row counts end inside a tile."""
    import mpsa
    step = 128 if dtype is torch.bfloat16 else 1024
    top = torch.arange(0, step, 1 if step == 128 else 37)                    # mantissa of the block's largest element
    one = 0x3f80 if dtype is torch.bfloat16 else 0x3c00
    blocks = []
    for t in top.tolist():
        below = torch.arange(one + t, one + t - 6 * step, -5 if step == 128 else -41)
        for part in below.split(29):
            b = torch.zeros(32, dtype=torch.int32)
            b[0], b[1], b[2] = one + t, 0x8000, 0
            b[3:3 + part.numel()] = part
            b[3::2] |= 0x8000
            blocks.append(b)
    x = torch.stack(blocks).to(torch.int16).view(dtype)
    x = x * (2.0 ** (torch.arange(len(blocks)) % 9 - 4)).to(dtype)[:, None]
    for D in (64, 128, 256):
        n = x.numel() // D // 3 * 3
        y = x.reshape(-1)[:n * D].view(1, 3, n // 3, D)
        r = mpsa.quantize_mx(y.cuda(), scale, reference_format=True)
        c4, s4 = O.quant_mxfp4_side(y, scale)
        c8, s8 = O.quant_mxfp8_side(y, scale)
        assert torch.equal(r.fp4_unpacked.cpu(), c4) and torch.equal(r.fp4_scales.cpu(), s4), (D, "E2M1")
        assert torch.equal(r.fp8.cpu(), c8) and torch.equal(r.fp8_scales.cpu(), s8), (D, "E5M2")
        assert torch.equal(r.fp4.cpu(), O.pack_e2m1(c4))


@pytest.mark.parametrize("S,Skv,D,layout,causal,dtype,kw", [
    (1, 1, 128, "HND", True, torch.bfloat16, dict(pv_mode="requant")),
    (129, 129, 64, "NHD", True, torch.float16, dict(pv_mode="fp16")),
    (300, 700, 128, "NHD", False, torch.bfloat16, dict(pv_mode="requant", smooth_k=True)),
    (257, 257, 64, "HND", False, torch.float16, dict(pv_mode="fp16", smooth_k=True, uniform="fp4")),
    (640, 640, 128, "HND", False, torch.bfloat16, dict(pv_mode="fp16", uniform="fp8", fp8_elem="e4m3")),
    (2500, 2500, 128, "HND", True, torch.bfloat16, dict(pv_mode="requant", router="online", tau=1.1)),   # 320 items: several per CTA
    (333, 333, 128, "HND", False, torch.bfloat16, dict(pv_mode="fp16", fp4_kind="nvfp4")),
    (2500, 2500, 128, "NHD", False, torch.float16, dict(pv_mode="requant", fp4_kind="nvfp4")),
])
def test_one_call_against_separate_steps(monkeypatch, S, Skv, D, layout, causal, dtype, kw):
    """attention_forward through its one C call and through the separate quantizers, V preparation, map and forward, as for
    operands that the one call does not take."""
    import mpsa
    B, Hq, Hkv = 1, 16, 8
    g = torch.Generator(device="cuda").manual_seed(S)
    def operand(H, L):
        t = torch.randn(*((B, H, L, D) if layout == "HND" else (B, L, H, D)), generator=g, device="cuda", dtype=dtype)
        return t if layout == "HND" else t.transpose(1, 2)
    q, k, v = operand(Hq, S), operand(Hkv, Skv), operand(Hkv, Skv)
    a = mpsa.attention_forward(q, k, v, causal=causal, out_dtype=torch.float32, check=True, **kw)
    monkeypatch.setattr(mpsa.ops, "_attention_one_call", lambda *a, **kw: None)
    b = mpsa.attention_forward(q, k, v, causal=causal, out_dtype=torch.float32, check=True, **kw)
    assert float((a - b).norm()) <= 1e-6 * float(b.norm())


@pytest.mark.parametrize("rows,D", [(1, 64), (200, 128), (131, 192)])
def test_nvfp4_next_to_code_boundaries(rows, D):
    """Elements on, and one or two fp32 steps around, the places where the E2M1 code changes."""
    import mpsa
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, D // 16, 16, generator=g)
    amax = x.abs().amax(-1, keepdim=True)
    for _ in range(2):                                   # the block scales depend on the block maxima only
        x[..., 0:1] = amax * 3.0
        _, sc, tsq = O.quant_nvfp4(x.view(rows, D))
        scf = (O.decode_e4m3(sc).float() * float(tsq)).view(rows, D // 16, 1)
        edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 0.5, 1.0, 2.0, 3.0, 4.0])
        near = (scf * edges).clone()
        ulps = torch.randint(-2, 3, near.shape, generator=g, dtype=torch.int32)
        x[..., 1:13] = (near.view(torch.int32) + ulps).view(torch.float32) * torch.where(torch.rand(near.shape, generator=g) < 0.5, -1.0, 1.0)
    x = x.view(rows, D)
    codes, scales, ts = mpsa.quantize_nvfp4(x.cuda())
    oc, osc, ots = O.quant_nvfp4(x)
    assert float(ts.cpu()) == float(ots) and torch.equal(codes.cpu(), O.pack_e2m1(oc))
    exp = O.swizzle_scales(osc, pad_code=0)
    assert torch.equal(scales.cpu().reshape(exp.shape), exp)

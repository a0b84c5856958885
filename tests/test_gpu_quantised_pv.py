"""Quantised P.V: log2 denominators against 64-bit arithmetic on the same quantised operands, over both formats of the score tiles,
ragged and masked tiles, and scores inside and outside the window of row maxima that one reference serves."""
import pytest
import torch

pytestmark = pytest.mark.gpu

E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _values(r, fmt):
    """What the codes of a QuantizedOperand (reference format) stand for, in 64 bits."""
    if fmt == "fp8":
        codes, scales = r.fp8.view(torch.float8_e5m2).double(), r.fp8_scales
    else:
        c = r.fp4_unpacked.long()
        codes = torch.tensor(E2M1, device=c.device, dtype=torch.float64)[c & 7] * torch.where(c & 8 > 0, -1.0, 1.0)
        scales = r.fp4_scales
    return codes * torch.exp2(scales.double() - 127.0).repeat_interleave(32, -1)


@pytest.mark.parametrize("fmt", ["fp8", "fp4"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S, Skv", [(1, 1), (1, 31), (127, 129), (128, 256), (257, 257), (40, 1000)])
@pytest.mark.parametrize("shift", [0.0, 60.0, -40.0, 110.0, -75.0])
def test_denominators(fmt, causal, S, Skv, shift):
    """Every score is moved by about `shift` octaves; row maxima beyond [-44, 84] make an item be done again.  Bound: a score is a
    sum in fp32 of up to four truncated additions, and a reference comes off it (five units in the last place of the largest);
    ex2 and the sums add 2^-20."""
    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(S * 1000 + Skv)
    q, k, v = (torch.randn(1, 2, n, 128, generator=g, device="cuda") for n in (S, Skv, Skv))
    q[..., 0], k[..., 0] = 4.0 / ops.q_side_scale(128), shift / 4.0
    qq = mpsa.quantize_mx(q, ops.q_side_scale(128), reference_format=True)
    kq = mpsa.quantize_mx(k, 1.0, reference_format=True)
    out, lse = ops.attention_forward_quantized(qq, kq, mpsa.quantize_v_seq(v), 1, 2, 2, S, Skv, 128, causal=causal, uniform=fmt,
                                               out_dtype=torch.float32, check=True, return_lse=True)
    s = _values(qq, fmt) @ _values(kq, fmt).transpose(-1, -2)
    if causal:
        s = s.masked_fill(torch.ones(S, Skv, dtype=torch.bool, device="cuda").triu(Skv - S + 1), float("-inf"))
    m = s.amax(-1, keepdim=True)
    ref = (m + torch.log2(torch.exp2(s - m).sum(-1, keepdim=True))).squeeze(-1)
    bound = 5 * 2.0 ** -23 * float(s[s > float("-inf")].abs().max()) + 2.0 ** -20
    err = float((lse.double() - ref).abs().max())
    assert err <= bound, (err, bound)
    assert bool(torch.isfinite(out).all())


@pytest.mark.parametrize("pv", ["fp16", "requant"])
def test_a_key_whose_scores_are_nan_spoils_its_rows_wherever_it_lies(pv):
    """Scores of a key whose scale codes are NaN, at every place of a 32-key block (the exponentials of some places are formed in another
    way): no row that sees it may come out as if the key were not there.  Rows are spoilt by not being finite or by vanishing."""
    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(1, 1, n, 128, generator=g, device="cuda") for n in (128, 256, 256))
    qq, kq = mpsa.quantize_mx(q, ops.q_side_scale(128)), mpsa.quantize_mx(k, 1.0)
    vt = mpsa.quantize_v_seq(v) if pv == "requant" else mpsa.prepare_vt(v)
    whole = kq.fp4_sf.clone()

    def call():
        return ops.attention_forward_quantized(qq, kq, vt, 1, 1, 1, 128, 256, 128, causal=False, uniform="fp4", out_dtype=torch.float32, check=True)

    usual = call().norm(dim=-1)
    assert bool(torch.isfinite(usual).all()) and float(usual.min()) > 0.1
    for place in range(32):
        kq.fp4_sf.copy_(whole)
        kq.fp4_sf[0, 0, 1, 0, place * 16:place * 16 + 4] = 255       # key 128 + place: its four blocks
        norm = call().norm(dim=-1)
        assert bool((~torch.isfinite(norm) | (norm < 1e-12 * usual)).all()), place

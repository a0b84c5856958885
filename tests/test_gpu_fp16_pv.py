"""fp16 P.V at the ends of what its row reference has to serve, against 64-bit arithmetic on the same quantised operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(scores, D=128):
    """Q and K whose score of every query against key j is scores[j] octaves, exactly: one depth element carries it, as a product
    of powers of two and small integers that MXFP8 holds (|scores[j]| = n / 8 up to 60, n with three significant bits)."""
    import mpsa
    from mpsa import ops
    n = scores.numel()
    q = torch.zeros(1, 1, 128, D, device="cuda")
    q[..., 0] = 1.0 / ops.q_side_scale(D)                 # the quantizer folds the scale in: 1.0 after it
    k = torch.zeros(1, 1, n, D, device="cuda")
    k[0, 0, :, 0] = scores.to("cuda")
    return mpsa.quantize_mx(q, ops.q_side_scale(D), reference_format=True), mpsa.quantize_mx(k, 1.0, reference_format=True)


def _mx8(r):
    return r.fp8.view(torch.float8_e5m2).double() * torch.exp2(r.fp8_scales.double() - 127.0).repeat_interleave(32, -1)


def _run(qq, kq, v, **kw):
    import mpsa
    from mpsa import ops
    n = kq.fp8.shape[2]
    return ops.attention_forward_quantized(qq, kq, mpsa.prepare_vt(v), 1, 1, 1, 128, n, v.shape[-1], causal=False, uniform="fp8",
                                           out_dtype=torch.float32, check=True, return_lse=True, **kw)


def test_row_sums_have_the_precision_of_the_exponential():
    """All weight on keys 28 .. 31 of every 32: the log2 denominators are those of exponentials good to 2^-22 (ex2.approx), at every
    place of a block.  Bound: 2^-22 relative in the sum, 1.44 times that in its logarithm, and fp32 rounding of a number near 5."""
    n = 256
    scores = torch.full((n,), -48.0)
    scores[torch.arange(n) % 32 >= 28] = 0.0
    qq, kq = _operands(scores)
    out, lse = _run(qq, kq, torch.ones(1, 1, n, 128, device="cuda", dtype=torch.float16))
    s = (_mx8(qq) @ _mx8(kq).transpose(-1, -2))
    ref = torch.log2(torch.exp2(s).sum(-1))
    err = float((lse.double() - ref).abs().max())
    assert err <= 1.45 * 2.0 ** -22 + 2.0 ** -21, err

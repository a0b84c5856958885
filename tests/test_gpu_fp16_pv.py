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


def _reference(q, k, v, visible):
    """Attention in 64 bits: scores in octaves from the quantised operands, P to a row's maximum, V in fp16.  Returns the output, the
    log2 denominators, and bounds on the errors of both.  A score's products are added in fp32 by four instructions that may
    truncate, and the reference is taken off: five units in the last place of the largest.  P is rounded to 11 bits: half a step of
    2^-10 for every key, once for P and once for what the sum has of it; below 2^-14 of the largest half a step of 2^-24."""
    s = (q @ k.transpose(-1, -2)).masked_fill(~visible, float("-inf"))
    m = s.amax(-1, keepdim=True)
    m = torch.where(m == float("-inf"), torch.zeros_like(m), m)
    p = torch.exp2(s - m)
    den = p.sum(-1, keepdim=True)
    vd = v.to(torch.float16).double()
    safe = torch.where(den > 0, den, torch.ones_like(den))
    out = torch.where(den > 0, p @ vd / safe, torch.zeros_like(p @ vd))
    n = visible.double().sum(-1, keepdim=True)
    s_err = 5 * 2.0 ** -23 * float(s[s > float("-inf")].abs().max()) + 2.0 ** -20       # in octaves; 2^-20: ex2, the sums
    bound = (2.0 ** -10 + 2 * s_err) * (p @ vd.abs()) / safe + n * 2.0 ** -25 / safe * float(vd.abs().max())
    lse = (m + torch.log2(den)).squeeze(-1)
    return out, lse, bound, s_err


def _shifted(S, Skv, D, H, octaves, how, seed):
    """q and k whose scores are noise of one octave plus a row's rate (1, 1/2 or 0) times a shift of the key that reaches `octaves`."""
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(1, H, S, D, generator=g, device="cuda") * 2.0
    k = torch.randn(1, H, Skv, D, generator=g, device="cuda") * 0.5
    v = torch.randn(1, H, Skv, D, generator=g, device="cuda")
    j = torch.arange(Skv, device="cuda", dtype=torch.float32)
    shift = {"steady": octaves * j / Skv, "steps": octaves * (j // 64) / max(1, Skv // 64), "late": octaves * (j >= Skv - 70).float(),
             "early": octaves * (j < 5).float(), "once": octaves * (j == Skv // 2).float()}[how]
    q[..., 0] = torch.tensor([1.0, 0.5, 0.0], device="cuda")[torch.arange(S, device="cuda") % 3] / ops.q_side_scale(D)
    k[..., 0] = shift
    return q.to(torch.bfloat16), k.to(torch.bfloat16), v.to(torch.bfloat16)


@pytest.mark.parametrize("how", ["steady", "steps", "late", "early", "once"])
@pytest.mark.parametrize("octaves", [0, 8, 16, 40, 300])
@pytest.mark.parametrize("S,Skv,D,causal", [(128, 128, 128, False), (100, 300, 64, True), (200, 1300, 128, True), (384, 4000, 128, False)])
def test_rows_whose_maximum_grows(S, Skv, D, causal, octaves, how):
    """Row maxima that move by 0 .. 300 octaves over the keys, at another place for every third row: steadily, from half tile to half
    tile, in the last tile, in the first keys, in one key.  Whole items (one CTA each) and divided ones."""
    import mpsa
    from mpsa import ops
    H = 2
    q, k, v = _shifted(S, Skv, D, H, octaves, how, S + Skv)
    sq = ops.q_side_scale(D)
    qr, kr = (mpsa.quantize_mx(ops._pad_depth_128(x), s, reference_format=True) for x, s in ((q, sq), (k, 1.0)))
    rows, keys = torch.arange(S, device="cuda"), torch.arange(Skv, device="cuda")
    visible = (keys[None, :] <= rows[:, None] + (Skv - S)) if causal else torch.ones(S, Skv, dtype=torch.bool, device="cuda")
    ref, lse_ref, bound, s_err = _reference(_mx8(qr), _mx8(kr), v, visible)
    whole, lse = ops.attention_forward_quantized(qr, kr, mpsa.prepare_vt(v), 1, H, H, S, Skv, D, causal=causal, uniform="fp8",
                                                 out_dtype=torch.float32, check=True, return_lse=True)
    call = mpsa.attention_forward(q, k, v, causal=causal, uniform="fp8", out_dtype=torch.float32, check=True)
    for out in (whole, call):
        assert bool(((out.double() - ref).abs() <= bound).all()), float(((out.double() - ref).abs() / bound).max())
    assert float((lse.double() - lse_ref).abs().max()) <= s_err


def test_weights_far_below_the_largest_keep_their_precision():
    """A first tile whose scores spread over ten octaves, then many equal keys 9.4 octaves below the maximum, which carry the row: a
    reference above the maximum would leave them to fp16's subnormal numbers (errors of 2^-9 here)."""
    n = 4096
    scores = torch.full((n,), -9.5)
    scores[:128] = torch.where(torch.arange(128) % 2 == 0, 0.0, -10.0)
    qq, kq = _operands(scores)
    v = torch.ones(1, 1, n, 128, device="cuda", dtype=torch.float16)
    out, _ = _run(qq, kq, v)
    assert float((out - 1.0).abs().max()) <= 2.0 ** -11


def test_rows_without_a_visible_key_and_maps_that_skip():
    """A map that leaves out the first key tile: rows that see no other key come out as zeros with an empty denominator."""
    import mpsa
    from mpsa import ops
    S, Skv, D, H = 130, 700, 128, 2
    q, k, v = _shifted(S, Skv, D, H, 40, "steps", 3)
    qr, kr = (mpsa.quantize_mx(x, s, reference_format=True) for x, s in ((q, ops.q_side_scale(D)), (k, 1.0)))
    vt = mpsa.prepare_vt(v)
    for keep in ([5], [2, 5], [4, 5], [0, 3]):
        pm = torch.zeros(2, 6, dtype=torch.uint8, device="cuda")
        pm[:, keep] = mpsa.TILE_FP8
        rows, keys = torch.arange(S, device="cuda"), torch.arange(Skv, device="cuda")
        visible = (keys[None, :] <= rows[:, None] + (Skv - S)) & torch.isin(keys // 128, torch.tensor(keep, device="cuda"))[None, :]
        ref, lse_ref, bound, s_err = _reference(_mx8(qr), _mx8(kr), v, visible)
        out, lse = ops.attention_forward_quantized(qr, kr, vt, 1, H, H, S, Skv, D, causal=True, prec_map=pm, out_dtype=torch.float32,
                                                   check=True, return_lse=True)
        assert bool(((out.double() - ref).abs() <= bound).all()), keep
        empty = ~visible.any(-1)
        assert bool((out[:, :, empty] == 0).all()) and bool((lse[:, :, empty] == float("-inf")).all())
        assert float((lse.double() - lse_ref)[:, :, ~empty].abs().max()) <= s_err


@pytest.mark.parametrize("S,D", [(333, 128), (1024, 64), (4096, 128)])
@pytest.mark.parametrize("outliers", [0, 5])
def test_error_is_that_of_rounding_p(S, D, outliers):
    """The error against 64 bits over whole outputs is that of rounding each P to 11 bits: with steps of 2^-10 / m for mantissas m that
    are spread over the logarithm, the root mean square of step / sqrt(12) is 2^-10 sqrt(0.541 / 12) = 2.07e-4; it comes out smaller
    where few keys carry a row.  Bound: 2^-12, 1.18 times that."""
    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(1, 2, S, D, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    if outliers:
        k[..., torch.randperm(D, generator=g, device="cuda")[:outliers]] *= 20.0
    out = mpsa.attention_forward(q, k, v, causal=False, uniform="fp8", out_dtype=torch.float32, check=True)
    qr, kr = (mpsa.quantize_mx(ops._pad_depth_128(x), s, reference_format=True) for x, s in ((q, ops.q_side_scale(D)), (k, 1.0)))
    ref = _reference(_mx8(qr), _mx8(kr), v, torch.ones(S, S, dtype=torch.bool, device="cuda"))[0]
    assert float((out.double() - ref).norm() / ref.norm()) <= 2.0 ** -12


@pytest.mark.parametrize("how", ["steps", "steady"])
def test_two_runs_are_the_same_bits(how):
    """Half tiles decide on the references in their order whatever their timing, so a problem with many raises repeats itself exactly,
    next to other work on the GPU too."""
    import mpsa
    q, k, v = _shifted(1500, 3000, 128, 8, 70, how, 11)
    kw = dict(causal=True, out_dtype=torch.float32, check=True)
    first = mpsa.attention_forward(q, k, v, **kw)
    side, busy = torch.cuda.Stream(), torch.randn(4096, 4096, device="cuda")
    for _ in range(5):
        with torch.cuda.stream(side):
            busy @ busy
        assert torch.equal(first, mpsa.attention_forward(q, k, v, **kw))
    torch.cuda.synchronize()

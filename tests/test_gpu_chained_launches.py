"""Calls back to back on a stream, each reading what the one before wrote into memory that is reused all the time: launches that
overlap their predecessor's tail must give what calls one at a time give, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _unit(x):
    """x at root mean square 1, so that a chain of any length stays in range."""
    return (x.float() / x.float().square().mean().sqrt()).to(x.dtype)


def _chain(q, k, v, wait, steps):
    """Outputs of every step, by name.  Where no torch operation lies between two calls, the second one's first launch overlaps the
    kernel that writes its operands."""
    import mpsa
    from ours.block_scaled_matmul import block_scaled_matmul
    from ours.quant_mxint8 import quant_mxfp4
    out = []
    for i in range(steps):
        for kw in (dict(causal=True), dict(causal=False, pv_mode="requant", smooth_k=True), dict(causal=False, fp4_kind="nvfp4")):
            a = mpsa.attention_forward(q, k, v, out_dtype=torch.bfloat16, **kw)
            wait()
            b = mpsa.attention_forward(a, k, v, out_dtype=torch.bfloat16, **kw)     # its queries straight from the call before
            wait()
            q = _unit(a) + 0.5 * _unit(b) + q.roll(1 + i, 2)
            wait()
        q = _unit(q)
        k = _unit(_unit(mpsa.attention_forward(k, q, v, causal=True, pv_mode="requant", router="online", tau=1.1)) + k)
        wait()
        codes = quant_mxfp4(q, k)
        wait()
        x = mpsa.quantize_mx(q.reshape(1, 1, -1, 128), want_fp4=False)
        wait()
        m = x.fp8.shape[2]
        # a product, which lets its successor start before it has stored anything, straight into quantizers, attention and a product
        y, n = x.fp8.view(m, 128).view(torch.float8_e5m2), min(m, 256)
        c = block_scaled_matmul(y, x.fp8_sf, y[:n], x.fp8_sf[:, :, :(n + 127) // 128].contiguous(), torch.float16, m, n, 128,
                                {"ELEM_PER_BYTE_A": 1, "ELEM_PER_BYTE_B": 1, "VEC_SIZE": 32, "alpha": 128 ** -0.5})
        rows = c.numel() // 512
        z = c.view(-1)[:rows * 512].view(1, 4, rows, 128)
        pair = mpsa.ops.quantize_pair(z, z, 1.0, 1.0, "e5m2")
        wait()
        o = mpsa.attention_forward(z, z, z, causal=False, smooth_k=True, out_dtype=torch.float16)
        wait()
        v = _unit(v + _unit(o)[:, :, :v.shape[2]].to(v.dtype))
        out.append(dict(q=q, k=k, v=v, c=c, o=o, codes_q=codes[0], scales_q=codes[1], codes_k=codes[2], pair=pair[0].view(torch.uint8), a=a, b=b))
    return out


@pytest.mark.parametrize("S", [130, 1024])
def test_back_to_back_equals_one_at_a_time(S):
    g = torch.Generator(device="cuda").manual_seed(S)
    t = [torch.randn(1, 4, S, 128, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    ref = _chain(*t, torch.cuda.synchronize, 6)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    got = _chain(*t, lambda: None, 6)
    with torch.cuda.stream(side):
        other = _chain(*t, lambda: None, 6)
    torch.cuda.synchronize()
    for i, step in enumerate(ref):
        for name, a in step.items():
            # operands that come late or too early would show: every value is finite and no step repeats the one before
            assert a.dtype == torch.uint8 or bool(torch.isfinite(a.float()).all()), (i, name)
            assert i == 0 or not torch.equal(a, ref[i - 1][name]), (i, name)
            for x in (got[i][name], other[i][name]):
                assert torch.equal(a.view(torch.uint8), x.view(torch.uint8)), (i, name)


def test_operands_made_on_another_stream():
    """The event between the streams comes before the launch, whatever kernel the launch overlaps on its own stream."""
    import mpsa
    g = torch.Generator(device="cuda").manual_seed(5)
    k, v, w = (torch.randn(1, 2, 512, 128, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    a = torch.randn(4096, 4096, generator=g, device="cuda")
    ref = mpsa.attention_forward(w * 3, k, v, causal=True)
    other = torch.cuda.Stream()
    q = torch.zeros_like(w)
    torch.cuda.synchronize()
    for _ in range(20):
        q.zero_()
        done = torch.cuda.Event()
        other.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(other):
            a @ a                                       # the operand comes late
            q.copy_(w).mul_(3)
            done.record()
        mpsa.attention_forward(w, k, v, causal=True)    # a launch of ours right before, on the consumer's stream
        torch.cuda.current_stream().wait_event(done)
        out = mpsa.attention_forward(q, k, v, causal=True)
        torch.cuda.synchronize()
        assert torch.equal(out, ref)

"""Calls back to back on a stream, each reading what the one before wrote into memory that is reused all the time: launches that
overlap their predecessor's tail must give what calls one at a time give, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(q, k, v, wait, steps):
    import mpsa
    from ours.block_scaled_matmul import block_scaled_matmul
    from ours.quant_mxint8 import quant_mxfp4
    out = []
    for i in range(steps):
        for kw in (dict(causal=True), dict(causal=False, pv_mode="requant", smooth_k=True), dict(causal=False, fp4_kind="nvfp4")):
            q = mpsa.attention_forward(q, k, v, out_dtype=torch.bfloat16, **kw) * (2.0 + i)
            wait()
        k = mpsa.attention_forward(k, q, v, causal=True, pv_mode="requant", router="online", tau=1.1) + k
        wait()
        codes = quant_mxfp4(q, k)
        wait()
        x = mpsa.quantize_mx(q.reshape(1, 1, -1, 128), want_fp4=False)
        wait()
        m = x.fp8.shape[2]
        c = block_scaled_matmul(x.fp8.view(m, 128).view(torch.float8_e5m2), x.fp8_sf, x.fp8[:, :, :256].reshape(256, 128).view(torch.float8_e5m2),
                                x.fp8_sf[:, :, :2].contiguous(), torch.float16, m, 256, 128,
                                {"ELEM_PER_BYTE_A": 1, "ELEM_PER_BYTE_B": 1, "VEC_SIZE": 32, "alpha": 1.0})
        wait()
        v = (v + c.reshape(v.shape[0], v.shape[1], -1)[:, :, :v.shape[2] * 128].reshape(v.shape).to(v.dtype)) * 0.5
        out += [q.clone(), k.clone(), *codes, c]
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
    for a, b, c in zip(ref, got, other):
        a, b, c = (x.view(torch.uint8) if x.dtype != torch.uint8 else x for x in (a, b, c))
        assert torch.equal(a, b) and torch.equal(a, c)


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

"""Smooth K in one launch (the CTAs of K add up their head's columns themselves) against the launch of its own that longer keys and many heads take:
the sums are formed in the same order, so the quantised keys and the output are the same bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 127, 129, 511, 512, 513])
@pytest.mark.parametrize("D, dtype", [(64, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("layout", ["HND", "NHD"])
def test_same_bits_as_the_column_sum_launch(S, D, dtype, layout):
    _compare((2, 3), S, D, dtype, layout)


@pytest.mark.parametrize("heads", [(4, 9), (4, 16)])
def test_many_heads(heads):
    """36 heads of 512 rows add up for themselves, 64 do not."""
    _compare(heads, 512, 128, torch.bfloat16, "HND")


def _compare(heads, S, D, dtype, layout):
    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(S * 7 + D)
    x = [torch.randn(*heads, S, D, generator=g, device="cuda", dtype=dtype) for _ in range(3)]
    x[1] += torch.randn(*heads, 1, D, generator=g, device="cuda", dtype=dtype) * 4
    q, k, v = x if layout == "HND" else (t.transpose(1, 2).contiguous().transpose(1, 2) for t in x)
    out = mpsa.attention_forward(q, k, v, causal=False, smooth_k=True, out_dtype=torch.float32)
    centred = (k.float() - ops.column_mean(k).unsqueeze(2)).to(dtype)
    ref = mpsa.attention_forward(q, centred, v, causal=False, out_dtype=torch.float32)
    assert torch.equal(out, ref)

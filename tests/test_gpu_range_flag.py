"""The range flag of a forward (quantised P.V: query tiles were done again) is that call's own."""
import threading

import pytest
import torch

from oracle import mx_oracle as O

pytestmark = pytest.mark.gpu


def _inputs(gain):
    q, k, v = (t.cuda() for t in O.make_qkv(9, 1, 4, 2, 512, 128, outliers=3))
    return q, (k.float() * gain).to(torch.bfloat16), v


@pytest.mark.parametrize("router", ["band", "online"])
def test_another_call_leaves_the_flag_alone(router):
    """A call that sets its flag (row maxima beyond the window), then one that does not, on another stream and on the same one: the first
    flag still says what the first call found, and the other way round."""
    import mpsa
    from mpsa import ops
    far, near = _inputs(100.0), _inputs(1.0)
    kw = dict(causal=True, pv_mode="requant", router=router, tau=1.1, check=True)
    mpsa.attention_forward(*far, **kw)
    first = ops._last_range_flag
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        mpsa.attention_forward(*near, **kw)
        second = ops._last_range_flag
    mpsa.attention_forward(*near, **kw)
    torch.cuda.synchronize()
    assert int(first.item()) == 1 and int(second.item()) == 0 and int(ops._last_range_flag.item()) == 0
    mpsa.attention_forward(*far, **kw)
    assert int(second.item()) == 0 and int(ops._last_range_flag.item()) == 1


def test_a_thread_sees_its_own_calls_only():
    import mpsa
    from mpsa import ops
    far, near = _inputs(100.0), _inputs(1.0)
    kw = dict(causal=True, pv_mode="requant", check=True)
    mpsa.attention_forward(*far, **kw)

    def other():
        mpsa.attention_forward(*near, **kw)
        seen.append(int(ops._last_range_flag.item()))
    seen = []
    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert seen == [0] and int(ops._last_range_flag.item()) == 1


def test_calls_without_the_word():
    """No word is kept without check=True, and none with fp16 P.V, whose references move instead."""
    import mpsa
    from mpsa import ops
    q, k, v = _inputs(1.0)
    for kw in (dict(pv_mode="requant"), dict(pv_mode="fp16", check=True)):
        mpsa.attention_forward(q, k, v, causal=True, **kw)
        assert ops._last_range_flag is None

"""Smooth K: where the CTAs of K add up their head's columns themselves and where a launch of its own does it once (no GPU: the partial
sums of the launch take room in the workspace)."""
import struct

import pytest

ARGS = struct.Struct("@3Q9q9Q2Qq2Q17i2f")                # mpsa_attention_args of include/mpsa.h


def _workspace(heads, rows, depth, smooth, fp8_fmt=1):
    from mpsa import _lib
    ints = (0, 0, 1, heads, heads, rows, rows, depth, 0, 0, 1, 0, 0, 0, fp8_fmt, smooth, 0)
    return _lib.load().mpsa_attention_workspace(ARGS.pack(256, 256, 256, *[0] * 9, *[0] * 9, 0, 0, 0, 0, 0, *ints, 1.0, 1.0))


@pytest.mark.parametrize("heads, rows, depth, launch", [
    (16, 333, 128, False), (64, 333, 128, False), (96, 333, 128, True), (48, 512, 128, False), (64, 512, 128, True), (256, 512, 128, True),
    (256, 256, 128, False), (64, 512, 64, False), (256, 512, 64, False), (1, 512, 128, False), (1, 513, 128, True), (1, 513, 64, True)])
def test_rule(heads, rows, depth, launch):
    """Each side where it was measured to be the faster one (the figures are beside prep_own_sums); beyond 512 rows the launch."""
    plain = _workspace(heads, rows, depth, 0)
    assert plain > 0
    assert (_workspace(heads, rows, depth, 1) > plain) == launch
    assert _workspace(heads, rows, depth, 1, fp8_fmt=0) > _workspace(heads, rows, depth, 0, fp8_fmt=0)      # E4M3: always the launch

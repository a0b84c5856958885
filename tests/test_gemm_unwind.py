"""A GEMM pair that gives up in the middle: before either CTA leaves, every copy that was requested into shared memory has landed.
The plan of csrc/drain.h runs here against a model of the kernel's barriers (phases that complete when the expected arrivals and
bytes are in), for every state that two producers can stop in; the kernel itself is checked for taking that plan and for waits
that do not look at the status word, which is set by then.  No GPU needed."""
import ctypes
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mp-sparse-attn_b200", "csrc")
BYTES = 100                                  # one CTA's share of a stage


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("drain") / "libdrain.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, os.path.join(ROOT, "tests", "host", "drain_host.cpp"), "-o", out],
                   check=True)
    return ctypes.CDLL(out)


class Barrier:
    """An mbarrier with one expected arrival per phase: a phase completes when its arrival has come and no bytes are pending.  Bytes may
    come before they are expected."""

    def __init__(self):
        self.phase, self.arrived, self.bytes = 0, False, 0

    def _check(self):
        if self.arrived and self.bytes == 0:
            self.phase, self.arrived = self.phase + 1, False

    def arm(self, n):
        assert not self.arrived, "a second arrival in one phase"
        self.arrived, self.bytes = True, self.bytes + n
        self._check()

    def land(self, n):
        self.bytes -= n
        self._check()


def _state(ring, used, n0, n1):
    """Barriers after stages 0 .. used - 1 have landed and been used, with the copies of the others still in flight, in the order in which
    they were requested; None if the two producers cannot have got that far."""
    if not (used <= n0 <= used + ring and used <= n1 <= used + ring):
        return None
    full = [Barrier() for _ in range(ring)]
    flying = []
    for u in range(max(n0, n1)):
        b = full[u % ring]
        if u < n0:
            b.arm(2 * BYTES)
        for r, n in ((0, n0), (1, n1)):
            if u < n:
                if u < used:
                    b.land(BYTES)
                else:
                    flying.append((u, r))
    return full, flying


@pytest.mark.parametrize("ring", [4, 5, 8])
def test_every_requested_copy_has_landed_before_the_pair_leaves(plan, ring):
    states = 0
    for used in range(2 * ring + 2):
        for n0 in range(used, used + ring + 1):
            for n1 in range(used, used + ring + 1):
                for order in ("as requested", "last first", "second CTA first"):
                    full, flying = _state(ring, used, n0, n1)
                    if order == "last first":
                        flying.reverse()
                    if order == "second CTA first":
                        flying.sort(key=lambda c: -c[1])
                    states += 1
                    for u in range(plan.host_drain_first(n0, n1, ring), plan.host_drain_end(n0, n1)):
                        b, step = full[u % ring], plan.host_drain_step(u, n0, n1)
                        # nothing may be done to a phase that completes, or has completed, by itself
                        assert b.phase == u // ring or (step == 0 and b.phase == u // ring + 1), (used, n0, n1, u)
                        if step == 1:
                            b.arm(BYTES)
                        elif step == 2:
                            b.land(BYTES)
                        while b.phase <= u // ring:          # the wait: copies land in some order until the phase is complete
                            assert flying, ("waits for a copy that was never requested", used, n0, n1, u)
                            v, _ = flying.pop(0)
                            full[v % ring].land(BYTES)
                    assert not flying, ("left with copies in flight", used, n0, n1, flying)
    assert states > 100


def test_counts_never_differ_by_more_than_the_ring(plan):
    """The plan looks at the last `ring` stages only; with fewer requested, at all of them."""
    assert plan.host_drain_first(3, 1, 4) == 0 and plan.host_drain_first(9, 7, 4) == 5 and plan.host_drain_end(7, 9) == 9


@pytest.mark.parametrize("name", ["gemm.cu", "attn.cu", "route.cu"])
def test_unwinding_waits_do_not_look_at_the_status_word(name):
    """A kernel unwinds because the status word is set: a wait for its own copies or tensor operations that gives up on a set word gives
    up at once.  Such waits are mbar_drain (no status word, a limit of its own), and no time is merely let pass."""
    src = open(os.path.join(CSRC, name)).read()
    common = open(os.path.join(CSRC, "common.cuh")).read()
    body = common[common.index("mbar_drain("):]
    body = body[:body.index("\n}")]
    assert "status" not in body and "kWaitLimitCycles" in body
    assert src.count("mbar_drain(") >= 3
    assert not re.search(r"while \(clock64\(\) - \w+ < \d+\) \{\}", src)

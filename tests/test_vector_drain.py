"""End of a vector-sweep item whose copies did not complete in time: every copy
still in flight is waited for before the shared memory is released, and no wait
is for a phase that its barrier has long left, which would only run out (about
a second each).  The loop's start is read from the source and played on a model
of the barriers."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rfsyn_b200" / "csrc"
SOURCE = (CSRC / "vsweep.cu").read_text()
V_NH = int(re.search(r"constexpr int V_NH = (\d+)", (CSRC / "vsweep.cuh").read_text()).group(1))
LOOP = re.search(r"for \(int g = (.+?); g < issued; g\+\+\) mbar_wait\(&bars\[g % V_NH\], \(unsigned\)\(g / V_NH\) & 1u\)",
                 SOURCE)


def _item(steps, fails_at):
    """Thread 0's counts at the end of an item of `steps` planes: the groups it
    waited for when a wait of its own ran out (at iteration fails_at; None when
    only other threads' waits did), and the groups it issued."""
    issued = min(V_NH, steps + 1)
    waited, failed = 0, False
    for n in range(steps + 1):
        if n == fails_at:
            failed, waited = True, n
        if n + V_NH <= steps and not failed:
            issued += 1
    return waited, issued


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 7, 28, 64])
def test_drain_waits_for_what_is_in_flight(steps):
    for fails_at in [None, *range(steps + 1)]:
        waited, issued = _item(steps, fails_at)
        first = eval(LOOP.group(1), {"max": max}, {"waited": waited, "issued": issued, "V_NH": V_NH})
        assert first >= 0
        in_flight = range(waited, issued) if fails_at is not None else range(0)
        assert set(in_flight) <= set(range(first, issued))
        for g in range(first, issued):
            # groups complete in order, so when g is waited for, its barrier
            # has completed its groups so far: a wait returns when it is for
            # the newest of them (or one still to come), and runs out when it
            # is for one before whose parity the barrier has taken again
            newest = max(q for q in range(issued) if q % V_NH == g % V_NH)
            assert g == newest, f"group {g} of {issued}: its barrier is at group {newest}"

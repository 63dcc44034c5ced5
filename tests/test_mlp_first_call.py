"""What a network's first training call costs beyond a later one (buffers, the
captured step) does not grow with its steps: a short call on a fresh network
is not made to pay for a graph that only long ones could repay."""
from __future__ import annotations

import time

import numpy as np
import pytest

import rfsyn_b200 as rb

pytestmark = pytest.mark.gpu


def _extra(steps, X, Y):
    """Seconds of the first call beyond the second, best of seven networks."""
    first, later = [], []
    for _ in range(7):
        net = rb.Mlp(54, 512, 4, 512, seed=3)
        try:
            net.set_data(X, Y)
            for out in (first, later):
                t = time.perf_counter()
                net.train(steps, batch=64, seed=1)
                out.append(time.perf_counter() - t)
        finally:
            net.close()
    return min(first) - min(later)


def test_first_call_cost_is_independent_of_its_steps():
    """One step is captured whatever the call's length, so the two extras
    differ by the timer's noise only; a graph of several steps on top of it
    would take the longer call's to more than twice the other's (0.8 to 2.7 ms
    for eight steps).  Bound between the two: 1.6 times and 0.2 ms."""
    r = np.random.RandomState(5)
    X = r.uniform(-1, 1, (2000, 54)).astype(np.float32)
    Y = r.uniform(-1, 1, (2000, 512)).astype(np.float32)
    _extra(2, X, Y)
    assert _extra(24, X, Y) <= 1.6 * _extra(4, X, Y) + 2e-4

"""The batch rule's tiles leave room for two CTAs on an SM, also in FP64 with
material tables, where the rows of one scene could need more than half of its
shared memory: 40 scenes of 32-90 cells an axis take no longer than by an
explicit plan of smaller CTAs, which fit twice whatever the scene."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb
from rfsyn_b200 import scenes

pytestmark = pytest.mark.gpu


def _batch(ws, plan, monkeypatch):
    if plan is None:
        monkeypatch.delenv("RFSYN_FDTD_PLAN", raising=False)
    else:
        monkeypatch.setenv("RFSYN_FDTD_PLAN", plan)
    setups = [scenes.scene_setup(w) for w in ws]
    b = rb.Batch([scenes.run_config(w) for w in ws], [s.ptr if s else None for s in setups])
    try:
        b.advance(32)
        ms = min(b.advance_timed(48) for _ in range(4))
        return ms, [b.probes(q) for q in range(len(ws))]
    finally:
        b.close()


def test_rule_keeps_two_ctas_an_sm(monkeypatch):
    """With one CTA an SM the rule's plan takes 1.34 times the explicit one's
    time; with two it is the faster of the two.  The bound lies between."""
    ws = scenes.c4(seed=3, n_scenes=40, precision=rb.FP64, n_steps=400, lo=32, hi=90, npml=8)
    ms, td = _batch(ws, None, monkeypatch)
    ref_ms, ref = _batch(ws, "160,2,32,32,5", monkeypatch)
    for q in range(len(ws)):
        assert np.array_equal(td[q], ref[q]), q
    assert ms <= 1.1 * ref_ms

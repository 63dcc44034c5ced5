"""Explicit plans of a batch's vector sweep: every width of CTA and unequal
segments for plain and slab items give the rule's results, what the plan names
is what runs, and fields it cannot honour are refused."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb
from rfsyn_b200 import scenes

pytestmark = pytest.mark.gpu


def _run(precision, plan, monkeypatch):
    if plan is None:
        monkeypatch.delenv("RFSYN_FDTD_PLAN", raising=False)
    else:
        monkeypatch.setenv("RFSYN_FDTD_PLAN", plan)
    ws = scenes.c4(seed=11, n_scenes=5, precision=precision, n_steps=40, lo=20, hi=44, npml=4)
    setups = [scenes.scene_setup(w) for w in ws]
    b = rb.Batch([scenes.run_config(w) for w in ws], [s.ptr if s else None for s in setups])
    try:
        i = b.info()
        b.advance(40)
        return (i.tile_j, i.ring_depth, i.seg_interior, i.seg_edge, i.mode), [b.probes(q) for q in range(len(ws))]
    finally:
        b.close()


@pytest.mark.parametrize("precision", [rb.FP32, rb.FP64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("plan", ["32,2,5,5,5", "64,2,3,17,5", "96,2,40,1,5", "128,2,9,9,5", "160,2,1,7,5",
                                  "192,2,16,6,5,1"])
def test_plans_agree(plan, precision, monkeypatch):
    _, want = _run(precision, None, monkeypatch)
    info, got = _run(precision, plan, monkeypatch)
    assert info == tuple(int(x) for x in plan.split(",")[:5])
    for q in range(len(want)):
        assert np.array_equal(got[q], want[q]), q


@pytest.mark.parametrize("plan", ["192,3,16,16,5", "192,2,16,0,5", "200,2,16,16,5", "224,2,16,16,5", "0,2,16,16,5",
                                  "192,2,16,16,5,2"])
def test_refuses_what_it_cannot_honour(plan, monkeypatch):
    with pytest.raises(RuntimeError, match="names no"):
        _run(rb.FP32, plan, monkeypatch)


def test_session_refuses_two_rows_with_vectors(monkeypatch):
    monkeypatch.setenv("RFSYN_FDTD_PLAN", "8,8,16,16,5,0,3")
    with pytest.raises(RuntimeError, match="two-rows"):
        rb.Sim(rb.RunConfig(20, 21, 22, 1e-3, 10, 4, precision=rb.FP32))

"""Tile and segment rule of the vector sweep: grids on both sides of its line
between small and large grids, thin in y or z, periodic in x and y, compute
every field sample bit-equal to a scalar sweep variant."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb

pytestmark = pytest.mark.gpu

# extents, precision, periodic mask, CPML cells, whether the large-grid rule
# takes them (CTAs of at most 128 threads, segments of at least 8 planes)
GRIDS = [((100, 100, 100), rb.FP32, 0, 8, False), ((112, 112, 112), rb.FP32, 0, 8, True),
         ((91, 93, 95), rb.FP64, 0, 5, True), ((96, 96, 203), rb.FP32, 3, 9, True),
         ((70, 90, 200), rb.FP32, 3, 9, False), ((300, 301, 9), rb.FP32, 0, 2, False),
         ((500, 301, 9), rb.FP32, 0, 2, True), ((300, 6, 301), rb.FP64, 0, 2, False),
         ((600, 6, 301), rb.FP64, 0, 2, True), ((12, 250, 340), rb.FP32, 0, 3, False),
         ((24, 250, 340), rb.FP32, 0, 3, True)]


def _fields(dims, precision, periodic, npml, plan, monkeypatch):
    if plan is None:
        monkeypatch.delenv("RFSYN_FDTD_PLAN", raising=False)
    else:
        monkeypatch.setenv("RFSYN_FDTD_PLAN", plan)
    c = [n // 2 for n in dims]
    sources = [dict(i=c[0], j=c[1], k=c[2]), dict(i=1, j=dims[1] - 1, k=dims[2] - 1, component=0),
               dict(i=dims[0] - 1, j=1, k=c[2], component=1)]
    sim = rb.Sim(rb.RunConfig(*dims, 1e-3, 100, npml, precision=precision, periodic=periodic, sources=sources,
                              probes=[dict(i=c[0], j=1, k=c[2])]))
    try:
        sim.advance(30)
        return sim.info(), [sim.field(q) for q in range(6)]
    finally:
        sim.close()


@pytest.mark.parametrize("dims,precision,periodic,npml,large", GRIDS, ids=str)
def test_rule_equals_scalar_sweep(dims, precision, periodic, npml, large, monkeypatch):
    info, f = _fields(dims, precision, periodic, npml, None, monkeypatch)
    assert info.tma == 5
    assert ((info.tile_j + 1) * (info.ring_depth + 1) <= 128 and info.seg_len >= 8) == large
    _, ref = _fields(dims, precision, periodic, npml, "8,4,32,16,2", monkeypatch)
    for c in range(6):
        assert np.any(ref[c]) and np.array_equal(f[c], ref[c]), c

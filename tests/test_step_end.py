"""The end of a step: every point probe's sample is the field the step left, at
probe counts around the gathering block's width, on scenes whose step graphs
link their kernels (small grids of the vector sweep) and on ones whose do not
(periodic z), and with a plane probe, which another kernel records."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb

pytestmark = pytest.mark.gpu

DIMS, STEPS = (11, 13, 18), 21


def _probes(n):
    r = np.random.RandomState(n)
    return [dict(i=int(r.randint(1, DIMS[0])), j=int(r.randint(1, DIMS[1])), k=int(r.randint(1, DIMS[2])),
                 component=int(r.randint(0, 6))) for _ in range(n)]


def _sim(n, precision, periodic, planes):
    c = [d // 2 for d in DIMS]
    src = [dict(i=c[0], j=c[1], k=c[2], component=0), dict(i=c[0] + 1, j=c[1], k=c[2], component=1),
           dict(i=c[0], j=c[1] + 1, k=c[2] + 1)]
    return rb.Sim(rb.RunConfig(*DIMS, 1e-3, STEPS, 3, precision=precision, periodic=periodic, sources=src,
                               probes=_probes(n), planes=planes))


@pytest.mark.parametrize("planes", [0, 1])
@pytest.mark.parametrize("periodic", [0, 4])
@pytest.mark.parametrize("precision", [rb.FP32, rb.FP64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 300])
def test_samples_are_the_fields(n, precision, periodic, planes):
    """No tolerance: a sample is a copy."""
    planes = [dict(axis=2, index=5, component=0)] * planes
    sim = _sim(n, precision, periodic, planes)
    try:
        assert (sim.info().tma == 5) == (periodic == 0)
        want = np.zeros((n, STEPS))
        for s in range(STEPS):
            sim.advance(1)
            f = [sim.field(c) for c in range(6)]
            for q, p in enumerate(_probes(n)):
                want[q, s] = f[p["component"]][p["i"], p["j"], p["k"]]
        assert np.array_equal(sim.probes()[:n], want) and np.any(want)
        sim.reset()
        sim.advance(STEPS)  # 16 steps of one graph, then single ones
        assert np.array_equal(sim.probes()[:n], want)
    finally:
        sim.close()

"""Batches past the vector sweep's 32-bit limits: planes of 2^29 bytes and more
run on the work-queue sweep, beside a small scene of the same batch, and give
the series of their own sessions."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb

pytestmark = pytest.mark.gpu


def _config(nx, ny, nz, precision):
    # probes around the source, which three steps reach
    c = (nx // 2, ny // 2, nz // 2)
    return rb.RunConfig(nx, ny, nz, 1e-3, 3, 0, precision=precision,
                        sources=[dict(i=c[0], j=c[1], k=c[2], component=rb.FIELD_EX)],
                        probes=[dict(i=c[0], j=c[1], k=c[2] + q, component=rb.FIELD_EX) for q in range(2)] +
                               [dict(i=c[0], j=c[1], k=c[2], component=rb.FIELD_HZ)])


@pytest.mark.parametrize("precision,dims", [(rb.FP64, (2, 8192, 8190)), (rb.FP32, (2, 16384, 8190))],
                         ids=["fp64", "fp32"])
def test_planes_past_the_vector_sweep(precision, dims, monkeypatch):
    """About 20 GB of fields; planes of 2^26 FP64 or 2^27 FP32 cells."""
    configs = [_config(9, 10, 11, precision), _config(*dims, precision)]
    try:
        batch = rb.Batch(configs)
        try:
            assert batch.info().mode != 5
            batch.advance(3)
            got = [batch.probes(s) for s in range(2)]
        finally:
            batch.close()
        rb.release_cached_memory()
        monkeypatch.setenv("RFSYN_FDTD_TUNE", "0")
        for s, rc in enumerate(configs):
            sim = rb.Sim(rc)
            try:
                assert (sim.info().tma == 5) == (s == 0)
                sim.advance(3)
                want = sim.probes()
            finally:
                sim.close()
            assert np.all(want[:, -1] != 0) and np.array_equal(got[s], want), s
    finally:
        rb.release_cached_memory()

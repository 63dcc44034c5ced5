"""Series and spectra read from a batch between advances: the device keeps a
scene's bins from one read to the next, so each read must still see the scene's
own bins and all samples recorded so far."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb

pytestmark = pytest.mark.gpu


def _config(n, freqs, precision):
    return rb.RunConfig(n, n + 1, n + 2, 1e-3, 60, 4, precision=precision, freqs=freqs,
                        sources=[dict(i=n // 2, j=n // 2, k=n // 2)],
                        probes=[dict(i=n // 2 + 1, j=n // 2, k=n // 2), dict(i=2, j=3, k=4, component=0)])


@pytest.mark.parametrize("precision,rtol", [(rb.FP64, 1e-12), (rb.FP32, 1e-5)])
def test_reads_between_advances(precision, rtol):
    """Reference: the sums over the series read back, in FP64.  FP64 runs sum
    <= 60 products of <= 1e-15 relative error each; FP32 runs sum with
    compensation products rounded twice to 2^-24."""
    bins = [np.linspace(5e9, 40e9, 7), np.linspace(8e9, 50e9, 7), np.linspace(6e9, 30e9, 33)]
    configs = [_config(12 + 3 * s, list(f), precision) for s, f in enumerate(bins)]
    batch = rb.Batch(configs, [None] * 3)
    try:
        for steps in (20, 1, 39):
            batch.advance(steps)
            done = {20: 20, 1: 21, 39: 60}[steps]
            for s, f in enumerate(bins):
                td, dt = batch.probes(s), rb.dt_of(1e-3)
                assert np.all(td[:, done:] == 0) and np.any(td[0, :done])
                t = (np.arange(done) + 1.0) * dt
                want = (td[:, None, :done] * np.exp(-2j * np.pi * f[None, :, None] * t)).sum(-1) * dt
                scale = np.abs(td[:, :done]).sum(-1)[:, None] * dt + 1e-300
                assert np.all(np.abs(batch.dft(s) - want) <= rtol * scale)
    finally:
        batch.close()

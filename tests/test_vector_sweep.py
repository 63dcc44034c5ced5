"""The vector sweep (mode 5, vsweep.cuh): FP64 probe series bit-equal to the
CPU oracle and FP32 series bit-equal to a scalar sweep variant, for tile
shapes and segment lengths at the edges of their ranges -- one row or one
vector a tile, tiles that do not divide the grid, one-plane items, extents
that are no multiple of a vector, slabs that straddle a vector, slabs that
meet in one vector, PEC walls with sources on padded planes, periodic x and
y, list cells inside a slab.

No tolerance: every sweep evaluates the same expressions in the same order."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
import rfsyn_b200 as rb
from oracle import Scene
from tests.cases import CASES, DT1, scene_run_config

pytestmark = pytest.mark.gpu

SRC = (2, 0, 1.0, 0, 12 * DT1, 4 * DT1, 0.0)


def _spread(nx, ny, nz):
    return [(i, j, k, c) for c, (i, j, k) in enumerate(
        [(1, 1, 1), (nx - 1, ny - 1, nz - 1), (nx // 2, 1, nz - 2), (2, ny // 2, 2), (nx - 2, 2, nz // 2),
         (nx // 2 + 1, ny // 2, nz // 2 + 1)])]


SCENES = {
    **{n: s for n, s in CASES.items() if not s.periodic & 4},
    # odd extents; 3- and 5-cell slabs end inside a vector
    "ragged_npml3": Scene(nx=13, ny=23, nz=41, n_steps=50, npml=3, sources=[(6, 11, 20, *SRC)],
                          probes=_spread(13, 23, 41), boxes=[(3, 9, 5, 18, 6, 33, 3.0, 0.02)], freqs=[20e9]),
    "ragged_npml5": Scene(nx=17, ny=12, nz=71, n_steps=50, npml=5, sources=[(8, 6, 35, *SRC)],
                          probes=_spread(17, 12, 71), comps=[(0, 8, 6, 34, 4.0, 0.1)], freqs=[]),
    # the low and the high z slab share a vector
    "slabs_meet": Scene(nx=14, ny=13, nz=10, n_steps=50, npml=4, sources=[(7, 6, 5, *SRC)],
                        probes=_spread(14, 13, 10)),
    # list cells inside the slabs (overrides), and a code-less scene whose
    # only list cell, the source, sits in a corner of the slabs
    "list_in_slab": Scene(nx=16, ny=16, nz=20, n_steps=50, npml=4, sources=[(8, 8, 10, *SRC)],
                          comps=[(c, i, 2, 3, 3.0, 0.05) for c in range(3) for i in (1, 2, 8, 14)] +
                                [(2, 8, 8, k, 5.0, 0.0) for k in (1, 2, 17, 18)],
                          probes=_spread(16, 16, 20)),
    "source_in_corner": Scene(nx=16, ny=15, nz=18, n_steps=40, npml=4, sources=[(2, 13, 1, *SRC)],
                              probes=_spread(16, 15, 18)),
    # periodic x and y around a z CPML; periodic y alone
    "periodic_xy": Scene(nx=9, ny=14, nz=37, n_steps=60, periodic=3, npml=5, sources=[(0, 0, 18, *SRC)],
                         probes=_spread(9, 14, 37) + [(0, 0, 9, 0), (8, 13, 20, 2)],
                         boxes=[(0, 9, 10, 14, 12, 20, 2.0, 0.0)]),
    "periodic_y": Scene(nx=15, ny=11, nz=19, n_steps=50, periodic=2, npml=4, sources=[(7, 10, 9, *SRC)],
                        probes=_spread(15, 11, 19) + [(7, 0, 9, 1)]),
}
# (rows, vectors, planes of a plain item, planes of a slab item); None: the rule
PICKS = [None, (1, 1, 1, 1), (3, 2, 5, 2), (7, 5, 2, 7), (16, 8, 64, 64), (20, 8, 3, 4)]


@pytest.fixture(scope="module")
def wants():
    return {name: oracle.run_oracle(s) for name, s in SCENES.items()}


def _run(s: Scene, precision: int, plan, monkeypatch):
    if plan is None:
        monkeypatch.delenv("RFSYN_FDTD_PLAN", raising=False)
    else:
        monkeypatch.setenv("RFSYN_FDTD_PLAN", plan)
    cs = s.to_c()
    needs = bool(s.boxes or s.comps or s.tensors or s.disp or s.spheres or s.tensor3)
    sim = rb.Sim(scene_run_config(s, precision, rb.FUSED), oracle.device_setup() if needs else None,
                 C.cast(C.pointer(cs), C.c_void_p) if needs else None)
    try:
        if plan is None or plan.split(",")[4] == "5":
            assert sim.info().tma == 5
        sim.advance(s.n_steps)
        return sim.probes(), [sim.field(c) for c in range(6)]
    finally:
        sim.close()


def _plan(pick):
    return None if pick is None else "%d,%d,%d,%d,5" % pick


@pytest.mark.parametrize("pick", PICKS, ids=str)
@pytest.mark.parametrize("name", list(SCENES))
def test_fp64_bit_exact(wants, name, pick, monkeypatch):
    td, _ = _run(SCENES[name], rb.FP64, _plan(pick), monkeypatch)
    assert np.array_equal(td, wants[name]["td"])


@pytest.mark.parametrize("pick", PICKS, ids=str)
@pytest.mark.parametrize("name", list(SCENES))
def test_fp32_equals_scalar_sweep(name, pick, monkeypatch):
    """Series and whole fields, padded samples included."""
    td, f = _run(SCENES[name], rb.FP32, _plan(pick), monkeypatch)
    ref, rf = _run(SCENES[name], rb.FP32, "8,4,32,16,2", monkeypatch)
    assert np.array_equal(td, ref)
    for c in range(6):
        assert np.array_equal(f[c], rf[c]), c


def test_refuses_periodic_z(monkeypatch):
    s = CASES["periodic_all_overrides"]
    with pytest.raises(RuntimeError, match="not periodic"):
        _run(s, rb.FP64, "8,8,32,32,5", monkeypatch)


def test_refuses_oversized_tile(monkeypatch):
    with pytest.raises(RuntimeError, match="exceeds a CTA"):
        _run(SCENES["ragged_npml3"], rb.FP64, "64,64,32,32,5", monkeypatch)

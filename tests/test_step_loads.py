"""Loads of the step kernels, read from the source: a step kernel may already be
resident while the kernel before it still writes (overlap.cuh), so nothing that
a step writes goes through the read-only path, whose data must stay constant
for the kernel's life."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rfsyn_b200" / "csrc"

# what kernels of a step write: fields, CPML and ADE state, the plane wave's
# line, series and sums, counters
WRITTEN = {"E", "H", "Eo", "Ho", "psi_e", "psi_hi", "psi_ho", "ade_s", "inc_e", "inc_h", "ts", "F", "acc", "part",
           "count", "d_step", "f"}


def _calls(text, name):
    """Arguments of every call of `name`."""
    out = []
    for m in re.finditer(r"\b%s\s*\(" % re.escape(name), text):
        depth, q = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[q], 0)
            q += 1
        out.append(text[m.end():q - 1])
    return out


@pytest.mark.parametrize("path", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_nothing_a_step_writes_is_read_as_constant(path):
    text = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    for arg in _calls(text, "__ldg"):
        first = re.match(r"\s*(?:reinterpret_cast<[^>]*>\s*\(\s*)?(?:\w+\s*\.\s*)?(\w+)", arg)
        assert first and first.group(1) not in WRITTEN, arg
    assert "ld.global.nc" not in text

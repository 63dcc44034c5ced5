"""Local arrays that device code reads or writes by wider accesses than their
elements, read from the source: each has to be declared with that alignment,
for a compiler that keeps it in memory (no optimisation, a loop not unrolled)
may place it anywhere its element type allows, and a misaligned access faults."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rfsyn_b200" / "csrc"
WIDTH = {"uint2": 8, "uint4": 16, "float2": 8, "float4": 16, "int2": 8, "int4": 16, "double2": 16, "ulonglong2": 16,
         "__nv_bfloat162": 4}
ELEMENT = {"bf16": 2, "__nv_bfloat16": 2, "float": 4, "int": 4, "unsigned": 4, "double": 8, "uint8_t": 1, "char": 1}


@pytest.mark.parametrize("path", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_local_arrays_are_aligned_for_their_accesses(path):
    text = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    for body in re.split(r"^\}", text, flags=re.M):  # one function (or type) each
        # its fixed-size arrays, with their alignment
        arrays = {}
        for m in re.finditer(r"^[ \t]+(?:(?:alignas|__align__)\((\d+)\) )?(%s) ([^;(){}]*\[\d+\][^;(){}]*);" %
                             "|".join(ELEMENT), body, re.M):
            for name in re.findall(r"(\w+)\[\d+\]", m.group(3)):
                arrays[name] = int(m.group(1) or ELEMENT[m.group(2)])
        for m in re.finditer(r"reinterpret_cast<(?:const )?(\w+) \*>\((\w+)\)", body):
            if m.group(1) in WIDTH and m.group(2) in arrays:
                assert arrays[m.group(2)] >= WIDTH[m.group(1)], m.group(0)
    # components of a vector type are not walked as an array
    assert not re.search(r"=\s*&\w+\.x\s*[;,]", text)

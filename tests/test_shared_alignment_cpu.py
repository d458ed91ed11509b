"""CPU: shared arrays that are accessed through a wider type than their own declare that alignment.

A `__shared__` array is aligned to its element type only. An access of 16 bytes to an array of a smaller type works
as long as the compiler happens to place it well and is a misaligned address (the context is lost) when another
shared variable moves it, so such an array has to say `__align__`. Read from the sources: no GPU is needed.
"""
from __future__ import annotations

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "tardiis_and_claritas_gb300", "csrc")
WIDE = {"uint4": 16, "int4": 16, "float4": 16, "double2": 16, "double4": 16, "uint2": 8, "float2": 8, "double": 8}
OWN = {"bf16": 2, "char": 1, "uint8_t": 1, "float": 4, "int": 4, "unsigned": 4, "uint32_t": 4, "double": 8, "cdx": 8}
FILES = sorted(os.path.basename(f) for e in ("*.cu", "*.cuh") for f in glob.glob(os.path.join(CSRC, e)))


def functions(text):
    """The top-level brace blocks: a shared array is known by its name within one of them."""
    depth, start, out = 0, 0, []
    body = re.sub(r"//[^\n]*", "", text)
    body = re.sub(r"namespace[\w\s]*\{|extern \"C\" \{", "", body)
    for m in re.finditer(r"[{}]", body):
        depth += 1 if m.group() == "{" else -1
        if depth <= 0:
            out.append(body[start:m.end()])
            start, depth = m.end(), 0
    return out


@pytest.mark.parametrize("name", FILES)
def test_wide_accesses_to_shared_arrays_are_aligned(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    bad = []
    for fn in functions(text):
        arrays = re.findall(r"__shared__\s+(?:__align__\((\d+)\)\s+)?(?:unsigned\s+)?(\w+)\s+(\w+)\s*\[", fn)
        for align, own, array in arrays:
            have = int(align) if align else OWN.get(own, 16)
            for wide in re.findall(r"reinterpret_cast<(?:const\s+)?(\w+)\s*\*>\(\s*&?" + array + r"\b", fn):
                if WIDE.get(wide, 1) > have:
                    bad.append((array, own, have, wide))
    assert not bad, bad

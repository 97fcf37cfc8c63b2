"""Local arrays read or written through a 16-byte vector type are declared on a 16-byte boundary, in every
translation unit (read from the source): a local array that ends up in memory -- a spill, a debug build
-- otherwise starts wherever its element type allows, and the access is misaligned."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem_taichi_gb300", "csrc")
CAST = re.compile(r"reinterpret_cast<(?:const )?(?:float4|uint4|int4|double2|ulonglong2)\s*[*&]>\(&?(\w+)\b(?!\.|->)")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_local_arrays(path):
    lines = re.sub(r"//[^\n]*", "", open(path).read()).split("\n")
    bad = []
    for k, line in enumerate(lines):
        for name in CAST.findall(line):
            # nearest declaration of an array of that name above, within the function
            for j in range(k, -1, -1):
                if re.match(r"[}_a-z]", lines[j]) and j != k and not lines[j].startswith(" "):
                    break   # top level: a parameter or a member, whose alignment the caller checks
                if re.search(r"\*\s*(?:__restrict__\s+)?" + name + r"\b", lines[j]) and j != k:
                    break   # a pointer
                d = re.search(r"^\s+(?!return)((?:alignas\(\d+\)\s+)?(?:const\s+)?[\w:]+)\s+(?:\w+(?:\[[^\]]*\])+(?:\s*=[^,;]*)?,\s*)*"
                              + name + r"\[", lines[j])
                if d:
                    if "alignas" not in lines[j] and "__shared__" not in lines[j]:
                        bad.append((k + 1, name, lines[j].strip()))
                    break
    assert not bad

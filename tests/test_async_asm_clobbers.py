"""Inline assembly that starts, commits, fences or awaits asynchronous work on memory says so to the compiler
(a "memory" clobber), in every translation unit (read from the source): the shared memory such a copy
fills is read by ordinary loads, which the compiler may otherwise move across the wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem_taichi_gb300", "csrc")
ASYNC = re.compile(r"cp\.async|fence|mbarrier\.\w*wait|tcgen05\.(?:mma|commit|wait|cp|st)")


def _statements(src):
    for m in re.finditer(r"\basm(?:\s+volatile)?\s*\(", src):
        depth = 0
        for j in range(m.end() - 1, len(src)):
            depth += (src[j] == "(") - (src[j] == ")")
            if depth == 0:
                yield src[:m.start()].count("\n") + 1, src[m.start():j + 1]
                break


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_memory_clobber(path):
    bad = [line for line, s in _statements(open(path).read())
           if ASYNC.search(s) and '"memory"' not in s and "mbarrier.init" not in s]
    assert not bad

"""Who may write the solver's `done` word, read from the source: a kernel whose grid writes it has either
had every CTA read it first (the last CTA writes, after all took their ticket), or agrees on it CTA by CTA
(step_done), or has one CTA that reads before a barrier and writes after it.  A kernel that breaks
this lets the warps of a CTA that starts late disagree on whether the solve goes on."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem_taichi_gb300", "csrc")


def _body(src, at):
    """The text of the braces that open after position `at`."""
    i = src.index("{", at)
    depth = 0
    for j in range(i, len(src)):
        depth += (src[j] == "{") - (src[j] == "}")
        if depth == 0:
            return src[i:j + 1]
    raise AssertionError("unbalanced braces")


def _kernels(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(k_\w+)\s*\(", src):
        out[m.group(1)] = _body(src, m.end())
    return src, out


@pytest.mark.parametrize("name", ["pcg.cu", "amg.cu"])
def test_writers_of_done(name):
    src, kernels = _kernels(name)
    assert kernels
    helpers = [m.group(1) for m in re.finditer(r"__device__ __forceinline__ \w+ (\w+)\(", src)
               if re.search(r"->done\s*=[^=]", _body(src, m.end()))]
    writers = 0
    for k, body in kernels.items():
        write = re.search("|".join([r"->done\s*=[^=]"] + [h + r"\(" for h in helpers]), body)
        read = re.search(r"if \(st->done\)", body)
        if not write or not (read or "step_done(" in body):
            continue
        writers += 1
        if "step_done(st)" in body[:write.start()]:
            assert not read, k
            continue
        last_cta = body.find("block_partials<")
        one_cta = re.search(k + r"<<<1, ", src) and "step_totals<" in body[read.end():write.start()]
        assert one_cta or 0 <= last_cta < write.start(), f"{k} writes done while its other warps may still read it"
    if name == "pcg.cu":
        assert writers >= 5

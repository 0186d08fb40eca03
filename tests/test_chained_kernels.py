"""Kernels that may start while the kernel in front of them still runs (they call pdl_wait) read
their inputs with ordinary loads.  A pointer that is const and __restrict__, or __ldg, lets the
compiler use read-only loads, which want the data unchanged for the kernel's whole life and are not
ordered by the wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moonshine_b200", "csrc")


def chained_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^\n]*\)\s*)?(\w+)\s*\(", text):
            body_at = text.index("{", m.end())
            end = text.index("\n}\n", body_at)
            params, body = text[m.end():body_at], text[body_at:end]
            if "pdl_wait()" in body:
                yield os.path.basename(path), m.group(1), params, body


def test_inputs_of_chained_kernels_are_read_with_ordinary_loads():
    kernels = list(chained_kernels())
    assert len(kernels) >= 20
    bad = []
    for path, name, params, body in kernels:
        for p in params.split(","):
            if "__restrict__" in p and re.search(r"\bconst\b", p):
                bad.append((path, name, " ".join(p.split())))
        if "__ldg(" in body or "ld.global.nc" in body or "ld_stream" in body:
            bad.append((path, name, "read-only load"))
    assert not bad, bad

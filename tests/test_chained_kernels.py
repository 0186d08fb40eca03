"""Kernels that may start while the kernel in front of them still runs (they call pdl_wait) read
their inputs with ordinary loads.  A pointer that is const and __restrict__, or __ldg, lets the
compiler use read-only loads, which want the data unchanged for the kernel's whole life and are not
ordered by the wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moonshine_b200", "csrc")


def functions():
    """(file, name, is a kernel, parameters, body) of every kernel and device function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"(__global__\s+void\s+(?:__launch_bounds__\([^\n]*\)\s*)?|\nK3_DEVINL\s+[\w:]+\s+)(\w+)\s*\(", text):
            body_at = text.index("{", m.end())
            line_end = text.index("\n", body_at)
            end = line_end if text[line_end - 1] == "}" else text.index("\n}\n", body_at)      # on one line, or not
            yield os.path.basename(path), m.group(2), "__global__" in m.group(1), text[m.end():body_at], text[body_at:end]


def chained_kernels():
    """The kernels that wait, themselves or in a device function they call; that function's text goes with them."""
    found = list(functions())
    waiting = {name: (params, body) for _, name, kernel, params, body in found if not kernel and "pdl_wait()" in body}
    for path, name, kernel, params, body in found:
        inner = [v for k, v in waiting.items() if re.search(r"\b%s\s*[<(]" % k, body)]
        if kernel and (inner or "pdl_wait()" in body):
            yield path, name, ",".join([params] + [p for p, _ in inner]), body + "".join(b for _, b in inner)


def test_every_wait_belongs_to_a_kernel_of_the_list():
    """A wait is in the list's kernels or in a device function that one of them calls."""
    texts = [re.sub(r"//[^\n]*", "", open(p).read()) for p in glob.glob(os.path.join(CSRC, "*.cu*"))]
    waits = sum(t.count("pdl_wait()") for t in texts) - 1                # one is its definition
    kernels = list(chained_kernels())
    own = [(n, b) for _, n, _, _, b in functions() if "pdl_wait()" in b]
    assert waits == sum(b.count("pdl_wait()") for _, b in own)
    called = "".join(b for _, _, _, b in kernels)
    names = {n for _, n, _, _ in kernels}
    assert all(n in names or re.search(r"\b%s\s*[<(]" % n, called) for n, _ in own)
    assert {"q8_few_kernel", "few_front_kernel", "exact_bf16_kernel"} <= names


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

"""The kernels that start as dependent launches overlap the kernels before
them, which write the offset records, the residual, the canvas, the change
tracking planes and the tile lists.  A read-only load (__ldg) of data that is
written while the kernel lives is undefined, so these planes may be read by
plain loads only, and a launch may be dependent only behind another kernel of
the chain.  Checked on the source: no test of results can show it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "painttween_gb300", "csrc")
# written by one kernel of the chain, read by another (p.A, p.B, p.C: the planes of load_patch)
SHARED = re.compile(r"__ldg\(\s*&?\s*(P\.(off|res|canvas|inc)\b|list\b|p\.[ABC]\b)[^;]*")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _function(text, name):
    """The body of the function `name`, to the brace that closes it at its own indentation."""
    m = re.search(r"^[^\n;]*\b%s\((?:[^;{]*)\{\n.*?^\}" % name, text, re.M | re.S)
    assert m, name
    return m.group(0)


def _reads(text):
    return [m.group(0) for m in SHARED.finditer(text)]


def test_tiled_kernels_read_shared_planes_by_plain_loads():
    assert "pdl_start();" in _text("pt_energy.cuh")
    assert _reads(_text("pt_energy.cuh")) == []


def test_helpers_of_dependent_kernels_read_shared_planes_by_plain_loads():
    for name in ("load_patch", "canvas_of"):
        assert _reads(_function(_text("pt_device.cuh"), name)) == [], name
    assert _reads(_function(_text("pt_common.cuh"), "propagate_offset")) == []
    kernel = _function(_text("pt_kernels.cu"), "k_canvas")
    assert "pdl_start();" in kernel
    assert _reads(kernel) == []


def test_only_kernels_that_wait_are_launched_dependent():
    """Every launch_dependent names a kernel that begins with pdl_start, and
    asks for the attribute only behind a launch of the chain."""
    text = {n: _text(n) for n in sorted(os.listdir(CSRC)) if n.endswith((".cu", ".cuh", ".h"))}
    calls = [(n, c) for n, t in text.items() for c in re.findall(r"return (?:pt::)?launch_dependent\((.*?);", t, re.S)]
    assert len(calls) == 4, calls
    for name, call in calls:
        m = re.match(r"dependent, (\w+)", call)
        assert m, (name, call)
        body = _function(text[name], m.group(1))
        assert body.index("pdl_start();") < body.index("P.inc"), m.group(1)
    header = text["pt_internal.h"]
    assert re.search(r"numAttrs = dependent && ", header)

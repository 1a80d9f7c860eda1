"""PTX's .aligned forms want every lane of the warp at the instruction together, which
nothing guarantees after a branch or loop that lanes leave at different times.  The
functions that hold such an instruction, and those that start a run of tensor-memory
loads, bring the warp together first."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hcore_gb300", "csrc")


def _body(name, text):
    """the body of the inline function `name`"""
    at = re.search(r"__forceinline__ void %s\([^{]*\{" % name, text)
    assert at, name
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.end():i - 1]


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("where,name,held", [
    ("hc_scalar.cuh", "cluster_sync", "barrier.cluster.arrive"),
    ("hc_tc.cuh", "tmem_alloc", "tcgen05.alloc"),
    ("hc_tc.cuh", "tmem_dealloc", "tcgen05.dealloc"),
    ("hc_digits.cuh", "combine_planes", "add_pair"),
    ("hc_dense_tc.cu", "combine4", "tmem_ld4"),
])
def test_the_warp_is_brought_together(where, name, held):
    body = _body(name, _source(where))
    assert "__syncwarp();" in body and body.index("__syncwarp();") < body.index(held)


def test_no_other_place_holds_one():
    found = {}
    for f in sorted(os.listdir(CSRC)):
        for m in re.finditer(r"barrier\.cluster\.\w+|tcgen05\.(?:alloc|dealloc|ld)\b", _source(f)):
            found.setdefault(f, set()).add(m.group())
    assert found == {"hc_scalar.cuh": {"barrier.cluster.arrive", "barrier.cluster.wait"},
                     "hc_tc.cuh": {"tcgen05.alloc", "tcgen05.dealloc", "tcgen05.ld"}}

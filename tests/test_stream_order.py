"""Set-up that writes device memory goes on the stream of the kernels that read
it. The engine's streams are non-blocking: they do not wait for the default
stream, where a fill, a device-to-device copy or the last part of a copy from
pageable memory may still be under way when the call returns. (The order
itself cannot be forced to go wrong in a run, so the sources are looked at.)"""

import os
import re

import pytest

import helpers as H

CSRC = os.path.join(H.ROOT, "d3-force-wasm_b200", "csrc")
# calls on the default stream that may return before the memory is written
UNORDERED = re.compile(r"cudaMemset\(|cudaMemcpy\((?:[^;]*?)cudaMemcpy(?:HostToDevice|DeviceToDevice)", re.S)


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def function(name, text):
    """The definition whose first line has `name(`."""
    at = re.search(r"^\w[^\n;]*\b%s\((?:[^;{]*)\{" % name, text, re.M)
    assert at, name
    return text[at.start():text.index("\n}\n", at.start())]


def test_link_plan_is_filled_on_the_stream():
    assert not UNORDERED.search(function("link_plan_build", source("forces.cu")))


# the sources whose kernels run on non-blocking streams, and the functions in
# them whose kernels run on the default stream as well
STREAMED = {"engine.cu": [], "tree.cu": [], "scan_sort.cu": [], "forces.cu": [], "fast.cu": [],
            "fmm.cu": [], "collide_spec.cu": [], "noalloc.cu": [], "fmm_tc.cu": ["fmm_tc_stats"],
            "batch.cu": []}


@pytest.mark.parametrize("name", sorted(STREAMED))
def test_set_up_is_on_the_stream(name):
    text = source(name)
    for f in STREAMED[name]:
        text = text.replace(function(f, text), "")
    assert [m.group(0) for m in UNORDERED.finditer(text)] == []

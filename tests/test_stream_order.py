"""Uploads and clears of the objects that step on streams of their own are made in those
streams: these do not wait for the legacy default stream, and a plain cudaMemcpy from
pageable memory or cudaMemset may return before it is done."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lattibol_0.3.31f_gb300", "csrc")


@pytest.mark.parametrize("name", ["lb_context.cu", "lb_closure.cu", "lb_ensemble.cu"])
def test_in_stream(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert "cudaStreamNonBlocking" in text
    calls = list(re.finditer(r"cudaMem(?:set|cpy)\s*\([^;]*;", text))
    for m in calls:
        if "cudaMemcpyDeviceToHost" in m.group(0):
            continue  # complete when it returns
        # the C ABI's plain copies, completed before they return
        assert text[m.end():].lstrip().startswith(
            "if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);"), m.group(0)
    # nothing is queued on a stream that has not been created yet
    for handle in ("c->stream", "m->stream", "e->stream"):
        made = text.find("cudaStreamCreateWithFlags(&" + handle)
        if made >= 0:
            create = text.rfind("\nint ", 0, made)
            assert handle + ")" not in text[create:made], handle

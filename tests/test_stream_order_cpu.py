"""Copies to the device are ordered before the kernels that read them.  A context's
stream is non-blocking: it does not wait for the legacy stream, which a plain cudaMemcpy
uses, and that call may return before data from pageable memory has arrived.  A missing
order shows itself only now and then on a GPU, so the sources are read instead."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amdat_gb300", "csrc")


def _calls(name):
    """(file, text from the call to the end of its statement) of every call of `name`"""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if path.endswith((".cu", ".cuh", ".h", ".cpp")):
            text = re.sub(r"//[^\n]*", "", open(path).read())
            out += [(os.path.basename(path), text[m.start():text.index(";", m.start())])
                    for m in re.finditer(r"\b%s\s*\(" % name, text)]
    return out


def test_no_host_to_device_copy_on_the_legacy_stream():
    assert [c for c in _calls("cudaMemcpy") if "HostToDevice" in c[1]] == []


def test_async_copies_name_the_stream():
    calls = _calls("cudaMemcpyAsync") + _calls("cudaMemsetAsync")
    assert len(calls) > 50
    assert [c for c in calls if not re.search(r"(ctx->stream|\bst)\s*\)+$", c[1])] == []

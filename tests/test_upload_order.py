"""Uploads from host memory are on the device before a kernel can read them.

Instances and batches run on non-blocking streams, which do not wait for work on
the legacy stream.  cudaMemcpy from pageable memory may return once the data is
staged, and cudaMemset returns before the memory is set: a kernel launched next on
a non-blocking stream could read a plan's items or its list of rebuilding instances
before they arrive, and use what it reads as an index.  That is a race, so it is
checked by reading the source and never provoked.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def test_no_copy_or_memset_outside_a_stream():
    found = [(name, m.group(0).strip()) for name, text in _sources()
             for m in re.finditer(r"[^\n]*\bcuda(Memcpy|Memset)\([^\n]*", text)]
    assert not found, found


def test_upload_waits_for_its_stream():
    text = dict(_sources())["fsim_sim.cu"]
    body = text[text.index("cudaError_t upload("):]
    body = body[:body.index("\n}\n")]
    assert body.index("cudaMemcpyAsync") < body.index("cudaStreamSynchronize(st)")
    # a plan's arena and its list of rebuilding instances go up this way and no other
    for dst in (r"pl->act", r"pl->arena", r"pl\.act", r"pl\.arena"):
        assert re.search(r"upload\(%s," % dst, text), dst
        assert not re.search(r"cuda\w*(Memcpy|Memset)\w*\(%s," % dst, text), dst

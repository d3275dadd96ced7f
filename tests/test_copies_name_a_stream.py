"""Every copy and fill of device memory in the library names the stream whose kernels use the memory. The library's own
streams are non-blocking, so nothing orders them after the default stream, and a copy from pageable memory on that one
may return to the host before it has ended."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mclics_b200", "csrc")


def test_no_copy_goes_to_the_default_stream():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cpp", ".cu", ".cuh", ".h")):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            found += [(name, m.group()) for m in re.finditer(r"\bcuda(Memcpy(2D|3D)?|Memset(2D)?|MemcpyToSymbol)\s*\(", text)]
    assert not found

"""Tables reach the device by copies from pageable memory on the legacy stream, which may return before the data is
in place, while kernels run on non-blocking streams that do not wait for it.  Every such copy therefore goes through a
place that waits before the table is published: TableArrays (level and operator tables) or PerDeviceOnce (constants).
Checked on the sources: the race itself has no test that could not fault a GPU."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyteg_b200", "csrc")


def sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cpp", ".cuh", ".hpp")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def body(text, start):
    """The braced block that opens after `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return i, j
    raise AssertionError("unbalanced braces")


def test_host_copies_wait_before_their_tables_are_used():
    found = 0
    for name, text in sources():
        waited = [body(text, m.start()) for m in re.finditer(r"\w*once\w*\.run\(\s*\[|class TableArrays\b", text)]
        for m in re.finditer(r"\bcudaMemcpy(ToSymbol)?\(\s*[^;]*;", text):
            if not m.group(1) and "cudaMemcpyHostToDevice" not in m.group(0):
                continue
            found += 1
            assert any(a < m.start() < b for a, b in waited), f"{name}: {m.group(0)[:90]}"
        assert not re.search(r"\bcudaMemset\( ", text), f"{name}: cudaMemset runs on the legacy stream"
    assert found > 10
    text = dict(sources())["hyb_internal.hpp"]
    for owner, method in (("class TableArrays", "void keep()"), ("class PerDeviceOnce", "void run(")):
        a, b = body(text, text.index(owner))
        c, d = body(text, text.index(method, a))
        assert "finish_uploads()" in text[c:d] and d < b, owner
    a, b = body(text, text.index("inline void finish_uploads()"))
    assert "cudaStreamSynchronize( cudaStreamLegacy )" in text[a:b]

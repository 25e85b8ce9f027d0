"""Every context's stream is non-blocking, so nothing orders its kernels after a
copy or fill on the legacy stream, and a copy from pageable memory there may
return before its transfer has ended.  What the host writes to the device
therefore goes through the context's own stream everywhere: no call of the
library copies to the device or fills device memory on the legacy one."""

import os
import re

import host_kernel as hk


def _calls(name):
    """(line, text) of each call of `name` in the library's sources."""
    for f in sorted(os.listdir(hk.CSRC)):
        if not f.endswith((".cu", ".cpp", ".hpp", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", hk.source(f))
        for m in re.finditer(rf"\b{name}\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            yield f"{f}:{text.count(chr(10), 0, m.start()) + 1}", text[m.start():i]


def test_no_upload_on_the_legacy_stream():
    assert [at for at, call in _calls("cudaMemcpy") if "DeviceToHost" not in call] == []
    assert list(_calls("cudaMemset")) == []


def test_asynchronous_ones_name_a_stream():
    for name, args in (("cudaMemcpyAsync", 5), ("cudaMemsetAsync", 4)):
        for at, call in _calls(name):
            depth, commas = 0, 0
            for ch in call:
                depth += {"(": 1, ")": -1}.get(ch, 0)
                commas += ch == "," and depth == 1
            assert commas + 1 == args, at

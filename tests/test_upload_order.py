"""Contexts work on their own non-blocking streams.  cudaMemcpy from pageable
memory may return before its data has arrived on the device, and cudaMemset
returns at once; both run on the default stream, which those streams do not wait
for.  So either goes on a context's stream or is followed, in the same function, by
a wait for the default stream."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "messi_gb300", "csrc")


def unordered(src):
    """Lines with a default-stream upload or memset and no wait for it further down in their function."""
    out, pending = [], []
    for n, line in enumerate(src.splitlines(), 1):
        code = line.split("//")[0]
        if re.search(r"\bcudaMemset\(|\bcudaMemcpy\([^;]*cudaMemcpyHostToDevice", code):
            pending.append(n)
        if re.search(r"\bcudaStreamSynchronize\(0\)|\bcudaDeviceSynchronize\(", code):
            pending = []
        if line.startswith("}"):
            out += pending
            pending = []
    return out


def test_the_scan_sees_both_kinds():
    bad = "void f()\n{\n    cudaMemcpy(d, h, n, cudaMemcpyHostToDevice);\n    cudaMemset(d, 0, n);\n}\n"
    assert unordered(bad) == [3, 4]
    assert unordered(bad.replace("\n}", "\n    cudaStreamSynchronize(0);\n}")) == []


def test_uploads_are_ordered_before_their_use():
    files = [f for k in ("*.cu", "*.cuh", "*.cpp", "*.h") for f in glob.glob(os.path.join(CSRC, k))]
    assert len(files) >= 10
    found = {}
    for path in files:
        with open(path) as f:
            lines = unordered(f.read())
        if lines:
            found[os.path.basename(path)] = lines
    assert not found

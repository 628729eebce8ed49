"""A handle's and an ensemble's kernels run on non-blocking streams, which the
legacy stream is not ordered with: a fill there is asynchronous, and a copy of a
pageable host array may still be under way when the call returns.  So the
library's fills and copies to the device name a stream."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "openqg_b200", "csrc")


def _calls(text, name):
    """The argument text of each call of name."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_device_fills_and_copies_name_a_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        text = open(path).read()
        for name in ("cudaMemset", "cudaMemset2D", "cudaMemcpyToSymbol"):
            found += [(os.path.basename(path), name, a) for a in _calls(text, name)]
        for name in ("cudaMemcpy", "cudaMemcpy2D"):
            found += [(os.path.basename(path), name, a) for a in _calls(text, name) if "cudaMemcpyDeviceToHost" not in a]
    assert not found

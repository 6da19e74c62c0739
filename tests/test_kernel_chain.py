"""Kernels are launched as a chain (a kernel's blocks may be placed before the kernel ahead of it is complete), so each one
has to begin by waiting for that kernel: read from the sources."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rust-compress_gb300", "csrc")


def _kernels(text):
    """(name, start of the body) of every kernel definition."""
    for m in re.finditer(r"__global__", text):
        at, depth = m.end(), 0
        while not (depth == 0 and text[at] in "{;"):
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        if text[at] == "{":
            yield re.findall(r"\b(k_\w+)\s*\(", text[m.end():at])[0], text[at + 1:].lstrip()


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_every_kernel_waits_first(path):
    with open(path) as f:
        bad = [name for name, body in _kernels(f.read()) if not body.startswith("grid_chain();")]
    assert not bad, bad


def test_kernels_are_found():
    texts = [open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu"))]
    found = [k for t in texts for k in _kernels(t)]
    assert found and len(found) == sum(t.count("__global__") for t in texts)

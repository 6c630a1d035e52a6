"""Kernels that launch ahead of their predecessors' ends (they call wait_previous) read what a predecessor may
still write with ordinary loads: a read-only load promises data that does not change while the kernel lives.
Checked on the source, since a stale line shows only where the schedule happens to allow it."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parabiofvm_b200", "csrc")
READ_ONLY = re.compile(r"__ldg\(\s*&?([\w.]+)|ld\.global\.nc")
# constant while their owner lives: coefficients, mask words, bias rows
CONSTANT = {"a.ltab", "a.vtab", "a.masks", "at", "from", "ts", "p.bias", "gqtab", "tgptab", "Gptab"}


def _body(text, start):
    """The braces' block that opens at or after `start`."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_convolution_epilogue_reads_activations_with_ordinary_loads():
    text = _source("surrogate.cu")
    assert "wait_previous();" in _body(text, text.index("sur_conv_kernel(const"))
    for what in ("struct bf16x32", "sur_conv_kernel(const"):
        found = {m.group(1) for m in READ_ONLY.finditer(_body(text, text.index(what)))}
        assert found <= {"p.bias"}, what


@pytest.mark.parametrize("name", ["small.cu", "gradient.cu", "bins.cu", "cell.cu"])
def test_overlapping_kernels_read_only_constants_as_read_only(name):
    text = re.sub(r"//.*", "", _source(name))
    if name == "cell.cu":  # the kernels of the chain; the others launch after their predecessors' ends
        text = "".join(_body(text, m.end()) for m in re.finditer(r"__global__[^{;]*", text)
                       if "wait_previous();" in _body(text, m.end() - 1))
    for m in READ_ONLY.finditer(text):
        if m.group(1):
            assert m.group(1) in CONSTANT, m.group(0)
        else:  # the predicated load of conditions in small.cu
            assert name == "small.cu" and "replace_where" in text[max(0, m.start() - 300):m.start()]

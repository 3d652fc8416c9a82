"""The order of tensor-core instructions on one accumulator: PTX keeps two tcgen05.mma in flight in
their order only where they share the accumulator and the shape, so a tile that is accumulated onto
must have been started by the same call, not by an MMA of another kind.  (What hardware does with
another pair cannot be shown by running it.)"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmp_b200", "csrc")


def _calls(text):
    """(kind, last argument) of every tc::Mma* call."""
    for m in re.finditer(r"\btc::Mma(I8|F16|Mxf8)\w*\(", text):
        depth, at, last = 1, m.end(), m.end()
        while depth:
            c = text[at]
            depth += (c == "(") - (c == ")")
            if c == "," and depth == 1:
                last = at + 1
            at += 1
        yield m.group(1), text[m.end():at - 1], text[last:at - 1].strip()


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_an_accumulating_mma_starts_its_own_tile(path):
    text = re.sub(r"//.*", "", open(path).read())
    for kind, arguments, last in _calls(text):
        # the Mxf8 wrappers take the scales after the accumulate argument
        accumulate = last if kind != "Mxf8" else arguments
        assert accumulate == "false" or re.search(r"> 0\b", accumulate), (kind, " ".join(arguments.split()))

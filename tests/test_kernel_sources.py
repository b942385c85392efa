"""Rules the kernel sources follow, checked on their text (no GPU).

Divisions, reciprocals, roots and elementary functions are the CUDA language's
operators and math functions: no source builds one of its own from the
hardware's approximate instructions."""
import os
import re

import pytest

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h", ".cpp")))


@pytest.mark.parametrize("name", SOURCES)
def test_no_arithmetic_from_approximate_instructions(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    found = re.findall(r"\b(?:rcp|div|rsqrt|sqrt|sin|cos|lg2|ex2|tanh)\.(?:approx|full)[.\w]*", text)
    assert not found, found

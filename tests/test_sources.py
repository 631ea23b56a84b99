"""The kernels call CUDA's own division, reciprocal and square root: the sources
hold no hand-made replacement built on the approximate instructions, whose rounding
nothing here states or tests."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mg-picola-public_gb300", "csrc")


def test_no_approximate_division_or_root():
    files = [f for f in glob.glob(os.path.join(CSRC, "*")) if f.endswith((".cu", ".cuh", ".h"))]
    assert files
    for f in files:
        with open(f) as src:
            assert not re.search(r"\b(rcp|rsqrt|sqrt|div)\.approx", src.read()), os.path.basename(f)

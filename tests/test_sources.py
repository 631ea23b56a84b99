"""Rules of the CUDA sources.

The kernels call CUDA's own division, reciprocal and square root: the sources
hold no hand-made replacement built on the approximate instructions, whose rounding
nothing here states or tests.

No copy to the device that returns before it is done reads a vector of the calling function:
where the device reads pageable memory itself the copy may run after the vector is freed.
Such tables go through page-locked slots, or live until the stream has passed the copy
(`host` and `tab`, of the initial conditions), or the call waits for the stream."""
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


def test_no_asynchronous_upload_from_a_local_vector():
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(f) as src:
            calls = re.findall(r"cudaMemcpyAsync\(([^;]*?)cudaMemcpyHostToDevice", src.read())
        for c in calls:
            assert not re.search(r"(?<!tab\.back\(\))(?<!host\.box)\.data\(\)", c), (os.path.basename(f), c)

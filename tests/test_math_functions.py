"""The kernels take roots and reciprocals from CUDA's own functions: no refinement of the hardware's first
approximations of their own, whose error nothing here bounds."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wantibexos_b200", "csrc")


def test_no_approximate_roots_or_reciprocals():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r"\b(rsqrt|sqrt|rcp|div)\.(approx|full)\b", text), name
            assert not re.search(r"\bfast_(rsqrt|rcp)\b", text), name

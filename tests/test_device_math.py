"""CPU test of the device sources: reciprocals, divisions, square roots and exponentials are CUDA's own
functions (correctly rounded or with CUDA's stated bounds over the whole range of their arguments), not
refinements of the hardware's approximations written out here."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(f for ext in ("cu", "cuh", "h")
                 for f in glob.glob(os.path.join(ROOT, "hubbard-attractive-u_b200", "**", "*." + ext), recursive=True))


def test_no_approximate_instructions():
    assert SOURCES
    bad = []
    for f in SOURCES:
        for k, line in enumerate(open(f), 1):
            if re.search(r"\b(rcp|rsqrt|sqrt|div|ex2|lg2|sin|cos|tanh)\.approx", line):
                bad.append("%s:%d: %s" % (os.path.relpath(f, ROOT), k, line.strip()))
    assert not bad, bad

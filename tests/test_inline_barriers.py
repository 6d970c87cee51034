"""Inline PTX barriers of the kernels are the forms that lanes of a warp may reach one
by one. The aligned forms (bar.*, barrier.*.aligned) are undefined unless the whole warp
executes them together, which nothing guarantees behind a branch or a loop whose trip
count differs between lanes."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "sphadjoint_gb300", "csrc")


def barriers(text):
    for asm in re.findall(r"asm\s+volatile\s*\((.*?)\);", text, re.S):
        ptx = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', asm))
        yield from re.findall(r"\bbar(?:rier)?\.[a-z_.]+", ptx)


def test_no_aligned_barrier():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            found += [(os.path.basename(path), b) for b in barriers(f.read())]
    assert found  # the pattern still finds the kernels' barriers
    bad = [x for x in found if x[1].startswith("bar.") or ".aligned" in x[1]]
    assert not bad, bad

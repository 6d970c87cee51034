"""Kernels that build neighbour masks and walk them in the same launch: a function that
sees the state's arrays through NLView must not also take the masks or centres it writes
as restrict pointers (the compiler could then move the walk's loads above the stores and
sum over the masks of the previous cell list)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "sphadjoint_gb300", "csrc")
WRITTEN = re.compile(r"(?<!const )\buint32_t \*__restrict__ (center|masks)\b")


def signatures(text):
    """(name, parameters) of the functions defined in a CUDA source."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\b(\w+)\(((?:[^(){};]|\([^()]*\))*)\)\s*\{", text):
        yield m.group(1), " ".join(m.group(2).split())


def test_masks_read_through_the_view_are_not_restrict_outputs():
    seen, bad = set(), []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            for name, params in signatures(f.read()):
                seen.add(name)
                if "NLView" in params and WRITTEN.search(params):
                    bad.append((os.path.basename(path), name))
    assert {"nl_window", "k_nl_density_win", "k_density_eos_coop", "k_density_flat"} <= seen
    assert not bad, bad

"""Shared-memory arrays of the kernels declare the alignment that their wide accesses need: where the compiler happens to put an array is no promise."""
import glob
import os
import re

import pytest

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inference-agent_b200")
SOURCES = sorted(f for part in ("csrc", "backend") for ext in ("*.cu", "*.cuh") for f in glob.glob(os.path.join(PACKAGE, part, ext)))
# accessed float by float
ELEMENTWISE = {"moe.cu": {"s_choice_all"}}


def declarations(path):
    """(array name or "", declaration) of every line that declares shared memory."""
    with open(path) as f:
        for line in f:
            m = re.match(r"\s*((?:extern\s+)?__shared__\s+[^;/]*);", line)
            if m:
                yield re.search(r"(\w+)\s*\[", m.group(1)).group(1) if "[" in m.group(1) else "", m.group(1)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_dynamic_arrays_are_aligned(path):
    with open(path) as f:
        text = f.read()
    for name, decl in declarations(path):
        if "extern" in decl and name not in ELEMENTWISE.get(os.path.basename(path), ()):
            assert "__align__(16)" in decl or f"(smem_u32({name}) + 1023u) & ~1023u" in text, decl


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_pairs_are_pairs_by_type(path):
    """Pairs of floats that other CTAs read in one access (cluster_load2) lie on 8 bytes by their type."""
    for name, decl in declarations(path):
        assert "__align__" in decl or not re.search(r"\bfloat\s+\w+\s*\[[^\]]*\]\s*\[2\]", decl), decl

"""Dynamic shared memory that is accessed wider than its elements says so: where the array begins beside a kernel's static shared
memory is the tool chain's choice unless the declaration asks for an alignment (or the kernel rounds the address up)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmplayer_b200", "csrc")
WIDE = re.compile(r"\b(float2|float4|uint2|uint4|ulonglong2|uint64_t|bulk_load|tma_load_2d|ldmatrix\w*)\b|cp\.async")


def bare_arrays(text):
    """(line, name) of every dynamic shared array without an alignment in a kernel that makes wide accesses."""
    found = []
    for m in re.finditer(r"extern __shared__ ([^;]*?)(\w+)\[\];", text):
        if "__align__" in m.group(1):
            continue
        body = text[m.end():text.index("\n}", m.end())]
        rounds_up = re.search(re.escape(m.group(2)) + r" \+ 1023\) & ~\(uintptr_t\)1023", body)
        if WIDE.search(body) and not rounds_up:
            found.append((text.count("\n", 0, m.start()) + 1, m.group(2)))
    return found


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_wide_accesses_ask_for_their_alignment(path):
    with open(path) as fh:
        assert bare_arrays(fh.read()) == []

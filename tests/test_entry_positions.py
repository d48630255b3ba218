"""No kernel walks a row's entries with a signed 32-bit index: a row may end at 2^31 - 1, and the step past it would wrap.

(tests/native/entry_positions.cu runs the loops' form at that limit.)
"""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "acc-gp_b200", "csrc")
BOUND = r"(?:\bend\b|\be_end\b|\brow_end\b|\bdegree\b|(?<!\w)off\[|chunk_end\()"
SIGNED_WALK = re.compile(r"for \(int \w+ = [^;]*;[^;]*" + BOUND + r"[^;]*;[^)]*\+=")
SIGNED_PARAMETER = re.compile(r"\bint (?:first|begin), int end\b|\bint first,\s+int end\b")
SIGNED_START = re.compile(r"chunk_begin\[\w+\] \+ static_cast<int>")
SIGNED_PROBE = re.compile(r"\bb \+ j < end\b")


def test_rows_are_walked_with_unsigned_positions():
    walks = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h")) or name == "gp_refine_cluster.cuh":  # levels of 2^18 entries at most
            continue
        text = open(os.path.join(CSRC, name)).read()
        for pattern in (SIGNED_WALK, SIGNED_PARAMETER, SIGNED_START, SIGNED_PROBE):
            found = pattern.search(text)
            assert not found, f"{name}: {found.group(0)}"
        walks += len(re.findall(r"for \(EntryPos ", text))
    assert walks >= 18

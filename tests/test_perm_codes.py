"""The walk records' permutation codes: each of the six permutations of a
shared face has a code of its own whose selector moves the exit face's bytes
(1 to 3 of the vertex map) into the next tet's order and leaves byte 0 alone;
0 (a boundary face) and 4 (ids that do not match) name none."""
import itertools
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT


def test_codes_and_selectors(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path / "perm_codes")
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "vfray_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "perm_codes.cc"), "-o", exe],
                   check=True, timeout=120)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60, check=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == 27
    seen = set()
    for p0, p1, p2, code, selector in rows:
        if (p0, p1, p2) in set(itertools.permutations(range(3))):
            # the selector's nibbles 0..3 name the source of bytes 0..3
            assert [selector >> 4 * k & 15 for k in range(4)] == [0, p0 + 1, p1 + 1, p2 + 1]
            assert code in range(1, 8) and code != 4
            # the walk's test for boundary and unmatched faces: bits 29 and 30
            assert (code << 29) & 0x60000000
            seen.add(code)
        else:
            assert code == 0
    assert len(seen) == 6

"""CPU: no two object files of the library define the same weak function of ours.  The linker keeps one of them, so that types of one name in two
files would make the one file's calls run the other's code (a dispatch that picked the other file's kernel read out of range)."""
import os
import shutil
import subprocess
from collections import defaultdict

import pytest

OBJ = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "f2cgt_b200", "csrc", "_obj")


@pytest.mark.skipif(shutil.which("nm") is None or not os.path.isdir(OBJ) or not os.listdir(OBJ), reason="no object files here")
def test_no_weak_function_of_ours_is_in_two_object_files():
    where = defaultdict(set)
    for name in sorted(os.listdir(OBJ)):
        if name.endswith(".o") and not name.startswith("native_"):
            out = subprocess.run(["nm", os.path.join(OBJ, name)], check=True, capture_output=True, text=True).stdout
            for line in out.splitlines():
                kind, symbol = line.split()[-2:]
                if kind in "WVu" and symbol.startswith(("_ZN3f2c", "_ZNK3f2c")):
                    where[symbol].add(name)
    assert not {s: f for s, f in where.items() if len(f) > 1}

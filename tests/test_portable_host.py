"""Host code compiles off x86: what one processor family alone has stands under that family's #if."""
import glob
import os
import re

from conftest import ROOT


def test_x86_intrinsics_are_guarded():
    bare = []
    for path in sorted(glob.glob(os.path.join(ROOT, "modules_b200", "csrc", "*.*"))):
        guards = []
        with open(path) as f:
            for number, line in enumerate(f, 1):
                if re.match(r"\s*#\s*if", line):
                    guards.append("__x86_64__" in line)
                elif re.match(r"\s*#\s*(elif|else)", line):
                    guards[-1] = "__x86_64__" in line
                elif re.match(r"\s*#\s*endif", line):
                    guards.pop()
                elif re.search(r"\b_mm_\w+|[xei]mmintrin\.h", line.split("//")[0]) and not any(guards):
                    bare.append(f"{os.path.basename(path)}:{number}")
    assert not bare, bare

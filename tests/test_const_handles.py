"""Queries of a const handle change nothing in it (they may run beside an evaluation of another thread). The compiler holds
the C ABI's const functions to that as long as no member is exempt from it."""
import glob
import os
import re

from conftest import ROOT


def test_no_member_changes_behind_const():
    bare = []
    for path in sorted(glob.glob(os.path.join(ROOT, "modules_b200", "csrc", "*.*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        # (a lambda may be mutable: its captures are its own)
        bare += [f"{os.path.basename(path)}: {m}" for m in re.findall(r"\bmutable\s+\w[^\n]*|const_cast<cc_handle[^\n]*", text)]
    assert not bare, bare

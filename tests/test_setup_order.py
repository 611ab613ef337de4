"""Set-up work and the streams that read it. Handles, batches and the server evaluate on non-blocking streams, which do not
wait for the legacy stream, and a copy from pageable memory may return before its last piece has landed: a fill or upload
on the legacy stream therefore ends with a synchronisation of that stream in the same function, or it is issued on the
stream that reads it. Read from the sources: the windows are too narrow to be seen in a run."""
import glob
import os
import re

from conftest import ROOT

LEGACY = re.compile(r"\bcudaMemset\(|\bcudaMemcpy\((?=.*cudaMemcpyHostToDevice)")
WAIT = "cudaStreamSynchronize(nullptr)"


def unordered(text):
    """Lines of legacy-stream fills and uploads that no synchronisation follows within their function."""
    out, open_ = [], []
    for number, line in enumerate(text.splitlines(), 1):
        code = line.split("//")[0]
        if LEGACY.search(code):
            open_.append((number, code.strip()))
        if WAIT in code:
            open_ = []
        if line.startswith("}"):   # the end of a function (or of a namespace)
            out += open_
            open_ = []
    return out + open_


def test_rule_sees_both_forms():
    bad = "int f()\n{\n\tcudaMemset(p, 0, 4);\n}\n"
    assert unordered(bad) == [(3, "cudaMemset(p, 0, 4);")]
    assert unordered(bad.replace("4);\n", "4);\n\tcudaStreamSynchronize(nullptr);\n")) == []
    assert unordered("int f()\n{\n\tcudaMemcpy(p, q, 4, cudaMemcpyDeviceToHost);\n}\n") == []
    assert len(unordered("int f()\n{\n\tcudaMemcpy(p, q, 4, cudaMemcpyHostToDevice);\n}\n")) == 1


def test_setup_on_the_legacy_stream_is_waited_for():
    found = {}
    for path in sorted(glob.glob(os.path.join(ROOT, "modules_b200", "csrc", "*.*"))):
        with open(path) as f:
            lines = unordered(f.read())
        if lines:
            found[os.path.basename(path)] = lines
    assert not found, found
